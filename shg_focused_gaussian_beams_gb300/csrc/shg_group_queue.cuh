// The queue of a persistent group of blocks (shg_group.cu): the next job, the same in every block.
#pragma once

#include <cuda_runtime.h>

namespace shg {

// take(): one block of the group writes the queue's next number to the group's slot (at njobs and
// beyond the queue is empty); meet(): barrier among the group's blocks, false once a wait gave
// up; read(): the slot; good(job): whether the job is to be marched, the same in every block.
// False when the block leaves. The slot is written again only after a barrier that follows every
// block's read of it: the march's own (two or more), or one more here for a job that is skipped.
template <class Take, class Meet, class Read, class Good>
__device__ __forceinline__ bool group_next(unsigned &job, unsigned njobs, Take take, Meet meet, Read read, Good good) {
    for (;;) {
        take();
        if (!meet()) return false;
        job = read();
        if (job >= njobs) return false;
        if (good(job)) return true;
        if (!meet()) return false;
    }
}

}  // namespace shg
