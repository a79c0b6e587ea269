// The end of a kernel in which a bounded wait ran out.
#pragma once

namespace mpq {

// By every thread, when all roles have left their loops and before the CTA hands back its shared and tensor memory: copies and
// MMAs that were in flight when the wait ran out must land first.  They take microseconds; they are given a millisecond.
__device__ __forceinline__ void settle_after_timeout(bool timed_out)
{
    if (timed_out)
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
}

}  // namespace mpq
