// Two kernels of a stream that run beside each other from start to end.
#pragma once

#include <cstdint>

namespace w8a8 {

// For a kernel that reads nothing of what the kernel before it writes and writes nothing that it reads, where that one
// lets it in only after its own wait (after_previous<false>): all that came before the two is then complete, and this one
// need not wait at its start.  It waits at its end instead (previous_complete), so that whoever waits for it has waited
// for both.
__device__ __forceinline__ int64_t beside_previous()
{
    int64_t zero;
    // no line that this SM's L1 holds from before
    asm volatile("griddepcontrol.launch_dependents;\n\tfence.acq_rel.gpu;\n\tmov.u64 %0, 0;" : "=l"(zero)::"memory");
    return zero;
}

__device__ __forceinline__ void previous_complete() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

}  // namespace w8a8
