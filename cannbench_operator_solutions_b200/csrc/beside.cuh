// Two kernels of a stream that run beside each other from start to end.
#pragma once

#include <cstdint>

namespace w8a8 {

// For a kernel that reads nothing of what the kernel before it writes and writes nothing that it reads, where that one
// lets it in only after its own wait (after_previous<false>): all that came before the two is then complete, and this one
// need not wait at its start.  It waits at its end instead (previous_complete), so that whoever waits for it has waited
// for both.
// It lets the next kernel in at once, on a grid of any size.  A large grid that waits does so after its wait, because its
// idle blocks and the next kernel's would share the SMs unevenly (see after_previous); these blocks work from the start, and
// the next kernel's find a place only once every one of them has had its own.  Let in at the end instead, expert layers of
// 8 to 8192 tokens take the same (64 tokens 62.7 us, 62.8; 512 76.6, 76.7; 2000 252, 252; 8192 623 - 635, 621 - 634).
__device__ __forceinline__ int64_t beside_previous()
{
    int64_t zero;
    // no line that this SM's L1 holds from before
    asm volatile("griddepcontrol.launch_dependents;\n\tfence.acq_rel.gpu;\n\tmov.u64 %0, 0;" : "=l"(zero)::"memory");
    return zero;
}

__device__ __forceinline__ void previous_complete() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

}  // namespace w8a8
