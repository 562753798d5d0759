// Programmatic dependent launch, device side (host side: KB_LAUNCH_PDL in launch.h).
//
// A kernel that is launched this way may start while the kernel before it on the stream is still running: its blocks take
// their place on the chip and set themselves up, and what they do with memory waits for pdl_wait().  Rules:
//  * every thread calls pdl_wait() before its first access to global memory, reads and writes alike, and before it returns.
//    It holds until the kernels before this one have completed and their writes are visible, so the order of
//    memory accesses on a stream is what it is without any of this;
//  * pdl_launch() lets the next kernel's blocks in once all blocks of this one have called it.  A kernel that allocates
//    TMEM calls it after the allocation: a block of a later kernel that got the SM's TMEM first would be waited for and
//    wait itself;
//  * kernels that wait for other GPUs are not launched this way and let nobody in early.
// What it is for: between two dependent kernels of a few us each lie 1 to 2 us of launch, barrier and TMEM set-up that need no
// data.  One B200, before / after: forward region of the 2-layer smoke model (44 kernels, replayed as a graph) 174 / 152 us,
// its recompute and backward (120) 525 / 486; three GEMMs of 328 x 1032 x 776 25.2 / 21.8.  137 GEMMs drawn up to 90 us, in graphs
// of 8: 12 % shorter as a mean below 6 us, 8 % to 12 us, 3 % to 30 us, 2 % above.  Not every call gains: some of 15 to 60 us lose 2 to 10 %
// (weight gradient 176 x 6240 over 4729 rows 21.3 / 23.4, 16806 x 512 → 1024 and its SwiGLU gradient 47.2 / 51.5, 290 x 3072 → 2 x 2048
// and its SwiGLU 17.6 / 19.2), whether a GEMM lets the next kernel in at its start or after its last load; elementwise kernels
// that let nobody in cost 3 % more.  No size or kind of call was found that tells them apart, so all are launched this way.
#pragma once

namespace kb {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_begin() {
  pdl_launch();
  pdl_wait();
}

}  // namespace kb
