// gridbar.cuh -- the grid barrier of the cooperative solver kernels.
#pragma once

namespace c2q {

// Every block of a cooperative launch (all blocks resident) meets here;
// `arrived` counts arrivals since the launch, `target` = blocks x barriers so
// far (an arrival short at the start of the launch, and no barrier completes: a test of
// the bound).  Writes before it are visible to every block after it (the acquiring
// load also drops the SM's L1 lines); data that the kernel changes must not be
// read through the non-coherent path.  Returns false once a wait has run out of
// polls (a fraction of a second; a block of a resident grid arrives within microseconds) or
// another block's wait has: the error word is then set and every block leaves,
// whatever it had got to; the fields hold any mixture of finished steps.
// (A constant: with the bound in a parameter the loop took 75 ns longer a barrier, 2 % of
// a solve at 8^4.)
constexpr unsigned GRIDBAR_POLLS = 1u << 20;
__device__ __forceinline__ bool grid_barrier(unsigned* arrived, unsigned* error, unsigned target, int* ok)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
        int good   = 1;
        unsigned n = 0, seen;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(arrived) : "memory");
            if ((int)(seen - target) >= 0) break;
            if (++n >= GRIDBAR_POLLS || ((n & 1023u) == 0 && *(volatile unsigned*)error)) {
                atomicExch(error, 1u);
                good = 0;
                break;
            }
        }
        *ok = good;
    }
    __syncthreads();
    return *ok != 0;
}

}  // namespace c2q
