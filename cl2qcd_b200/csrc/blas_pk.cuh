// blas_pk.cuh -- the level-1 BLAS of blas.cuh and the precision conversions on the
// paired-site slots of the FP32 / FP16 fields (pack.cuh): one thread per slot, whole
// 16-byte words, packed FP32 arithmetic.
//
// The passes are bound by memory.  Read site by site, a warp uses half of every
// sector of these fields (its two sites share each word) and the other half is
// fetched again by the block that handles the other half of the time axis.
#pragma once

#include "blas.cuh"
#include "pack.cuh"

namespace c2q {

constexpr int BLAS_PK_THREADS = 128;

template <int P>
__device__ __forceinline__ void slot_load(const SpinorPtr<P>& f, int ss, int j, C2 s[12])
{
    if constexpr (P == 16)
        SlotF16::load(f.data, f.norm, ss, j, s);
    else
        SlotF32::load(f.data, ss, j, s);
}
template <int P>
__device__ __forceinline__ void slot_store(const SpinorPtr<P>& f, int ss, int j, const C2 s[12])
{
    if constexpr (P == 16)
        SlotF16::store(f.data, f.norm, ss, j, s);
    else
        SlotF32::store(f.data, ss, j, s);
}

struct CoefPk {
    float2 re, im, nim;
};
__device__ __forceinline__ CoefPk coef_pk(const Coef& c)
{
    const Cplx<double> v = coef_value(c);
    return CoefPk{bc2((float)v.re), bc2((float)v.im), bc2((float)-v.im)};
}
// c b, a + c b, a - c b
__device__ __forceinline__ C2 cmul_pk(const CoefPk& c, C2 b)
{
    return C2{fma2(b.im, c.nim, mul2(b.re, c.re)), fma2(b.re, c.im, mul2(b.im, c.re))};
}
__device__ __forceinline__ C2 caxpy_pk(C2 a, const CoefPk& c, C2 b)
{
    return C2{fma2(b.im, c.nim, fma2(b.re, c.re, a.re)), fma2(b.re, c.im, fma2(b.im, c.re, a.im))};
}
__device__ __forceinline__ CoefPk neg_pk(const CoefPk& c)
{
    const float2 m = bc2(-1.0f);
    return CoefPk{mul2(c.re, m), c.nim, c.im};
}
__device__ __forceinline__ C2 neg_pk(C2 a) { return C2{mul2(a.re, bc2(-1.0f)), mul2(a.im, bc2(-1.0f))}; }

// conj(x) y, its two sites added to re and im in FP64
__device__ __forceinline__ void dot_pk(C2 x, C2 y, double& re, double& im)
{
    const float2 r = fma2(x.re, y.re, mul2(x.im, y.im));
    const float2 i = fma2(x.im, mul2(y.re, bc2(-1.0f)), mul2(x.re, y.im));
    re += (double)r.x + (double)r.y;
    im += (double)i.x + (double)i.y;
}
// |x|^2 in FP64
__device__ __forceinline__ double norm_pk(C2 x)
{
    return ((double)x.re.x * x.re.x + (double)x.im.x * x.im.x) + ((double)x.re.y * x.re.y + (double)x.im.y * x.im.y);
}

template <int P>
__global__ void __launch_bounds__(BLAS_PK_THREADS) blas_pk_kernel(const BlasArgs<P> A)
{
    pdl_enter();
    if (halted(A.red)) return;  // a stopped device-driven solve: every block leaves
    const int j = blockIdx.x * BLAS_PK_THREADS + threadIdx.x;
    const int ss = A.stride >> 1;
    double dv[4] = {0.0, 0.0, 0.0, 0.0};
    if (j < A.n / 2) {
        if (A.op == B_COPY && !A.dot) {  // word for word
            const uint4* p  = static_cast<const uint4*>(A.x.data) + j;
            uint4* q        = static_cast<uint4*>(A.out.data) + j;
            constexpr int n = P == 16 ? 6 : 12;
#pragma unroll
            for (int L = 0; L < n; ++L) q[(size_t)L * ss] = __ldg(p + (size_t)L * ss);
            if (P == 16) reinterpret_cast<float2*>(A.out.norm)[j] = __ldg(reinterpret_cast<const float2*>(A.x.norm) + j);
            return;
        }
        C2 xv[12], r[12];
        slot_load<P>(A.x, ss, j, xv);
        if (A.op == B_BICG_XR) {
            // x = alpha p + omega s + x; rn = s - omega t; |rn|^2 and (rhat, rn)
            const CoefPk a = coef_pk(A.a), b = coef_pk(A.b), nb = neg_pk(b);
            C2 yv[12];
            slot_load<P>(A.y, ss, j, yv);
            slot_load<P>(A.out, ss, j, r);
#pragma unroll
            for (int k = 0; k < 12; ++k) r[k] = caxpy_pk(caxpy_pk(r[k], a, xv[k]), b, yv[k]);
            slot_store<P>(A.out, ss, j, r);
            slot_load<P>(A.z, ss, j, xv);
#pragma unroll
            for (int k = 0; k < 12; ++k) r[k] = caxpy_pk(yv[k], nb, xv[k]);
            slot_store<P>(A.out2, ss, j, r);
            // (the reductions use the values computed here, not a load of what was just stored)
            slot_load<P>(A.w, ss, j, yv);
#pragma unroll
            for (int k = 0; k < 12; ++k) {
                dv[0] += norm_pk(r[k]);
                dot_pk(yv[k], r[k], dv[2], dv[3]);
            }
        } else if (A.dot == 1 || A.dot == 3) {
            C2 yv[12];
            slot_load<P>(A.y, ss, j, yv);
#pragma unroll
            for (int k = 0; k < 12; ++k) {
                dot_pk(xv[k], yv[k], dv[0], dv[1]);
                if (A.dot == 3) dv[2] += norm_pk(xv[k]);
            }
        } else {
            const CoefPk a = coef_pk(A.a), b = coef_pk(A.b);
            switch (A.op) {
                case B_SAXPY:
                case B_SAXPY_G5: {
                    const CoefPk na = neg_pk(a);
                    slot_load<P>(A.y, ss, j, r);
#pragma unroll
                    for (int k = 0; k < 12; ++k) {
                        r[k] = caxpy_pk(r[k], na, xv[k]);
                        if (A.op == B_SAXPY_G5 && k >= 6) r[k] = neg_pk(r[k]);
                    }
                    break;
                }
                case B_SAX:
#pragma unroll
                    for (int k = 0; k < 12; ++k) r[k] = cmul_pk(a, xv[k]);
                    break;
                case B_SAXSBYPZ: {
                    C2 yv[12];
                    slot_load<P>(A.y, ss, j, yv);
                    slot_load<P>(A.z, ss, j, r);
#pragma unroll
                    for (int k = 0; k < 12; ++k) r[k] = caxpy_pk(caxpy_pk(r[k], a, xv[k]), b, yv[k]);
                    break;
                }
                case B_COPY:
#pragma unroll
                    for (int k = 0; k < 12; ++k) r[k] = xv[k];
                    break;
                case B_GAMMA5:
#pragma unroll
                    for (int k = 0; k < 12; ++k) r[k] = k >= 6 ? neg_pk(xv[k]) : xv[k];
                    break;
                case B_DIAG:
#pragma unroll
                    for (int k = 0; k < 12; ++k) r[k] = cmul_pk(k < 6 ? a : b, xv[k]);
                    break;
            }
            slot_store<P>(A.out, ss, j, r);
            if (A.dot == 2)
#pragma unroll
                for (int k = 0; k < 12; ++k) dv[0] += norm_pk(r[k]);
        }
    }
    if (A.dot == 3 || A.dot == 4) {
        __shared__ double smem4[128];
        block_sum<4>(dv, smem4);
        finish_reduction<4>(dv, A.red, smem4);
    } else if (A.dot) {
        __shared__ double smem[64];
        block_sum<2>(dv, smem);
        finish_reduction<2>(dv, A.red, smem);
    }
}

// Precision conversion between slots, and between slots and FP64 fields (the
// slot's two sites are the FP64 sites j and j + n / 2).
template <int PO, int PI>
__global__ void __launch_bounds__(BLAS_PK_THREADS) convert_pk_kernel(SpinorPtr<PO> out, SpinorPtr<PI> in, int n,
                                                                     int stride)
{
    const int j = blockIdx.x * BLAS_PK_THREADS + threadIdx.x;
    const int H = n / 2, ss = stride >> 1;
    if (j >= H) return;
    C2 v[12];
    if constexpr (PI == 64) {
        const double2* p = static_cast<const double2*>(in.data);
#pragma unroll
        for (int k = 0; k < 12; ++k) {
            const double2 a = __ldg(p + (size_t)k * stride + j), b = __ldg(p + (size_t)k * stride + j + H);
            v[k]            = C2{make_float2((float)a.x, (float)b.x), make_float2((float)a.y, (float)b.y)};
        }
    } else {
        slot_load<PI>(in, ss, j, v);
    }
    if constexpr (PO == 64) {
        double2* p = static_cast<double2*>(out.data);
#pragma unroll
        for (int k = 0; k < 12; ++k) {
            p[(size_t)k * stride + j]     = make_double2((double)v[k].re.x, (double)v[k].im.x);
            p[(size_t)k * stride + j + H] = make_double2((double)v[k].re.y, (double)v[k].im.y);
        }
    } else {
        slot_store<PO>(out, ss, j, v);
    }
}

}  // namespace c2q
