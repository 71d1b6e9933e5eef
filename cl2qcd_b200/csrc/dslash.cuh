// dslash.cuh -- the even-odd Wilson hopping term with fused twisted-mass
// epilogues: its spin projection and SU(3) products.  The sweeps over one output
// parity are dslash64.cuh (FP64, one thread per site) and pdslash.cuh (FP32 / FP16,
// one thread per slot of two sites).
//
// Computes, at every site x of the output parity,
//   h(x) = sum_mu [ c_mu^+ (1 - g_mu) U_mu(x) psi(x+mu)
//                  + c_mu^- (1 + g_mu) U_mu(x-mu)^dagger psi(x-mu) ]
// with c^{+/-} = -kappa e^{+/- i theta pi / N} (times the chemical-potential
// factors on T links), which is the reference's dslash_eo
// (ocl_kernel/fermionmatrix_eo.cl:30-253, fermionmatrix_eo_dslash.cl:28-58),
// then applies one of the epilogues of c2q_internal.cuh:
//   EPI_PLAIN  dslash_eo
//   EPI_DIAG   dslash_AND_M_tm_inverse_sitediagonal(_minus)_eo
//              (fermionmatrix_eo_dslash_AND_M_tm_inverse_sitediagonal.cl:30-62)
//   EPI_AXPY   the tail of Aee / Aee_AND_gamma5_eo: [g5](M_diag(x) - h)
//              (physics/fermionmatrix/fermionmatrix.cpp:250-258, :330-338)
// and optionally reduces <y, out> (DOT_Y) or |out|^2 (DOT_SELF) across the
// grid with the deterministic last-block scheme of reduce.cuh.
//
// Spin projection: each 1 -/+ g_mu has rank two.  For upper spin rows a = 0, 1
// the half spinor is h_a = psi_a + c psi_p, c -> -c for 1 + g_mu; the lower
// row p receives conj(c) * (U h_a).  Forward (p, c) pairs, read off
// fermionmatrix_eo.cl:56-136:  T (2,1)(3,1)  X (3,i)(2,i)  Y (3,1)(2,-1)
// Z (2,i)(3,-i).  Multiplications by +-1, +-i are exact sign/swap operations.
#pragma once

#include "c2q_internal.cuh"
#include "reduce.cuh"

namespace c2q {

// multiply by c in {1, -1, i, -i}, encoded as K = 0, 1, 2, 3
template <int K, typename R>
__device__ __forceinline__ Cplx<R> mul_unit(Cplx<R> v)
{
    if (K == 0) return v;
    if (K == 1) return {-v.re, -v.im};
    if (K == 2) return {-v.im, v.re};
    return {v.im, -v.re};
}
// conj of the unit K
template <int K>
struct ConjUnit {
    static constexpr int value = K == 2 ? 3 : (K == 3 ? 2 : K);
};
template <int K>
struct NegUnit {
    static constexpr int value = K == 0 ? 1 : K == 1 ? 0 : K == 2 ? 3 : 2;
};

// forward projector table
template <int MU>
struct Proj;
template <>
struct Proj<0> {  // T
    static constexpr int p0 = 2, c0 = 0, p1 = 3, c1 = 0;
};
template <>
struct Proj<1> {  // X
    static constexpr int p0 = 3, c0 = 2, p1 = 2, c1 = 2;
};
template <>
struct Proj<2> {  // Y
    static constexpr int p0 = 3, c0 = 0, p1 = 2, c1 = 1;
};
template <>
struct Proj<3> {  // Z
    static constexpr int p0 = 2, c0 = 2, p1 = 3, c1 = 3;
};

// One half-spinor channel: acc_a += k U h, acc_p += conj(c) k U h, h = psi_a + c psi_p.
// KREAL: k is real (k.im ignored).  Everything is written as FMA chains.
template <typename R, int A, int PP, int CK, bool DAG, bool KREAL>
__device__ __forceinline__ void hop_channel(Cplx<R> acc[12], const Cplx<R> h[3], const Cplx<R> u[9], Cplx<R> k)
{
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        Cplx<R> s;
        if (!DAG) {
            s = cmul(u[3 * r + 0], h[0]);
            cmac(s, u[3 * r + 1], h[1]);
            cmac(s, u[3 * r + 2], h[2]);
        } else {
            s = cmulc(u[0 * 3 + r], h[0]);
            cmacc(s, u[1 * 3 + r], h[1]);
            cmacc(s, u[2 * 3 + r], h[2]);
        }
        // lower row: acc_p += conj(c) * (k s); conj(c) * s is an exact sign/swap
        const Cplx<R> sp = mul_unit<ConjUnit<CK>::value>(s);
        if (KREAL) {
            acc[3 * A + r].re  = fmad(s.re, k.re, acc[3 * A + r].re);
            acc[3 * A + r].im  = fmad(s.im, k.re, acc[3 * A + r].im);
            acc[3 * PP + r].re = fmad(sp.re, k.re, acc[3 * PP + r].re);
            acc[3 * PP + r].im = fmad(sp.im, k.re, acc[3 * PP + r].im);
        } else {
            cmac(acc[3 * A + r], s, k);
            cmac(acc[3 * PP + r], sp, k);
        }
    }
}

// Projected half spinors of a (decoded) spinor for channel A with partner PP and unit CK.
template <typename R, int A, int PP, int CK>
__device__ __forceinline__ void project(Cplx<R> h[3], const Cplx<R> psi[12])
{
#pragma unroll
    for (int col = 0; col < 3; ++col) h[col] = psi[3 * A + col] + mul_unit<CK>(psi[3 * PP + col]);
}
template <typename R, int MU, bool BACK, bool KREAL>
__device__ __forceinline__ void hop_decoded(Cplx<R> acc[12], const Cplx<R> psi[12], const Cplx<R> u[9], Cplx<R> k)
{
    using T          = Proj<MU>;
    constexpr int c0 = BACK ? NegUnit<T::c0>::value : T::c0;
    constexpr int c1 = BACK ? NegUnit<T::c1>::value : T::c1;
    Cplx<R> h[3];
    project<R, 0, T::p0, c0>(h, psi);
    hop_channel<R, 0, T::p0, c0, BACK, KREAL>(acc, h, u, k);
    project<R, 1, T::p1, c1>(h, psi);
    hop_channel<R, 1, T::p1, c1, BACK, KREAL>(acc, h, u, k);
}

// Phase patterns known at compile time (the common boundary conditions): PH_REAL
// all hop phases real, PH_TCPLX only the T phases complex (antiperiodic time,
// periodic space), PH_ANY decided per launch from HopCoef::real_mask.
// PH_TG (paired-site sweeps only): the field is in the temporal gauge (every T
// link is the identity except the one leaving the last time slice, and the T
// phase sits in the transformation), all hop coefficients are real.
enum PhasePattern : int { PH_REAL = 0, PH_TCPLX = 1, PH_ANY = 2, PH_TG = 3 };

}  // namespace c2q
