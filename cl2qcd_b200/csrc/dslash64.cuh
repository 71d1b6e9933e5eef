// dslash64.cuh -- the FP64 sweep: the hopping term of dslash.cuh on one output
// parity, one thread per site, with the fused epilogues and reductions.
//
// Bound by HBM: 8 links of 144 bytes, the neighbours through L2 and the output, 1536
// bytes a site, at 94 % of the measured copy rate on 24^3x48.  The vector updates of the
// CG and BiCGStab's (t, s) ride along where their operands are at hand (DOT_XUPD,
// DOT_CGR, DOT_OX, DOT_RES), each saving the passes of its own kernel over p, v, x and r.
// (In the temporal gauge, with a fifth fewer bytes, the sweep was no faster: 97 us
// against 83 us; prefetching the next direction's links to L2 did not change that.)
#pragma once

#include "dslash.cuh"

namespace c2q {

// <out, x> and |out|^2 with the EPI_AXPY operand x, from registers: BiCGStab's
// (t, s) and (t, t) for t = A s.
constexpr int DOT_OX = 5;
// out = y - (EPI_AXPY result) with |out|^2: the true residual b - A x, y = b.
constexpr int DOT_RES = 6;

struct Dslash64Params {
    SpinorPtr<64> out;
    SpinorPtr<64> in;   // opposite-parity input field
    SpinorPtr<64> x;    // EPI_AXPY: same-parity field multiplied by M_diag; DOT_XUPD: the search direction
    SpinorPtr<64> y;    // DOT_Y partner (same parity as out); DOT_CGR: the residual; DOT_XUPD: the solution
    const void* gauge;  // [parity][mu][lane][stride]
    Geom g;
    HopCoef c;
    EpiArgs e;
    int out_parity;         // parity of the output sites: 0 = (x+y+z+t) even
    RedArgs red;            // red.sc: alpha of the fused CG updates
    int pdl;                // launched as a dependent launch (launch_dep)
};

// One hop: load the neighbour spinor and the link, weight by the hop phase.
template <int NL, int MU, bool BACK>
__device__ __forceinline__ void hop_fp64(Cplx<double> acc[12], const Dslash64Params& prm, size_t link_idx, int i_nb)
{
    const Geom& g    = prm.g;
    const int d      = BACK ? 1 : 0;
    const int lpar   = BACK ? 1 - prm.out_parity : prm.out_parity;
    const char* base = static_cast<const char*>(prm.gauge) + (size_t)((lpar * 4 + MU) * NL) * g.stride * 16;
    Cplx<double> psi[12];
    SpinorIO<64>::load(prm.in, g.stride, i_nb, psi);
    Cplx<double> u[9];
    LinkIO<64, NL>::load(base, (size_t)g.stride, link_idx, u);
    if (NL == 6) reconstruct_row2(u);
    const Cplx<double> k = cmk(prm.c.re[MU][d], prm.c.im[MU][d]);
    if ((prm.c.real_mask >> (2 * MU + d)) & 1u)
        hop_decoded<double, MU, BACK, true>(acc, psi, u, k);
    else
        hop_decoded<double, MU, BACK, false>(acc, psi, u, k);
}

template <int NL, int MU>
__device__ __forceinline__ void direction_fp64(Cplx<double> acc[12], const Dslash64Params& prm, int i_fwd, int i_bwd,
                                               int i_site)
{
    hop_fp64<NL, MU, false>(acc, prm, (size_t)i_site, i_fwd);  // U_mu(x) psi(x+mu)
    hop_fp64<NL, MU, true>(acc, prm, (size_t)i_bwd, i_bwd);    // U_mu(x-mu)^dagger psi(x-mu)
}

template <int NL, int EPI, int DOT>
__global__ void __launch_bounds__(128) dslash64_kernel(const Dslash64Params prm)
{
    static_assert(DOT != DOT_XUPD || EPI != EPI_AXPY, "the solution update shares the EPI_AXPY operand");
    static_assert(DOT != DOT_CGR || EPI == EPI_AXPY, "the residual update follows EPI_AXPY");
    pdl_enter();
    if (halted(prm.red)) return;  // a stopped device-driven solve: every block leaves
    using C       = Cplx<double>;
    const Geom& g = prm.g;
    const int i   = blockIdx.x * blockDim.x + threadIdx.x;
    double dv[4]  = {0.0, 0.0, 0.0, 0.0};

    if (i < g.seo) {
        // coordinates of the output site carrying eo index i
        int rest     = i / g.nsh;
        const int xh = i - rest * g.nsh;
        const int y  = rest % g.ns;
        rest /= g.ns;
        const int z   = rest % g.ns;
        const int t   = rest / g.ns;
        const int x   = 2 * xh + ((prm.out_parity + y + z + t) & 1);
        const int yzt = g.nsh * (y + g.ns * (z + g.ns * t));

        C acc[12];
#pragma unroll
        for (int k = 0; k < 12; ++k) acc[k] = cmk(0.0, 0.0);

        {  // T
            const int tp = t + 1 == g.nt ? 0 : t + 1, tm = t == 0 ? g.nt - 1 : t - 1;
            const int base = xh + g.nsh * (y + g.ns * z);
            direction_fp64<NL, 0>(acc, prm, base + g.vs_h * tp, base + g.vs_h * tm, i);
        }
        {  // X
            const int xp = x + 1 == g.ns ? 0 : x + 1, xm = x == 0 ? g.ns - 1 : x - 1;
            direction_fp64<NL, 1>(acc, prm, (xp >> 1) + yzt, (xm >> 1) + yzt, i);
        }
        {  // Y
            const int yp = y + 1 == g.ns ? 0 : y + 1, ym = y == 0 ? g.ns - 1 : y - 1;
            const int zt = g.ns * (z + g.ns * t);
            direction_fp64<NL, 2>(acc, prm, xh + g.nsh * (yp + zt), xh + g.nsh * (ym + zt), i);
        }
        {  // Z
            const int zp = z + 1 == g.ns ? 0 : z + 1, zm = z == 0 ? g.ns - 1 : z - 1;
            direction_fp64<NL, 3>(acc, prm, xh + g.nsh * (y + g.ns * (zp + g.ns * t)),
                                      xh + g.nsh * (y + g.ns * (zm + g.ns * t)), i);
        }

        // the hopping sum is h = scale * acc (scale = -kappa)
        const double sc = prm.c.scale;
        if (EPI == EPI_PLAIN) {
#pragma unroll
            for (int k = 0; k < 12; ++k) acc[k] = cmk(sc * acc[k].re, sc * acc[k].im);
        } else if (EPI == EPI_DIAG) {
            const C f1 = cmk(prm.e.f1re * sc, prm.e.f1im * sc);
            const C f2 = cmk(prm.e.f2re * sc, prm.e.f2im * sc);
#pragma unroll
            for (int k = 0; k < 12; ++k) acc[k] = cmul(k < 6 ? f1 : f2, acc[k]);
        } else if (EPI == EPI_AXPY) {
            C xv[12];
            SpinorIO<64>::load(prm.x, g.stride, i, xv);
            const C f1 = cmk(prm.e.f1re, prm.e.f1im), f2 = cmk(prm.e.f2re, prm.e.f2im);
#pragma unroll
            for (int k = 0; k < 12; ++k) {
                const C m = cmul(k < 6 ? f1 : f2, xv[k]);
                C r       = cmk(m.re - sc * acc[k].re, m.im - sc * acc[k].im);
                if (prm.e.gamma5 && k >= 6) r = cmk(-r.re, -r.im);
                acc[k] = r;
                if (DOT == DOT_OX) {
                    const C p = cmulc(r, xv[k]), q = cmulc(r, r);
                    dv[0] += p.re;
                    dv[1] += p.im;
                    dv[2] += q.re;
                    dv[3] += q.im;
                }
            }
        }
        if (DOT == DOT_RES) {
            C yv[12];
            SpinorIO<64>::load(prm.y, g.stride, i, yv);
#pragma unroll
            for (int k = 0; k < 12; ++k) {
                acc[k] = yv[k] - acc[k];
                dv[0] += acc[k].re * acc[k].re + acc[k].im * acc[k].im;
            }
        }
        if (DOT != DOT_CGR) SpinorIO<64>::store(prm.out, g.stride, i, acc);

        if (DOT == DOT_Y) {
            C yv[12];
            SpinorIO<64>::load(prm.y, g.stride, i, yv);
#pragma unroll
            for (int k = 0; k < 12; ++k) {
                const C p = cmulc(yv[k], acc[k]);
                dv[0] += p.re;
                dv[1] += p.im;
            }
        } else if (DOT == DOT_SELF) {
#pragma unroll
            for (int k = 0; k < 12; ++k) dv[0] += acc[k].re * acc[k].re + acc[k].im * acc[k].im;
        } else if (DOT == DOT_CGR) {  // r -= alpha out, |r|^2
            const C al = cmk(prm.red.sc->alpha[0], prm.red.sc->alpha[1]);
            C rv[12];
            SpinorIO<64>::load(prm.y, g.stride, i, rv);
#pragma unroll
            for (int k = 0; k < 12; ++k) {
                rv[k] = rv[k] - cmul(acc[k], al);
                dv[0] += rv[k].re * rv[k].re + rv[k].im * rv[k].im;
            }
            SpinorIO<64>::store(prm.y, g.stride, i, rv);
        } else if (DOT == DOT_XUPD) {  // x += alpha p
            const C al = cmk(prm.red.sc->alpha[0], prm.red.sc->alpha[1]);
            C pv[12], xv[12];
            SpinorIO<64>::load(prm.x, g.stride, i, pv);
            SpinorIO<64>::load(prm.y, g.stride, i, xv);
#pragma unroll
            for (int k = 0; k < 12; ++k) cmac(xv[k], al, pv[k]);
            SpinorIO<64>::store(prm.y, g.stride, i, xv);
        }
    }
    if (DOT == DOT_OX) {
        __shared__ double smem4[4 * 32];
        block_sum<4>(dv, smem4);
        finish_reduction<4>(dv, prm.red, smem4);
    } else if (DOT != DOT_NONE && DOT != DOT_XUPD) {
        __shared__ double smem[2 * 32];
        block_sum<2>(dv, smem);
        finish_reduction<2>(dv, prm.red, smem);
    }
}

}  // namespace c2q
