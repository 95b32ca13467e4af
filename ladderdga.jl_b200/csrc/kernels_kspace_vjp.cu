// Adjoints of the k-space stages: EoM, bubble and lattice G.
#include "kspace_common.cuh"

namespace {

// ---------------------------------------------------------------------------------------------
// Adjoint of the EoM (calc_Σ, ladderDGATools_singleCore.jl:49-136) for a real loss with upstream
// Sbar[q, n] = dL/dRe Σ + i dL/dIm Σ over the stored (irreducible) values.  The forward is
//   Σ(q, n) = (1/(β N_k²)) S( Σ_ω S(K(·, n, ω)) Ĝ(ν_n + ω) )(q) + tail(n) + Hartree,
// and on symmetric functions the transform satisfies Sᵀ = kMult S kMult⁻¹, so
//   K̄(q, n, ω) = kMult(q)/(β N_k²) S( conj(Ĝ(ν_n + ω)) · S(Sbar(·, n)/kMult) )(q),
// the same transform-product-transform shape as the bubble.  From K = eom(γm, γd, χm^λ, χd^λ, λ₀):
//   γ̄m = 1.5 U (1 + U χm^λ) K̄,  γ̄d = -0.5 U (1 - U χd^λ) K̄,  λ̄₀ = U K̄,
//   χ̄m^λ += Σ_n Re(conj(K̄) 1.5 U² γm),  χ̄d^λ += Σ_n Re(conj(K̄) 0.5 U² γd),
// plus, with the tail correction, χ̄m^λ(q, ω) += s̄ kMult(q)/(β N_k) with s̄ = U Σ Im(Sbar)/ν_n
// (the tail is -U(sum_kω χm^λ - χloc_m_sum)/(iν_n)), and finally χ̄ = χ̄^λ/(λχ + 1)².
// ---------------------------------------------------------------------------------------------
template <int DIM, int N>
__global__ void __launch_bounds__((kThr<DIM, N, false>), (kMinB<DIM, N, false>)) k_vjp_sbar(const CosTab<N> T, int numax, const double* __restrict__ kmult,
                                                       const double2* __restrict__ sbar, double2* __restrict__ shat, int np_max) {
    using S = TransformSmem<DIM, N / 2 + 1>;
    constexpr int NQ = S::NQ;
    extern __shared__ double2 smem[];
    const int p0 = blockIdx.x * np_max;
    const int np = min(np_max, numax - p0);
    double2* bufA = smem;
    double2* bufB = smem + np_max * S::BUF_A;
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        bufA[p * NQ + q] = cscale(sbar[(size_t)(p0 + p) * NQ + q], 1.0 / kmult[q]);
    }
    __syncthreads();
    const double2* res = sym_transform<DIM, N>(np, bufA, bufB, T);
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        const double2 v = res[it];
        shat[(size_t)(p0 + p) * NQ + q] = v;
    }
}

struct EomVjpArgs {
    int nnu, nw, n_iv, n_iw, shift, fft_lo, numax;
    double U, lam_m, lam_d, scale;   // scale = 1/(beta N_k^2)
};

template <int DIM, int N>
__global__ void __launch_bounds__((kThr<DIM, N, false>), (kMinB<DIM, N, false>)) k_eom_vjp(
    const CosTab<N> T, const EomVjpArgs a, const double* __restrict__ kmult, const double2* __restrict__ ghat,
    const double2* __restrict__ shat, const double* __restrict__ chi_m, const double2* __restrict__ gam_m,
    const double* __restrict__ chi_d, const double2* __restrict__ gam_d, double2* __restrict__ gm_bar,
    double2* __restrict__ gd_bar, double2* __restrict__ l0_bar, double* __restrict__ cm, double* __restrict__ cd, int np_max) {
    using S = TransformSmem<DIM, N / 2 + 1>;
    constexpr int NQ = S::NQ;
    extern __shared__ double2 smem[];
    const int total = a.numax * a.nw;
    const int p0 = blockIdx.x * np_max;
    const int np = min(np_max, total - p0);
    double2* bufA = smem;
    double2* bufB = smem + np_max * S::BUF_A;
    __shared__ int s_vi[16];
    if (threadIdx.x < np) {
        const int pi = p0 + threadIdx.x;
        const int wi = pi / a.numax, n = pi - wi * a.numax;
        const int v0 = a.n_iv + a.shift * ((wi - a.n_iw) / 2);          // ν0Index_of_ωIndex - 1
        const int len = min(a.numax, 2 * a.n_iv - v0);
        s_vi[threadIdx.x] = (n < len && v0 + n >= 0) ? v0 + n : -1;
    }
    __syncthreads();
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        const int pi = p0 + p;
        const int wi = pi / a.numax, n = pi - wi * a.numax;
        const int wn = wi - a.n_iw;
        double2 v = make_double2(0.0, 0.0);
        if (s_vi[p] >= 0) v = cmul(shat[(size_t)n * NQ + q], cconj(ghat[(size_t)(n + wn - a.fft_lo) * NQ + q]));
        bufA[p * NQ + q] = v;
    }
    __syncthreads();
    const double2* res = sym_transform<DIM, N>(np, bufA, bufB, T);
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        const double2 v = res[it];
        const int pi = p0 + p;
        const int wi = pi / a.numax, n = pi - wi * a.numax;
        const int vi = s_vi[p];
        const size_t cslot = (size_t)n * NQ * a.nw + (size_t)q + (size_t)NQ * wi;
        if (vi < 0) {
            cm[cslot] = 0.0;
            cd[cslot] = 0.0;
            continue;
        }
        const double2 kb = cscale(v, kmult[q] * a.scale);
        const size_t iq = (size_t)q + (size_t)NQ * wi;
        const size_t iv = (size_t)q + (size_t)NQ * (vi + (size_t)a.nnu * wi);
        const double U = a.U;
        const double xm = chi_lam(chi_m[iq], a.lam_m), xd = chi_lam(chi_d[iq], a.lam_d);
        if (gm_bar) gm_bar[iv] = cscale(kb, 1.5 * U * (1.0 + U * xm));
        if (gd_bar) gd_bar[iv] = cscale(kb, -0.5 * U * (1.0 - U * xd));
        if (l0_bar) l0_bar[iv] = cscale(kb, U);
        const double2 gm = gam_m[iv], gd = gam_d[iv];
        cm[cslot] = 1.5 * U * U * (kb.x * gm.x + kb.y * gm.y);    // Re(conj(kb) gm) 1.5 U^2
        cd[cslot] = 0.5 * U * U * (kb.x * gd.x + kb.y * gd.y);
    }
}

// s̄ = U Σ_{q,n} Im(Sbar(q, n)) / ν_n, one CTA, fixed order: a warp takes whole n, four loads in flight
// (256 threads with a division per element 16 us at 325 q x 20 ν; 5 us)
__global__ void __launch_bounds__(1024) k_vjp_tail(int nq, int numax, double beta, double U,
                                                   const double2* __restrict__ sbar, double* __restrict__ out) {
    __shared__ double red[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double acc = 0.0;
    for (int n = warp; n < numax; n += 32) {
        double s = 0.0;
#pragma unroll 4
        for (int q = lane; q < nq; q += 32) s += sbar[(size_t)n * nq + q].y;
        acc += s / ((2.0 * n + 1.0) * M_PI / beta);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (lane == 0) red[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double r = 0.0;
        for (int i = 0; i < 32; ++i) r += red[i];
        out[0] = U * r;
    }
}

__global__ void __launch_bounds__(256) k_eom_vjp_chi(int nq, int nw, int numax, double lam_m, double lam_d, double tail_w,
                                                      const double* __restrict__ kmult, const double* __restrict__ sb_dev,
                                                      const double* __restrict__ chi_m, const double* __restrict__ chi_d,
                                                      const double* __restrict__ cm, const double* __restrict__ cd,
                                                      double* __restrict__ xm_bar, double* __restrict__ xd_bar) {
    const size_t n_qw = (size_t)nq * nw;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n_qw; e += (size_t)gridDim.x * blockDim.x) {
        const int q = (int)(e % nq);
        double am = 0.0, ad = 0.0;
        for (int n = 0; n < numax; ++n) {
            am += cm[(size_t)n * n_qw + e];
            ad += cd[(size_t)n * n_qw + e];
        }
        if (tail_w != 0.0) am += sb_dev[0] * kmult[q] * tail_w;
        const double fm = lam_m * chi_m[e] + 1.0, fd = lam_d * chi_d[e] + 1.0;
        if (xm_bar) xm_bar[e] = am / (fm * fm);
        if (xd_bar) xd_bar[e] = ad / (fd * fd);
    }
}

// ---------------------------------------------------------------------------------------------
// Adjoint of the lattice G (setup + bubble + the EoM's direct use of Ĝ) -> dL/dΣ_loc.
//   bubble: χ₀(ν, ω) = s_b S(Ĝ(ν) Ĝ(ν+ω)), s_b = -β/N_k²  ->  P̄ = s_b kMult S(χ̄₀/kMult),
//           Ĝ̄(ν) += conj(Ĝ(ν+ω)) P̄,  Ĝ̄(ν+ω) += conj(Ĝ(ν)) P̄          (k_bubble_vjp)
//   EoM:    Σ(n) = c S(Σ_ω K̂(n,ω) Ĝ(ν_n+ω)), K̂ = S(K), c = 1/(β N_k²)
//           ->  Ĝ̄(ν_n+ω) += c kMult Ŝ̄(n) conj(K̂(n,ω)),  Ŝ̄ = S(Σ̄/kMult)   (k_eom_gvjp)
// Each (ν, ω) term writes its contribution to its own scratch row; k_ghat_gather sums, per
// frequency of fft_range, the rows that touch it in a fixed (host-computed) order.  Then
// Ḡ = kMult S(Ĝ̄/kMult) (k_vjp_transform) and, from G = 1/(iν + μ - ε - Σ_loc),
//   Σ̄_loc(m) = Σ_q conj(G²) Ḡ over ν_m,  + Σ_q conj(Ḡ) G² over ν_{-m-1}   (k_sigma_loc_grad).
// ---------------------------------------------------------------------------------------------
template <int DIM, int N>
__global__ void __launch_bounds__((kThr<DIM, N, false>), (kMinB<DIM, N, false>)) k_bubble_vjp(
    const CosTab<N> T, int nnu, int nw, int n_iv, int n_iw, int shift, int fft_lo, double sb,
    const double* __restrict__ kmult, const double2* __restrict__ ghat, const double2* __restrict__ chi0_bar,
    double2* __restrict__ rows, int np_max) {
    using S = TransformSmem<DIM, N / 2 + 1>;
    constexpr int NQ = S::NQ;
    extern __shared__ double2 smem[];
    const int total = nnu * nw;
    const int p0 = blockIdx.x * np_max;
    const int np = min(np_max, total - p0);
    double2* bufA = smem;
    double2* bufB = smem + np_max * S::BUF_A;
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        bufA[p * NQ + q] = cscale(chi0_bar[(size_t)(p0 + p) * NQ + q], 1.0 / kmult[q]);
    }
    __syncthreads();
    const double2* res = sym_transform<DIM, N>(np, bufA, bufB, T);
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        const double2 v = res[it];
        const int pi = p0 + p;
        const int wi = pi / nnu, vi = pi - wi * nnu;
        const int wn = wi - n_iw;
        const int vn = (vi - n_iv) - shift * (wn / 2);
        const double2 pb = cscale(v, sb * kmult[q]);
        const double2 g1 = ghat[(size_t)(vn - fft_lo) * NQ + q], g2 = ghat[(size_t)(vn + wn - fft_lo) * NQ + q];
        rows[(size_t)(2 * pi) * NQ + q] = cmul(cconj(g2), pb);       // -> frequency vn
        rows[(size_t)(2 * pi + 1) * NQ + q] = cmul(cconj(g1), pb);   // -> frequency vn + wn
    }
}

template <int DIM, int N>
__global__ void __launch_bounds__((kThr<DIM, N, false>), (kMinB<DIM, N, false>)) k_eom_gvjp(
    const CosTab<N> T, const EomArgs a, double c, const double* __restrict__ kmult, const double2* __restrict__ shat,
    const double* __restrict__ chi_m, const double2* __restrict__ gam_m, const double* __restrict__ chi_d,
    const double2* __restrict__ gam_d, const double2* __restrict__ lambda0, double2* __restrict__ rows, int np_max) {
    using S = TransformSmem<DIM, N / 2 + 1>;
    constexpr int NQ = S::NQ;
    extern __shared__ double2 smem[];
    const int total = a.numax * a.nw;
    const int p0 = blockIdx.x * np_max;
    const int np = min(np_max, total - p0);
    double2* bufA = smem;
    double2* bufB = smem + np_max * S::BUF_A;
    __shared__ int s_vi[16];
    if (threadIdx.x < np) {
        const int pi = p0 + threadIdx.x;
        const int wi = pi / a.numax, n = pi - wi * a.numax;
        const int v0 = a.n_iv + a.shift * ((wi - a.n_iw) / 2);
        const int len = min(a.numax, 2 * a.n_iv - v0);
        s_vi[threadIdx.x] = (n < len && v0 + n >= 0) ? v0 + n : -1;
    }
    __syncthreads();
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        const int wi = (p0 + p) / a.numax;
        const int vi = s_vi[p];
        double2 K = make_double2(0.0, 0.0);
        if (vi >= 0) {
            const size_t iq = (size_t)q + (size_t)NQ * wi;
            const size_t iv = (size_t)q + (size_t)NQ * (vi + (size_t)a.nnu * wi);
            K = eom_value(a, gam_m[iv], gam_d[iv], chi_lam(chi_m[iq], a.lam_m), chi_lam(chi_d[iq], a.lam_d), lambda0[iv]);
        }
        bufA[p * NQ + q] = K;
    }
    __syncthreads();
    const double2* res = sym_transform<DIM, N>(np, bufA, bufB, T);
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        const double2 v = res[it];
        const int pi = p0 + p;
        const int n = pi - (pi / a.numax) * a.numax;
        double2 r = make_double2(0.0, 0.0);
        if (s_vi[p] >= 0) r = cmul(cscale(shat[(size_t)n * NQ + q], c * kmult[q]), cconj(v));
        rows[(size_t)pi * NQ + q] = r;
    }
}

// out(f) = (mul_kmult ? kMult : 1) S(in(f) / kMult) for nf vectors of the wedge
template <int DIM, int N>
__global__ void __launch_bounds__((kThr<DIM, N, false>), (kMinB<DIM, N, false>)) k_vjp_transform(const CosTab<N> T, int nf, int mul_kmult,
                                                            const double* __restrict__ kmult,
                                                            const double2* __restrict__ in, double2* __restrict__ out, int np_max) {
    using S = TransformSmem<DIM, N / 2 + 1>;
    constexpr int NQ = S::NQ;
    extern __shared__ double2 smem[];
    const int p0 = blockIdx.x * np_max;
    const int np = min(np_max, nf - p0);
    double2* bufA = smem;
    double2* bufB = smem + np_max * S::BUF_A;
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        bufA[p * NQ + q] = cscale(in[(size_t)(p0 + p) * NQ + q], 1.0 / kmult[q]);
    }
    __syncthreads();
    const double2* res = sym_transform<DIM, N>(np, bufA, bufB, T);
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        const double2 v = res[it];
        out[(size_t)(p0 + p) * NQ + q] = mul_kmult ? cscale(v, kmult[q]) : v;
    }
}

// Ĝ̄[f][q] = Σ_{j in list(f)} rows[idx[j]][q], CSR over the fft_range frequencies: 32 q x 8 slices of the list per
// CTA, eight rows of a slice in flight, the slices added in order (one thread per (f, q) walked its whole list
// of up to about 120 rows: 49 us at 2D 48^2, Nν = 40, 41 ω; 8 us)
__global__ void __launch_bounds__(256) k_ghat_gather(int nq, const int32_t* __restrict__ start,
                                                      const int32_t* __restrict__ idx, const double2* __restrict__ rows,
                                                      double2* __restrict__ gbar) {
    __shared__ double2 red[8][32];
    const int tx = threadIdx.x & 31, sl = threadIdx.x >> 5, q = blockIdx.x * 32 + tx, f = blockIdx.y;
    const int j0 = start[f], j1 = start[f + 1];
    double2 acc = make_double2(0.0, 0.0);
    if (q < nq)
        for (int j = j0 + sl; j < j1; j += 64) {
            double2 r[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
                r[k] = j + 8 * k < j1 ? rows[(size_t)idx[j + 8 * k] * nq + q] : make_double2(0.0, 0.0);
#pragma unroll
            for (int k = 0; k < 8; ++k) acc = cadd(acc, r[k]);
        }
    red[sl][tx] = acc;
    __syncthreads();
    if (sl == 0 && q < nq) {
        for (int k = 1; k < 8; ++k) acc = cadd(acc, red[k][tx]);
        gbar[(size_t)f * nq + q] = acc;
    }
}

// Σ̄_loc(m), m = 0..n_sigma-1: one CTA per m, fixed-order block reduction over q
__global__ void __launch_bounds__(256) k_sigma_loc_grad(int nq, int nf, int fft_lo, int n_sigma,
                                                         const double2* __restrict__ gloc, const double2* __restrict__ gbar,
                                                         double2* __restrict__ out) {
    __shared__ double2 red[8];
    const int m = blockIdx.x;
    if (m >= n_sigma) return;
    double2 acc = make_double2(0.0, 0.0);
    const int fp = m - fft_lo, fn = -m - 1 - fft_lo;   // columns of ν_m and ν_{-m-1}
    for (int q = threadIdx.x; q < nq; q += blockDim.x) {
        if (fp >= 0 && fp < nf) {
            const double2 g = gloc[(size_t)fp * nq + q];
            acc = cadd(acc, cmul(cconj(cmul(g, g)), gbar[(size_t)fp * nq + q]));
        }
        if (fn >= 0 && fn < nf) {
            const double2 g = gloc[(size_t)fn * nq + q];
            acc = cadd(acc, cmul(cconj(gbar[(size_t)fn * nq + q]), cmul(g, g)));
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        acc.x += __shfl_down_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_down_sync(0xffffffffu, acc.y, o);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double2 r = make_double2(0.0, 0.0);
        for (int i = 0; i < 8; ++i) r = cadd(r, red[i]);
        out[m] = r;
    }
}

template <int DIM, int N>
int run_gloc_vjp(ldga_ctx* ctx, const double2* chi0_bar, const double2* sbar, int numax, double lam_m, double lam_d,
                 double2* shat, double2* rows, const int32_t* start, const int32_t* idx, double2* gbar_hat,
                 double2* gbar) {
    const int nbub = chi0_bar ? ctx->Nnu * ctx->Nw : 0;
    if (chi0_bar) {
        const int np = pairs_per_cta<DIM, N>(nbub);
        const size_t sm = smem_bytes<DIM, N>(np);
        auto kern = k_bubble_vjp<DIM, N>;
        LDGA_CUDA(ctx, set_smem(ctx, kern, sm));
        dim3 grid((nbub + np - 1) / np);
        const double sb = -ctx->mp.beta / ((double)ctx->Nk * (double)ctx->Nk);
        kern<<<grid, kThr<DIM, N, false>, sm, ctx->stream>>>(make_cos<N>(), ctx->Nnu, ctx->Nw, ctx->sp.n_iv, ctx->sp.n_iw,
                                                   ctx->sp.shift, ctx->fft_lo, sb, ctx->d_kmult, ctx->d_ghat, chi0_bar,
                                                   rows, np);
        LDGA_LAUNCHED(ctx, "k_bubble_vjp");
    }
    if (sbar) {
        {
            const int np = pairs_per_cta<DIM, N>(numax);
            const size_t sm = smem_bytes<DIM, N>(np);
            auto kern = k_vjp_transform<DIM, N>;
            LDGA_CUDA(ctx, set_smem(ctx, kern, sm));
            dim3 grid((numax + np - 1) / np);
            kern<<<grid, kThr<DIM, N, false>, sm, ctx->stream>>>(make_cos<N>(), numax, 0, ctx->d_kmult, sbar, shat, np);
            LDGA_LAUNCHED(ctx, "k_vjp_transform");
        }
        const int total = numax * ctx->Nw;
        const int np = pairs_per_cta<DIM, N>(total);
        const size_t sm = smem_bytes<DIM, N>(np);
        auto kern = k_eom_gvjp<DIM, N>;
        LDGA_CUDA(ctx, set_smem(ctx, kern, sm));
        EomArgs a;
        a.nnu = ctx->Nnu; a.nw = ctx->Nw; a.n_iv = ctx->sp.n_iv; a.n_iw = ctx->sp.n_iw; a.shift = ctx->sp.shift;
        a.fft_lo = ctx->fft_lo; a.numax = numax; a.w_per_chunk = 1;
        a.U = ctx->mp.U; a.lam_m = lam_m; a.lam_d = lam_d; a.part = -1;
        a.lam_m_dev = nullptr; a.lam_d_dev = nullptr;
        dim3 grid((total + np - 1) / np);
        const double c = 1.0 / (ctx->mp.beta * (double)ctx->Nk * (double)ctx->Nk);
        kern<<<grid, kThr<DIM, N, false>, sm, ctx->stream>>>(make_cos<N>(), a, c, ctx->d_kmult, shat, ctx->d_chi[0], ctx->d_gam[0],
                                                   ctx->d_chi[1], ctx->d_gam[1], ctx->d_lambda0,
                                                   rows + (size_t)2 * nbub * ctx->Nq, np);
        LDGA_LAUNCHED(ctx, "k_eom_gvjp");
    }
    k_ghat_gather<<<dim3((ctx->Nq + 31) / 32, ctx->Nf), 256, 0, ctx->stream>>>(ctx->Nq, start, idx, rows, gbar_hat);
    LDGA_LAUNCHED(ctx, "k_ghat_gather");
    {
        const int np = pairs_per_cta<DIM, N>(ctx->Nf);
        const size_t sm = smem_bytes<DIM, N>(np);
        auto kern = k_vjp_transform<DIM, N>;
        LDGA_CUDA(ctx, set_smem(ctx, kern, sm));
        dim3 grid((ctx->Nf + np - 1) / np);
        kern<<<grid, kThr<DIM, N, false>, sm, ctx->stream>>>(make_cos<N>(), ctx->Nf, 1, ctx->d_kmult, gbar_hat, gbar, np);
        LDGA_LAUNCHED(ctx, "k_vjp_transform");
    }
    return LDGA_OK;
}

template <int DIM, int N>
int run_eom_vjp(ldga_ctx* ctx, int numax, double lam_m, double lam_d, int tc, const double2* sbar,
                double2* gm_bar, double2* gd_bar, double2* l0_bar, double* xm_bar, double* xd_bar, double2* shat,
                double* cm, double* cd) {
    {   // Ŝbar = S(Sbar / kMult)
        const int np = pairs_per_cta<DIM, N>(numax);
        const size_t sm = smem_bytes<DIM, N>(np);
        auto kern = k_vjp_sbar<DIM, N>;
        LDGA_CUDA(ctx, set_smem(ctx, kern, sm));
        dim3 grid((numax + np - 1) / np);
        kern<<<grid, kThr<DIM, N, false>, sm, ctx->stream>>>(make_cos<N>(), numax, ctx->d_kmult, sbar, shat, np);
        LDGA_LAUNCHED(ctx, "k_vjp_sbar");
    }
    {
        const int total = numax * ctx->Nw;
        const int np = pairs_per_cta<DIM, N>(total);
        const size_t sm = smem_bytes<DIM, N>(np);
        auto kern = k_eom_vjp<DIM, N>;
        LDGA_CUDA(ctx, set_smem(ctx, kern, sm));
        EomVjpArgs a;
        a.nnu = ctx->Nnu; a.nw = ctx->Nw; a.n_iv = ctx->sp.n_iv; a.n_iw = ctx->sp.n_iw; a.shift = ctx->sp.shift;
        a.fft_lo = ctx->fft_lo; a.numax = numax; a.U = ctx->mp.U; a.lam_m = lam_m; a.lam_d = lam_d;
        a.scale = 1.0 / (ctx->mp.beta * (double)ctx->Nk * (double)ctx->Nk);
        dim3 grid((total + np - 1) / np);
        kern<<<grid, kThr<DIM, N, false>, sm, ctx->stream>>>(make_cos<N>(), a, ctx->d_kmult, ctx->d_ghat, shat, ctx->d_chi[0],
                                                   ctx->d_gam[0], ctx->d_chi[1], ctx->d_gam[1], gm_bar, gd_bar, l0_bar,
                                                   cm, cd, np);
        LDGA_LAUNCHED(ctx, "k_eom_vjp");
    }
    if (tc) {
        k_vjp_tail<<<1, 1024, 0, ctx->stream>>>(ctx->Nq, numax, ctx->mp.beta, ctx->mp.U, sbar, ctx->d_red + 60);
        LDGA_LAUNCHED(ctx, "k_vjp_tail");
    }
    const double tail_w = tc ? 1.0 / (ctx->mp.beta * (double)ctx->Nk) : 0.0;
    k_eom_vjp_chi<<<2 * 148, 256, 0, ctx->stream>>>(ctx->Nq, ctx->Nw, numax, lam_m, lam_d, tail_w, ctx->d_kmult,
                                                    ctx->d_red + 60, ctx->d_chi[0], ctx->d_chi[1], cm, cd, xm_bar,
                                                    xd_bar);
    LDGA_LAUNCHED(ctx, "k_eom_vjp_chi");
    return LDGA_OK;
}

}  // namespace

int launch_eom_vjp(ldga_ctx* ctx, int numax, double lam_m, double lam_d, int tc, const double2* sbar,
                   double2* gm_bar, double2* gd_bar, double2* l0_bar, double* xm_bar, double* xd_bar, double2* shat,
                   double* cm, double* cd) {
#define BODY(D, NS) run_eom_vjp<D, NS>(ctx, numax, lam_m, lam_d, tc, sbar, gm_bar, gd_bar, l0_bar, xm_bar, xd_bar, shat, cm, cd)
    LDGA_FOR_EACH_GRID(LDGA_CASE)
#undef BODY
    return ctx_fail(ctx, LDGA_ERR_ARG, "unsupported k-grid size");
}

int launch_gloc_vjp(ldga_ctx* ctx, const double2* chi0_bar, const double2* sbar, int numax, double lam_m,
                    double lam_d, double2* shat, double2* rows, const int32_t* start, const int32_t* idx,
                    double2* gbar_hat, double2* gbar) {
#define BODY(D, NS) run_gloc_vjp<D, NS>(ctx, chi0_bar, sbar, numax, lam_m, lam_d, shat, rows, start, idx, gbar_hat, gbar)
    LDGA_FOR_EACH_GRID(LDGA_CASE)
#undef BODY
    return ctx_fail(ctx, LDGA_ERR_ARG, "unsupported k-grid size");
}

int launch_sigma_loc_grad(ldga_ctx* ctx, const double2* gbar, int n_sigma, double2* out) {
    k_sigma_loc_grad<<<n_sigma, 256, 0, ctx->stream>>>(ctx->Nq, ctx->Nf, ctx->fft_lo, n_sigma, ctx->d_gloc, gbar, out);
    LDGA_LAUNCHED(ctx, "k_sigma_loc_grad");
    return LDGA_OK;
}
