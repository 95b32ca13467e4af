// Shared by the k-space kernels (kernels_kspace.cu, kernels_eom.cu, kernels_kspace_vjp.cu): CTA shapes,
// coefficient operands and launches of the symmetry-reduced transform, and the EoM's kernel function.
#pragma once

#include <algorithm>
#include <cmath>

#include "transform.cuh"

using namespace ldga;

namespace {

constexpr int kThreads = 256;
constexpr size_t kSmemBudgetTC = 110 * 1024;   // tensor-path kernels: two CTAs per SM

// CTA shape of a transform kernel: the CUDA-core form's plan (transform.cuh), or 256 threads and two
// CTAs per SM on the tensor path
template <int DIM, int N, bool TC>
constexpr int kThr = TC ? kThreads : TransformPlan<DIM, N>::NT;
template <int DIM, int N, bool TC>
constexpr int kThrOne = TC ? kThreads : TransformPlan<DIM, N>::NT_ONE;
template <int DIM, int N, bool TC>
constexpr int kMinB = TC ? 2 : TransformPlan<DIM, N>::MINB;

// vectors per CTA: the plan's (tensor path: what fits), but batched only when there are more vectors
// than SMs: a short list (the EoM inverse's numax vectors) runs one vector per CTA on as many SMs
template <int DIM, int N>
int pairs_per_cta(int total, bool tc = false) {
    int np = tc ? std::min(16, (int)(kSmemBudgetTC / TransformPlan<DIM, N>::SMEM1)) : TransformPlan<DIM, N>::NP;
    np = std::min(np, std::min((total + 147) / 148, total));
    return std::max(np, 1);
}

template <int DIM, int N>
size_t smem_bytes(int np) {
    return (size_t)np * TransformPlan<DIM, N>::SMEM1;
}

// the tensor-path kernels take T as data: an odd N runs on the instantiation of the even N with its M
constexpr int tc_ns(int n) { return n <= 1 ? 1 : 2 * (n / 2); }

template <int M>
TMat<M> make_T(const ldga_ctx* ctx) {
    TMat<M> T;
    for (int i = 0; i < M * M; ++i) T.t[i] = ctx->Tmat[i];
    return T;
}

template <int N>
CosTab<N> make_cos() {
    CosTab<N> T;
    for (int j = 0; j < CosTab<N>::NC; ++j) T.c[j] = (double)(2.0L * cosl(2.0L * 3.14159265358979323846264338327950288L * j / N));
    return T;
}

// For it = tid, tid + NT, ... < n (n <= KL NT): load(it, raw) for B of them at a time, so that their
// global loads are all in flight, then store(it, raw).
template <int NT, int KL, int B, class Raw, class Load, class Store>
__device__ __forceinline__ void batched(int n, Load&& load, Store&& store) {
#pragma unroll
    for (int k0 = 0; k0 < KL; k0 += B) {
        Raw raw[B];
#pragma unroll
        for (int k = 0; k < B; ++k) {
            const int it = threadIdx.x + (k0 + k) * NT;
            if (k0 + k < KL && it < n) load(it, raw[k]);
        }
#pragma unroll
        for (int k = 0; k < B; ++k) {
            const int it = threadIdx.x + (k0 + k) * NT;
            if (k0 + k < KL && it < n) store(it, raw[k]);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// a9/a10: EoM.  Forward: for one nu_n and a chunk of w, K(q) = eom(...) -> S(K) * Ghat(nu+w),
// summed over the chunk in a fixed order -> partial[chunk][nu][q].  The inverse kernel then sums
// the chunks (fixed order), applies S, and adds 1/beta, the tail and the Hartree term.
// ---------------------------------------------------------------------------------------------
struct EomArgs {
    int nnu, nw, n_iv, n_iw, shift, fft_lo, numax, w_per_chunk;
    int w_begin = 0, w_end = 0;   // the ω range the forward kernel sums ([0, nw) without a shard)
    double U, lam_m, lam_d;
    const double* lam_m_dev;   // device scalars added to lam_m / lam_d (may be null)
    const double* lam_d_dev;
    int part;   // -1: full eom; 0..5: calc_Σ_parts contributions
};

__device__ __forceinline__ double chi_lam(double x, double lam) {
    return lam == 0.0 ? x : x / (lam * x + 1.0);
}

__device__ __forceinline__ double2 eom_value(const EomArgs& a, double2 gm, double2 gd, double xm, double xd,
                                             double2 l0) {
    const double U = a.U;
    switch (a.part) {
        case 0: {  // eom_χ_m = U*(γm*1.5*(U*χm))
            const double f = 1.5 * (U * xm);
            return make_double2(U * (gm.x * f), U * (gm.y * f));
        }
        case 1:    // eom_γ_m = U*(γm*1.5)
            return make_double2(U * (gm.x * 1.5), U * (gm.y * 1.5));
        case 2: {  // eom_χ_d = -U*(γd*0.5*(-U*χd))
            const double f = 0.5 * (-U * xd);
            return make_double2(-U * (gd.x * f), -U * (gd.y * f));
        }
        case 3:    // eom_γ_d = -U*(γd*0.5)
            return make_double2(-U * (gd.x * 0.5), -U * (gd.y * 0.5));
        case 4:    // eom_rest_01 = -U*1.0 + 0im
            return make_double2(-U * 1.0, 0.0);
        case 5:    // eom_rest = U*λ₀
            return make_double2(U * l0.x, U * l0.y);
        default: {
            // eom = U*(γm*1.5*(1+U*χm) - γd*0.5*(1-U*χd) - 1.5 + 0.5 + λ₀), left to right
            const double fm = 1.5 * (1.0 + U * xm);
            const double fd = 0.5 * (1.0 - U * xd);
            double re = gm.x * fm - gd.x * fd;
            double im = gm.y * fm - gd.y * fd;
            re = re - 1.5;
            re = re + 0.5;
            re = re + l0.x;
            im = im + l0.y;
            return make_double2(U * re, U * im);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// host-side dispatch on (DIM, N)
// ---------------------------------------------------------------------------------------------
// one launch of the tensor-path (ktc) or the CUDA-core (kcc) form
template <int DIM, int N, class KTC, class KCC, class... Args>
int launch_form(ldga_ctx* ctx, KTC ktc, KCC kcc, dim3 grid, size_t sm, const char* what, int nt, Args... args) {
    if (ctx->transform_tc) {
        LDGA_CUDA(ctx, set_smem(ctx, ktc, sm));
        ktc<<<grid, kThr<DIM, N, true>, sm, ctx->stream>>>(make_T<N / 2 + 1>(ctx), args...);
    } else {
        LDGA_CUDA(ctx, set_smem(ctx, kcc, sm));
        kcc<<<grid, nt, sm, ctx->stream>>>(make_cos<N>(), args...);
    }
    LDGA_LAUNCHED(ctx, what);
    return LDGA_OK;
}
#define LDGA_FORMS(K) K<DIM, tc_ns(N), true>, K<DIM, N, false>

}  // namespace

#define LDGA_CASE(D, NS)                                  \
    if (ctx->dim == D && ctx->ns == NS) { return BODY(D, NS); }

