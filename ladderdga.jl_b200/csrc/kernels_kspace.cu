// k-space kernels: the lattice G and its transform (setup) and the bubble chi0, on the symmetry-reduced
// transform of transform.cuh; one CTA processes a batch of independent (nu, w) vectors entirely in
// shared memory.
#include "kspace_common.cuh"

namespace {

// ---------------------------------------------------------------------------------------------
// a1: G(k, nu) for nu in fft_range and Ghat = S(G)
// ---------------------------------------------------------------------------------------------
template <int DIM, int N, bool TC>
__global__ void __launch_bounds__((kThr<DIM, N, TC>), (kMinB<DIM, N, TC>)) k_gloc_transform(
    const TransformCoef<N, TC> T, int nf, int fft_lo, double beta, double mu, const double* __restrict__ eps,
    const double2* __restrict__ sigma_loc, int n_sigma, double2* __restrict__ gloc, int from_sigma,
    double2* __restrict__ ghat, int np_max) {
    using S = TransformSmem<DIM, N / 2 + 1>;
    constexpr int NQ = S::NQ;
    extern __shared__ double2 smem[];
    const int p0 = blockIdx.x * np_max;
    const int np = min(np_max, nf - p0);
    double2* bufA = smem;
    double2* bufB = smem + np_max * S::BUF_A;
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        const int f = p0 + p;
        double2 g;
        if (from_sigma) {
            const int vn = fft_lo + f;
            const double2 s = vn < 0 ? cconj(sigma_loc[-vn - 1]) : sigma_loc[vn];
            const double2 z = make_double2(mu - eps[q] - s.x, (2.0 * vn + 1.0) * M_PI / beta - s.y);
            g = cinv(z);
            gloc[(size_t)f * NQ + q] = g;
        } else {
            g = gloc[(size_t)f * NQ + q];
        }
        bufA[p * NQ + q] = g;
    }
    __syncthreads();
    const double2* res = sym_transform_any<DIM, N, TC>(np, bufA, bufB, T);
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        ghat[(size_t)(p0 + p) * NQ + q] = res[it];
    }
}

// ---------------------------------------------------------------------------------------------
// a2: chi0[q, nu, w] = -beta/N_k^2 S(Ghat(nu) Ghat(nu+w))(q)
// G(k, -nu) = conj(G(k, nu)) (nu_n -> nu_{-n-1}) and G is even in k, so
//   chi0(q, nu'', w) = conj(chi0(q, nu, w)),  nu'' = -nu - w - 1,
// and a pair whose partner lies in the box is computed once: `pairs` lists the representatives
// (pair index vi + Nnu wi, partner's index or -1), built on the host with the handle.
// The scale goes onto the product before the transform (one multiplication per input either way, equally accurate:
// 4e-16).  Which of two such roundings is taken decides where the lambda_m Newton of the 3D 32^3 test input, which
// steps into a region of poles, ends: after the transform, tests of that root and of lambda_dm fail
// with every array at its parity tolerance.
// Measured, cold caches: 3D 32^3, Nnu = 40, Nw = 41 (1040 vectors) 35 us, 72 us with the unfolded
// matrix at two threads per column; 2D 64^2, Nnu = 60, Nw = 61 (2310 vectors) 25 us, 108 us before.
// ---------------------------------------------------------------------------------------------
template <int DIM, int N, bool TC>
__global__ void __launch_bounds__((kThr<DIM, N, TC>), (kMinB<DIM, N, TC>)) k_bubble(
    const TransformCoef<N, TC> T, int nnu, int nw, int n_iv, int n_iw, int shift, int fft_lo, double scale,
    const double2* __restrict__ ghat, const int2* __restrict__ pairs, int total, double2* __restrict__ chi0, int np_max) {
    using S = TransformSmem<DIM, N / 2 + 1>;
    constexpr int NQ = S::NQ;
    extern __shared__ double2 smem[];
    const int p0 = blockIdx.x * np_max;
    const int np = min(np_max, total - p0);
    double2* bufA = smem;
    double2* bufB = smem + np_max * S::BUF_A;
    __shared__ int2 s_f[16], s_pp[16];     // frequencies of the two factors; the pair and its partner
    if (threadIdx.x < np) {
        const int2 pp = pairs[p0 + threadIdx.x];
        const int pi = pp.x;
        s_pp[threadIdx.x] = pp;
        const int wi = pi / nnu, vi = pi - wi * nnu;
        const int wn = wi - n_iw;
        const int vn = (vi - n_iv) - shift * (wn / 2);    // C division truncates like trunc(Int, .)
        s_f[threadIdx.x] = make_int2(vn - fft_lo, vn + wn - fft_lo);
    }
    __syncthreads();
    struct Raw { double2 a, b; };
    constexpr int NT = kThr<DIM, N, TC>, NPM = TC ? 16 : TransformPlan<DIM, N>::NP;
    batched<NT, (NPM * NQ + NT - 1) / NT, 4, Raw>(
        np * NQ,
        [&](int it, Raw& r) {
            const int p = it / NQ, q = it - p * NQ;
            r.a = ghat[(size_t)s_f[p].x * NQ + q];
            r.b = ghat[(size_t)s_f[p].y * NQ + q];
        },
        [&](int it, const Raw& r) { bufA[it] = cscale(cmul(r.a, r.b), scale); });
    __syncthreads();
    const double2* res = sym_transform_any<DIM, N, TC>(np, bufA, bufB, T);
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        const int2 pp = s_pp[p];
        const double2 c = res[it];
        chi0[(size_t)pp.x * NQ + q] = c;
        if (pp.y >= 0) chi0[(size_t)pp.y * NQ + q] = cconj(c);
    }
}

template <int DIM, int N>
int run_gloc(ldga_ctx* ctx, bool from_sigma) {
    const int np = pairs_per_cta<DIM, N>(ctx->Nf, ctx->transform_tc);
    StageTimer st_(ctx, LDGA_STAGE_GLOC);
    return launch_form<DIM, N>(ctx, LDGA_FORMS(k_gloc_transform), dim3((ctx->Nf + np - 1) / np), smem_bytes<DIM, N>(np), "k_gloc_transform", kThr<DIM, N, false>,
                               ctx->Nf, ctx->fft_lo, ctx->mp.beta, ctx->mp.mu, ctx->d_eps, ctx->d_sigma_loc,
                               ctx->n_sigma_loc, ctx->d_gloc, from_sigma ? 1 : 0, ctx->d_ghat, np);
}

template <int DIM, int N>
int run_bubble(ldga_ctx* ctx) {
    // an ω shard takes the pairs of its frequencies: a contiguous range of the ω-major list
    const int first = ctx->bub_pair_w_start[ctx->w_lo];
    const int total = ctx->bub_pair_w_start[ctx->w_hi] - first;
    if (total <= 0) return LDGA_OK;
    const int np = pairs_per_cta<DIM, N>(total, ctx->transform_tc);
    const double scale = -ctx->mp.beta / ((double)ctx->Nk * (double)ctx->Nk);
    StageTimer st_(ctx, LDGA_STAGE_BUBBLE);
    return launch_form<DIM, N>(ctx, LDGA_FORMS(k_bubble), dim3((total + np - 1) / np), smem_bytes<DIM, N>(np), "k_bubble", kThr<DIM, N, false>, ctx->Nnu,
                               ctx->Nw, ctx->sp.n_iv, ctx->sp.n_iw, ctx->sp.shift, ctx->fft_lo, scale, ctx->d_ghat,
                               ctx->d_bub_pairs + first, total, ctx->d_chi0, np);
}

}  // namespace

int launch_gloc_transform(ldga_ctx* ctx, bool from_sigma) {
#define BODY(D, NS) run_gloc<D, NS>(ctx, from_sigma)
    LDGA_FOR_EACH_GRID(LDGA_CASE)
#undef BODY
    return ctx_fail(ctx, LDGA_ERR_ARG, "unsupported k-grid size");
}

int launch_bubble(ldga_ctx* ctx) {
    ++ctx->chi0_gen;
#define BODY(D, NS) run_bubble<D, NS>(ctx)
    LDGA_FOR_EACH_GRID(LDGA_CASE)
#undef BODY
    return ctx_fail(ctx, LDGA_ERR_ARG, "unsupported k-grid size");
}

