// The equation of motion: forward (K, its transform, the product with G and the sum over w) and inverse.
#include "kspace_common.cuh"

namespace {

// Forward.  Bound by the latency of a step's loads (64 bytes per wedge point) and of the transform's
// barriers; two to eight CTAs per SM overlap them, every load of a thread's points is in flight at once,
// and the operands of the product and the running sum are read and written as whole columns.
// Measured, cold caches: 3D 32^3, 20 nu x 41 w 41 us (72 us before: one 512-thread CTA per SM, two
// threads per column); 2D 64^2, 22 nu x 61 w 30 us (100 us before).
template <int DIM, int N, bool TC>
__global__ void __launch_bounds__((kThr<DIM, N, TC>), (kMinB<DIM, N, TC>)) k_eom_forward(
    const TransformCoef<N, TC> T, const EomArgs a, const double2* __restrict__ ghat, const double* __restrict__ chi_m,
    const double2* __restrict__ gam_m, const double* __restrict__ chi_d, const double2* __restrict__ gam_d,
    const double2* __restrict__ lambda0, double2* __restrict__ partial, int np_max) {
    using S = TransformSmem<DIM, N / 2 + 1>;
    constexpr int NQ = S::NQ;
    constexpr int NT = kThr<DIM, N, TC>, NPM = TC ? 16 : TransformPlan<DIM, N>::NP;
    struct Raw { double2 gm, gd, l0; double xm, xd; };
    extern __shared__ double2 smem[];
    const int chunk = blockIdx.x, nu_n = blockIdx.y;
    const int c0 = a.w_begin + chunk * a.w_per_chunk, c1 = min(c0 + a.w_per_chunk, a.w_end);
    double2* bufA = smem;
    double2* bufB = smem + np_max * S::BUF_A;
    double2* sum = bufB + np_max * S::BUF_B;   // [NQ], between the steps of a CTA with several
    __shared__ int s_vi[16];
    const double lm = a.lam_m + (a.lam_m_dev ? a.lam_m_dev[0] : 0.0);
    const double ld = a.lam_d + (a.lam_d_dev ? a.lam_d_dev[0] : 0.0);
    for (int w0 = c0; w0 < c1; w0 += np_max) {
        const int np = min(np_max, c1 - w0);
        if (threadIdx.x < np) {
            const int wi = w0 + threadIdx.x;
            const int v0 = a.n_iv + a.shift * ((wi - a.n_iw) / 2);          // ν0Index_of_ωIndex - 1
            const int len = min(a.numax, 2 * a.n_iv - v0);
            s_vi[threadIdx.x] = (nu_n < len && v0 + nu_n >= 0) ? v0 + nu_n : -1;
        }
        __syncthreads();   // also: the previous step's reads of the buffers are complete
        batched<NT, (NPM * NQ + NT - 1) / NT, (N > 32 ? 2 : 3), Raw>(
            np * NQ,
            [&](int it, Raw& r) {
                const int p = it / NQ, q = it - p * NQ, wi = w0 + p, vi = max(s_vi[p], 0);
                const size_t iq = (size_t)q + (size_t)NQ * wi;
                const size_t iv = (size_t)q + (size_t)NQ * (vi + (size_t)a.nnu * wi);
                r.gm = gam_m[iv];
                r.gd = gam_d[iv];
                r.l0 = lambda0[iv];
                r.xm = chi_m[iq];
                r.xd = chi_d[iq];
            },
            [&](int it, const Raw& r) {
                bufA[it] = s_vi[it / NQ] < 0 ? make_double2(0.0, 0.0)
                                             : eom_value(a, r.gm, r.gd, chi_lam(r.xm, lm), chi_lam(r.xd, ld), r.l0);
            });
        __syncthreads();
        const double2* res = sym_transform_any<DIM, N, TC>(np, bufA, bufB, T);
        const bool last = w0 + np_max >= c1;
        for (int q = threadIdx.x; q < NQ; q += blockDim.x) {
            double2 acc = w0 == c0 ? make_double2(0.0, 0.0) : sum[q];
            for (int p = 0; p < np; ++p)
                if (s_vi[p] >= 0)
                    acc = cadd(acc, cmul(res[p * NQ + q], ghat[(size_t)(nu_n + w0 + p - a.n_iw - a.fft_lo) * NQ + q]));
            if (last) partial[((size_t)chunk * a.numax + nu_n) * NQ + q] = acc;
            else sum[q] = acc;
        }
        __syncthreads();
    }
}

// Inverse: numax vectors, one per CTA, so a CTA has its SM alone and takes the threads that stage y has
// columns for.  Measured: 3D 32^3, 20 nu 12 us (24 before), 2D 64^2, 22 nu 10 us (23 before).
template <int DIM, int N, bool TC>
__global__ void __launch_bounds__((kThrOne<DIM, N, TC>), 1) k_eom_inverse(
    const TransformCoef<N, TC> T, int numax, int nchunk, double scale, double beta, double U, double hartree,
    const double* __restrict__ tail_sum, int tc, double chiloc_m_sum, const double2* __restrict__ partial,
    double2* __restrict__ out, int out_ld, int add_hartree, int np_max) {
    using S = TransformSmem<DIM, N / 2 + 1>;
    constexpr int NQ = S::NQ;
    extern __shared__ double2 smem[];
    const int p0 = blockIdx.x * np_max;
    const int np = min(np_max, numax - p0);
    double2* bufA = smem;
    double2* bufB = smem + np_max * S::BUF_A;
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        const int nu = p0 + p;
        double2 acc = make_double2(0.0, 0.0);
        for (int c0 = 0; c0 < nchunk; c0 += 8) {      // eight loads in flight
            double2 r[8];
#pragma unroll
            for (int c = 0; c < 8; ++c)
                r[c] = c0 + c < nchunk ? partial[((size_t)(c0 + c) * numax + nu) * NQ + q] : make_double2(0.0, 0.0);
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (c0 + c < nchunk) acc = cadd(acc, r[c]);
        }
        bufA[p * NQ + q] = acc;
    }
    __syncthreads();
    // tail: (tc ? -U (sum_kω χm - χloc_m_sum) : 0) / (i ν_n), ν_n = (2n+1)π/β
    const double tnum = tc ? -U * (tail_sum[0] - chiloc_m_sum) : 0.0;
    const double2* res = sym_transform_any<DIM, N, TC>(np, bufA, bufB, T);
    for (int it = threadIdx.x; it < np * NQ; it += blockDim.x) {
        const int p = it / NQ, q = it - p * NQ;
        const double2 v = res[it];
        const int nu = p0 + p;
        const double w = (2.0 * nu + 1.0) * M_PI / beta;
        // tnum / (i w) = -i tnum / w
        double re = v.x * scale / beta + 0.0;
        double im = v.y * scale / beta - tnum / w;
        if (add_hartree) re += hartree;
        out[(size_t)nu * out_ld + q] = make_double2(re, im);
    }
}

// ω per CTA of the EoM forward kernel: a CTA takes one ν and a run of ω, np vectors at a time, and
// writes their sum.  Its steps are bound by the latencies of their loads and barriers, so a step of np
// vectors costs about 1 + np / 2 whatever np is, and the launch takes the rounds its CTAs need on the
// SMs' slots times the steps of one CTA (3D 32^3, 20 ν x 41 ω: 2 ω per CTA in 1.4 rounds 48 us, 3 ω
// in one round 41 us; 2D 64^2, 22 ν x 61 ω: 2 ω 36 us, 5 ω 30 us).
// The split is not monotone in numax: fewer ν can need more partial sums (2D 64^2, 61 ω: 270 rows at
// 30 ν, 589 at 19), so the handle's buffer is sized for every numax up to n_iv at once (eom_partial_need).
template <int DIM, int N>
EomShape eom_shape(int numax, int nw, bool tc) {
    using P = TransformPlan<DIM, N>;
    const int npm = tc ? std::max(1, std::min(16, (int)(kSmemBudgetTC / P::SMEM1))) : P::NP;
    EomShape best;
    double bt = 1e300;
    for (int np = 1; np <= npm; ++np) {
        const int by_smem = (int)((size_t)227 * 1024 / (np * P::SMEM1 + P::S::NQ * sizeof(double2) + 2048));
        const int slots = 148 * std::max(1, std::min(tc ? 2 : P::THREADS_SM / P::NT, by_smem));
        for (int w = np; w <= nw || w == np; ++w) {
            const int ctas = numax * ((nw + w - 1) / w);
            const double t = (double)((ctas + slots - 1) / slots) * ((w + np - 1) / np * (1.0 + 0.5 * np) + 0.5);
            if (t < bt) { bt = t; best = {w, np}; }
        }
    }
    return best;
}

// eom_shape, computed once per numax and number of ω (the search takes 1.5 to 6.5 us)
template <int DIM, int N>
EomShape eom_shape_of(ldga_ctx* ctx, int numax, int nw) {
    if (ctx->eom_shapes_nw != nw || (int)ctx->eom_shapes.size() < numax) {
        ctx->eom_shapes.assign(std::max(numax, ctx->Nnu), EomShape{});
        ctx->eom_shapes_nw = nw;
    }
    EomShape& s = ctx->eom_shapes[numax - 1];
    if (s.np == 0) s = eom_shape<DIM, N>(numax, nw, ctx->transform_tc);
    return s;
}

template <int DIM, int N>
size_t partial_need(ldga_ctx* ctx) {
    size_t need = 0;
    for (int numax = 1; numax <= ctx->sp.n_iv; ++numax) {
        const int wpc = eom_shape_of<DIM, N>(ctx, numax, ctx->Nw).wpc;
        need = std::max(need, (size_t)((ctx->Nw + wpc - 1) / wpc) * numax * ctx->Nq);
    }
    return need;
}

template <int DIM, int N>
int run_eom(ldga_ctx* ctx, int numax, double lam_m, double lam_d, const double* lm_dev, const double* ld_dev,
            int part, int& nchunk_out) {
    const int nws = shard_nw(ctx);
    const EomShape shape = eom_shape_of<DIM, N>(ctx, numax, nws);
    const int wpc = shape.wpc, np = shape.np;
    const int nchunk = (nws + wpc - 1) / wpc;
    // allocated with the handle; numax above n_iv and an ω shard can need more
    const int gs = grow_buffer(ctx, &ctx->d_partial, &ctx->partial_elems, (size_t)nchunk * numax * ctx->Nq);
    if (gs != LDGA_OK) return gs;
    EomArgs a;
    a.nnu = ctx->Nnu; a.nw = ctx->Nw; a.n_iv = ctx->sp.n_iv; a.n_iw = ctx->sp.n_iw; a.shift = ctx->sp.shift;
    a.fft_lo = ctx->fft_lo; a.numax = numax; a.w_per_chunk = wpc;
    a.w_begin = ctx->w_lo; a.w_end = ctx->w_hi;
    a.U = ctx->mp.U; a.lam_m = lam_m; a.lam_d = lam_d; a.part = part;
    a.lam_m_dev = lm_dev; a.lam_d_dev = ld_dev;
    nchunk_out = nchunk;
    StageTimer st_(ctx, LDGA_STAGE_EOM_FORWARD);
    return launch_form<DIM, N>(ctx, LDGA_FORMS(k_eom_forward), dim3(nchunk, numax), smem_bytes<DIM, N>(np) + (wpc > np ? ctx->Nq * sizeof(double2) : 0), "k_eom_forward", kThr<DIM, N, false>, a, ctx->d_ghat,
                               ctx->d_chi[0], ctx->d_gam[0], ctx->d_chi[1], ctx->d_gam[1], ctx->d_lambda0,
                               ctx->d_partial, np);
}

template <int DIM, int N>
int run_eom_inverse(ldga_ctx* ctx, int numax, int nchunk, const double* d_tail, int tc, double chiloc_m_sum,
                    double2* out, int out_ld, int add_hartree) {
    const int np = pairs_per_cta<DIM, N>(numax, ctx->transform_tc);
    const double scale = 1.0 / ((double)ctx->Nk * (double)ctx->Nk);
    const double hartree = ctx->mp.n * ctx->mp.U / 2.0;
    if (!ctx->shard_constants) {   // another rank of the ω shards adds the tail and Hartree terms
        tc = 0;
        add_hartree = 0;
    }
    StageTimer st_(ctx, LDGA_STAGE_EOM_INVERSE);
    return launch_form<DIM, N>(ctx, LDGA_FORMS(k_eom_inverse), dim3((numax + np - 1) / np), smem_bytes<DIM, N>(np), "k_eom_inverse", kThrOne<DIM, N, false>, numax,
                               nchunk, scale, ctx->mp.beta, ctx->mp.U, hartree, d_tail, tc, chiloc_m_sum,
                               ctx->d_partial, out, out_ld, add_hartree, np);
}

}  // namespace

// EoM: forward kernel then inverse kernel; `part` selects the contribution (-1: full EoM; 0..5 the
// calc_Σ_parts pieces).  d_tail: device scalar sum_kω(chi_m^lam) (read only when tc != 0).
namespace {
template <int DIM, int N>
int run_eom_all(ldga_ctx* ctx, int numax, double lam_m, double lam_d, const double* lm_dev, const double* ld_dev,
                int part, const double* d_tail, int tc, double chiloc_m_sum, double2* out, int out_ld,
                int add_hartree) {
    int nchunk = 0;
    int st = run_eom<DIM, N>(ctx, numax, lam_m, lam_d, lm_dev, ld_dev, part, nchunk);
    if (st != LDGA_OK) return st;
    return run_eom_inverse<DIM, N>(ctx, numax, nchunk, d_tail, tc, chiloc_m_sum, out, out_ld, add_hartree);
}
}  // namespace

size_t eom_partial_need(ldga_ctx* ctx) {
#define BODY(D, NS) partial_need<D, NS>(ctx)
    LDGA_FOR_EACH_GRID(LDGA_CASE)
#undef BODY
    return 0;
}

int launch_eom(ldga_ctx* ctx, int numax, double lam_m, double lam_d, const double* lam_m_dev,
               const double* lam_d_dev, int part, const double* d_tail, int tc, double chiloc_m_sum,
               double2* out, int out_ld, int add_hartree) {
#define BODY(D, NS)                                                                                      \
    run_eom_all<D, NS>(ctx, numax, lam_m, lam_d, lam_m_dev, lam_d_dev, part, d_tail, tc, chiloc_m_sum, out, \
                       out_ld, add_hartree)
    LDGA_FOR_EACH_GRID(LDGA_CASE)
#undef BODY
    return ctx_fail(ctx, LDGA_ERR_ARG, "unsupported k-grid size");
}

