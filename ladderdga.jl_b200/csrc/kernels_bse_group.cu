// MIXED, grouped preconditioned iteration without exchanges ("iterg").
//
// The method of k_bse_iter (kernels_bse.cu): the q of one w share Gamma(w) and differ in the diagonal
// D_q = 1/chi0(q, :, w); sorted by D at the two lowest |nu|, QC consecutive q form B_bar = Gamma(w)^T +
// diag(mean D), its inverse C comes from Newton-Schulz on tcgen05 tensor cores (Gauss-Jordan in FP32
// where that does not converge), and every q iterates
//     r = 1 - B_q x   (FP64),    x += (I - C dD_q + (C dD_q)^2) C r   (TF32 products),   dD_q = D_q - mean D,
// until its FP64 backward error is small enough.
//
// What differs is the layout.  The products are formed transposed, X^T B^T and R^T C^T, with q on the
// rows of the mma.sync tiles.  Lane (g, t) of a warp (g = lane / 4, t = lane % 4) owns, for q = g, the columns
// nu = 8 n + 2 t + e, e = 0, 1: exactly what the accumulator tiles give it (row g, columns 2 t, 2 t + 1).  As an A operand a tile wants row g, column t: the k index is only summed over, so
// tile (n, e) takes nu = 8 n + 2 t + e as its column t, and the B operand is stored with the same
// permutation.  x, r and the corrections therefore stay in registers in both roles, and a pass has
// no shared-memory exchange and no warp synchronisation; in k_bse_iter each of its three products
// stages its input and its output through shared memory (eight synchronised round trips per pass).
//
// C is one Newton-Schulz step from the Jacobi seed, which is elementwise; only where its error bound
// is above 1e-2 do the tensor-core iterations run.
//
// Built for tiles of 64 rows (the box of 60), 8 warps of 8 q: all of a CTA's 64 q share one
// inverse and one copy of Gamma, and 8 warps share an SM (k_bse_iter at N = 64 has 4).  The third-order
// correction makes up for the wider groups: 4.9 passes per warp on the 2D 64^2 matrices, against
// 5.6 at 32 q and second order.  Bound: the FP64 tensor path (three real products per complex tile, 16 cycles per
// m8n8k4 and SM sub-partition) and the TF32 one, whose 16-row tiles are half empty at 8 q; by clock64
// 63 % of a CTA's time is at that bound, 28 % is set-up and output.
// Measured, Nnu = 60, 2D 64^2 (561 q x 61 w), one channel: 497 us; k_bse_iter 792 us.
// At N = 40 this layout gave nothing over k_bse_iter (two 16-q or three 8-q CTAs per SM: 241 and 215 us
// against 242 on one channel, 5 % slower on well-conditioned chains), so that size keeps k_bse_iter.
#include <cmath>

#include "bse_common.cuh"
#include "ns_inverse.cuh"

namespace {

constexpr int kGrpNsIts = 6;        // Newton-Schulz iterations at most
constexpr float kGrpNsTol = 1e-2f;  // stop once (max row sum of |I - B_bar X|)^2 <= kGrpNsTol
// Iterate to a backward error of 4e-15, accept 1e-14 like k_bse_iter (a matrix that has not got below 4e-15 at the
// sweep limit): stopping
// at 1e-14 left the solutions of this contraction 2.2x further from the exact ones than k_bse_iter's, with
// 4e-15 they are nearer (2.1e-15 against 3.7e-15, Nnu = 60, 2D 64^2) in the same time.  3e-15 and 2.5e-15 are nearer
// still (1.3e-15, 0.8e-15); of these only 4e-15 passes test_config2_lambda_dm, whose Newton ends at a
// root that depends on the last bits of chi: a change of this constant, or of an order of summation
// before that Newton, can fail the test with every array at its parity tolerance.
constexpr double kGrpStop = 4e-15, kGrpTol = 1e-14;

__device__ __forceinline__ double2 dmk(double r, double i) { return make_double2(r, i); }
__device__ __forceinline__ uint32_t tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
// d += a b, one m16n8k8 TF32 tile
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// d += a b, one m8n8k4 FP64 tile
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

// Shared memory of a CTA of NW warps with 8 q each (QC in all): [0, max(Gamma + C fragments, the
// Newton-Schulz buffers)), then D, the row sums, the mean diagonal, reduction scratch.
template <int N, int NW>
struct GrpSmem {
    static constexpr int QC = 8 * NW, NT = 32 * NW, T8 = N / 8;
    static constexpr int LDD = N + 1;                 // row stride of D: 16 bytes off a bank line per q
    static constexpr int LDE = N + 4;                 // row stride of dD (float2): 32 bytes off
    static constexpr int TPR = NT / N < 1 ? 1 : (NT / N > 4 ? 4 : NT / N);   // threads per row of the set-up
    static constexpr size_t g_bytes = (size_t)N * N * sizeof(double2);
    static constexpr size_t c_bytes = (size_t)T8 * T8 * 32 * sizeof(float4);
    static constexpr size_t ns_bytes = ns::NsSmem<N>::bytes;
    static constexpr size_t off_C = g_bytes;
    static constexpr size_t off_D = g_bytes + c_bytes > ns_bytes ? g_bytes + c_bytes : ns_bytes;
    static constexpr size_t off_E = off_D + (size_t)QC * LDD * sizeof(double2);
    static constexpr size_t off_part = off_E + (size_t)QC * LDE * sizeof(float2);
    static constexpr size_t off_dbar = off_part + (size_t)TPR * N * sizeof(double2);
    static constexpr size_t off_rowabs = off_dbar + (size_t)N * sizeof(double2);
    static constexpr size_t off_x0 = off_rowabs + (size_t)N * sizeof(double);   // Jacobi seed, float2
    static constexpr size_t off_bar = off_x0 + (size_t)N * sizeof(float2), off_slot = off_bar + 8;
    static constexpr size_t off_red = off_bar + 16;
    static constexpr size_t bytes = off_red + ((NW * sizeof(float) + 15) & ~size_t(15));
    static_assert(off_bar % 8 == 0 && off_D % 16 == 0 && off_part % 16 == 0, "alignment");
};

// position of C_ij in the fragments (float index): tile (i / 8, j / 8), lane 4 (i mod 8) + (j mod 8) / 2,
// {Re j even, Re j odd, Im j even, Im j odd}
template <int N>
__device__ __forceinline__ int cfrag(int i, int j) {
    return (((i >> 3) * (N / 8) + (j >> 3)) * 32 + (i & 7) * 4 + ((j & 7) >> 1)) * 4 + (j & 1);
}
// position of B_ij in the Gamma fragments (double2 index): tile (i / 8, k tile 2 (j / 8) + j mod 2), lane
// 4 (i mod 8) + (j mod 8) / 2
template <int N>
__device__ __forceinline__ int gfrag(int i, int j) {
    return ((i >> 3) * (N / 4) + 2 * (j >> 3) + (j & 1)) * 32 + (i & 7) * 4 + ((j & 7) >> 1);
}

// C = (B)^-1 in FP32 by Gauss-Jordan without pivoting on [N][N] float2 in `m` (row-major, holding B);
// a poor result only costs sweeps.  All threads; col: scratch [N] float2.
template <int N>
__device__ void gauss_jordan(float2* m, float2* col) {
    for (int k = 0; k < N; ++k) {
        __syncthreads();
        const float2 p = m[k * N + k];
        const float d = 1.f / (p.x * p.x + p.y * p.y);
        const float2 pi = make_float2(p.x * d, -p.y * d);
        for (int i = threadIdx.x; i < N; i += blockDim.x) col[i] = m[i * N + k];
        __syncthreads();
        for (int j = threadIdx.x; j < N; j += blockDim.x)      // row k: u / p, the pivot's column 1 / p
            m[k * N + j] = j == k ? pi : fmul(m[k * N + j], pi);
        __syncthreads();
#pragma unroll 1
        for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
            const int i = e / N, j = e - i * N;
            if (i == k) continue;
            const float2 t = fmul(col[i], m[k * N + j]);
            const float2 v = j == k ? make_float2(0.f, 0.f) : m[e];
            m[e] = make_float2(v.x - t.x, v.y - t.y);
        }
    }
    __syncthreads();
}

// C where one step from the Jacobi seed does not do: Newton-Schulz on the tensor cores (ns_inverse.cuh),
// Gauss-Jordan where that does not converge either.  All threads; C fragments out, the Gamma fragments
// (whose space the buffers take) written again from Gw.
template <int N, int NW>
__device__ __forceinline__ void group_inverse(unsigned char* sm, const double2* __restrict__ Gw, int nl) {
    using S = GrpSmem<N, NW>;
    using NSm = ns::NsSmem<N>;
    constexpr int NT = S::NT;
    const int tid = threadIdx.x;
    double2* Gf = reinterpret_cast<double2*>(sm);
    float* Cf = reinterpret_cast<float*>(sm + S::off_C);
    const double2* dbar = reinterpret_cast<const double2*>(sm + S::off_dbar);
    const float2* x0 = reinterpret_cast<const float2*>(sm + S::off_x0);
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + S::off_bar);
    uint32_t* slot = reinterpret_cast<uint32_t*>(sm + S::off_slot);
    float* red = reinterpret_cast<float*>(sm + S::off_red);
    auto belt = [&](int i, int j) {      // B_bar_ij
        double2 v = (i < nl && j < nl) ? Gw[(size_t)i * nl + j] : dmk(0.0, 0.0);
        return i == j ? cadd(v, dbar[i]) : v;
    };
#pragma unroll 1
    for (int e = tid; e < N * N; e += NT) {
        const int i = e / N, j = e - i * N;
        const double2 v = belt(i, j);
        const float2 xv = i == j ? x0[i] : make_float2(0.f, 0.f);
        const uint32_t oa = tc05::kmajor_offset(N, i, j), ob = tc05::kmajor_offset(N, j, i);
        *reinterpret_cast<float*>(sm + NSm::off_br + oa) = tc05::to_tf32f((float)v.x);
        *reinterpret_cast<float*>(sm + NSm::off_bi + oa) = tc05::to_tf32f((float)v.y);
        *reinterpret_cast<float*>(sm + NSm::off_xr + oa) = tc05::to_tf32f(xv.x);
        *reinterpret_cast<float*>(sm + NSm::off_xi + oa) = tc05::to_tf32f(xv.y);
        *reinterpret_cast<float*>(sm + NSm::off_tr + ob) = tc05::to_tf32f(xv.x);
        *reinterpret_cast<float*>(sm + NSm::off_ti + ob) = tc05::to_tf32f(xv.y);
    }
    tc05::fence_before();
    __syncthreads();                           // the TMEM address is visible
    tc05::fence_after();
    ns::NsState st{*slot, 0u, true};
    auto emit = [&](int i, int c, const float (&re)[16], const float (&im)[16]) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (c + j < N) {
                const int f = cfrag<N>(i, c + j);
                Cf[f] = __uint_as_float(tf32(re[j]));
                Cf[f + 2] = __uint_as_float(tf32(im[j]));
            }
    };
    const bool ok = ns::newton_schulz<N>(sm, bar, red, st, kGrpNsIts, kGrpNsTol, emit, nullptr);
    ns::drain(st, bar);
    tc05::fence_before();
    __syncthreads();
    if (!ok) {
        float2* mtx = reinterpret_cast<float2*>(sm);        // [N][N] float2: half of Gamma's space
        float2* col = reinterpret_cast<float2*>(sm + S::off_part);
#pragma unroll 1
        for (int e = tid; e < N * N; e += NT) {
            const double2 v = belt(e / N, e - (e / N) * N);
            mtx[e] = make_float2((float)v.x, (float)v.y);
        }
        gauss_jordan<N>(mtx, col);
#pragma unroll 1
        for (int e = tid; e < N * N; e += NT) {
            const int f = cfrag<N>(e / N, e - (e / N) * N);
            Cf[f] = __uint_as_float(tf32(mtx[e].x));
            Cf[f + 2] = __uint_as_float(tf32(mtx[e].y));
        }
        __syncthreads();
    }
#pragma unroll 1
    for (int e = tid; e < N * N; e += NT) {
        const int i = e / N, j = e - i * N;
        Gf[gfrag<N>(i, j)] = (i < nl && j < nl) ? Gw[(size_t)i * nl + j] : dmk(0.0, 0.0);
    }
    __syncthreads();
}

template <int N, int NW>
__global__ void __launch_bounds__(32 * NW, 1) k_bse_group(const BseArgs a_m, const BseArgs a_d, int qpc,
                                                             const int32_t* __restrict__ perm) {
    using S = GrpSmem<N, NW>;
    constexpr int NT = S::NT, T8 = S::T8, LDD = S::LDD, LDE = S::LDE, QC = S::QC, TPR = S::TPR;
    extern __shared__ __align__(128) unsigned char gr_raw[];
    BseArgs a = a_m;
    if (blockIdx.z) {
        a.s = a_d.s; a.Gamma = a_d.Gamma; a.chi = a_d.chi; a.gam = a_d.gam; a.flags = a_d.flags;
        a.fail_list = a_d.fail_list; a.fail_count = a_d.fail_count;
    }
    double2* Gf = reinterpret_cast<double2*>(gr_raw);
    float* Cf = reinterpret_cast<float*>(gr_raw + S::off_C);
    double2* Dq = reinterpret_cast<double2*>(gr_raw + S::off_D);
    double2* part = reinterpret_cast<double2*>(gr_raw + S::off_part);
    double2* dbar = reinterpret_cast<double2*>(gr_raw + S::off_dbar);
    double* rowabs = reinterpret_cast<double*>(gr_raw + S::off_rowabs);
    float2* Eq = reinterpret_cast<float2*>(gr_raw + S::off_E);
    float2* x0 = reinterpret_cast<float2*>(gr_raw + S::off_x0);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int nl = a.nnu, w = blockIdx.y, g0 = blockIdx.x * qpc;
    const int nvalid = min(qpc, a.nq - g0);
    const int32_t* pw = perm + (size_t)w * a.nq + g0;
    const double2* Gw = a.Gamma + (size_t)w * nl * nl;

    // The tensor-core inverse's mbarrier and TMEM are set up here, although few CTAs need them: with the
    // allocation inside the branch that does, the launch is given one CTA per SM whatever it needs
    // (tile of 40: 294 us against 241 with it here).
    uint64_t* bar = reinterpret_cast<uint64_t*>(gr_raw + S::off_bar);
    uint32_t* slot = reinterpret_cast<uint32_t*>(gr_raw + S::off_slot);
    if (tid == 0) {
        tc05::mbar_init(bar, 1);
        tc05::mbar_fence_init();
    }
    if (tid < 32) tc05::tmem_alloc(slot, ns::NsSmem<N>::tmem_cols);
    // ---- Gamma(w) and chi0 of the CTA's q into registers (every load in flight).  Element e = tid + NT m of
    // Gamma is B_ij, i = e / N; of D, q = e / N, nu = e mod N.
    constexpr int NG = (N * N + NT - 1) / NT, ND = (QC * N + NT - 1) / NT;
    constexpr int NB = ND % 10 == 0 ? 10 : ND % 9 == 0 ? 9 : ND % 8 == 0 ? 8 : ND % 7 == 0 ? 7 : ND % 6 == 0 ? 6 : 4;
    static_assert(ND % NB == 0, "whole batches");
    {
        int qg[ND];
#pragma unroll
        for (int m = 0; m < ND; ++m) {
            const int qq = (tid + NT * m) / N;
            qg[m] = qq < nvalid ? pw[qq] : -1;
        }
        double2 gv[NG];
#pragma unroll
        for (int m = 0; m < NG; ++m) {
            const int e = tid + NT * m, i = e / N, j = e - i * N;
            gv[m] = (e < N * N && i < nl && j < nl) ? Gw[(size_t)i * nl + j] : dmk(0.0, 0.0);
        }
        double2 cv[ND];
#pragma unroll
        for (int m = 0; m < ND; ++m) {
            const int e = tid + NT * m, v = e - (e / N) * N;      // padding rows (nu >= nl): D = 1
            cv[m] = qg[m] >= 0 && v < nl ? a.chi0[(size_t)qg[m] + (size_t)a.nq * (v + (size_t)nl * w)] : dmk(1.0, 0.0);
        }
#pragma unroll
        for (int m = 0; m < NG; ++m) {
            const int e = tid + NT * m, i = e / N, j = e - i * N;
            if (e < N * N) Gf[gfrag<N>(i, j)] = gv[m];
        }
        // D = 1 / chi0 by batch inversion (prefix products of the squared moduli, one division, two
        // products each), element by element where a product leaves [1e-300, 1e300]
#pragma unroll
        for (int b0 = 0; b0 < ND; b0 += NB) {
            double nrm[NB], pre[NB], prod = 1.0;
#pragma unroll
            for (int m = 0; m < NB; ++m) {
                nrm[m] = cv[b0 + m].x * cv[b0 + m].x + cv[b0 + m].y * cv[b0 + m].y;
                pre[m] = prod;
                prod *= nrm[m];
            }
            const bool fine = prod > 1e-300 && prod < 1e300;
            double r = 1.0 / prod;
#pragma unroll
            for (int m = NB - 1; m >= 0; --m) {
                const int e = tid + NT * (b0 + m), qq = e / N, v = e - qq * N;
                const double inv = r * pre[m];
                r *= nrm[m];
                const double2 d = dmk(cv[b0 + m].x * inv, -cv[b0 + m].y * inv);
                if (e < QC * N) Dq[qq * LDD + v] = qg[b0 + m] >= 0 ? d : dmk(0.0, 0.0);
            }
            if (!fine) {
#pragma unroll 1
                for (int m = b0; m < b0 + NB; ++m) {      // rare: rolled, from chi0 again
                    const int e = tid + NT * m, qq = e / N, v = e - qq * N;
                    if (qq < nvalid && v < nl)
                        Dq[qq * LDD + v] = cinv(a.chi0[(size_t)pw[qq] + (size_t)a.nq * (v + (size_t)nl * w)]);
                    else if (e < QC * N) Dq[qq * LDD + v] = qq < nvalid ? dmk(1.0, 0.0) : dmk(0.0, 0.0);
                }
            }
        }
    }
    __syncthreads();
    // ---- mean diagonal (TPR partial sums per nu, then their sum) and the Jacobi seed 1 / B_bar_ii
    if (tid < TPR * N) {
        const int i = tid % N, p = tid / N;
        double2 m = dmk(0.0, 0.0);
#pragma unroll 4
        for (int q = p; q < nvalid; q += TPR) m = cadd(m, Dq[q * LDD + i]);
        part[tid] = m;
    }
    __syncthreads();
    if (tid < N) {
        double2 m = part[tid];
        for (int p = 1; p < TPR; ++p) m = cadd(m, part[p * N + tid]);
        m = cscale(m, 1.0 / (double)max(nvalid, 1));
        dbar[tid] = m;
        const double2 v = cadd(Gf[gfrag<N>(tid, tid)], m);
        const float br = (float)v.x, bi = (float)v.y, sc = 1.f / (br * br + bi * bi);
        x0[tid] = make_float2(br * sc, -bi * sc);
    }
    __syncthreads();
    // ---- C: one Newton-Schulz step from the Jacobi seed X_0 = diag(x) is elementwise,
    //     X_1 = X_0 (2 I - B_bar X_0):  C_ii = x_i,  C_ij = -x_i B_ij x_j,   I - B_bar X_1 = (I - B_bar X_0)^2,
    // formed with the row sums of |B| off the diagonal and of |I - B_bar X_0|; dD = D - mean D in FP32
#pragma unroll 2
    for (int e = tid; e < QC * N; e += NT) {
        const int qq = e / N, v = e - qq * N;
        const double2 d = Dq[qq * LDD + v], db = dbar[v];
        Eq[qq * LDE + v] = make_float2((float)(d.x - db.x), (float)(d.y - db.y));
    }
    if (tid < TPR * N) {
        const int i = tid % N, p = tid / N;
        const float2 xi = x0[i];
        double s = 0.0;
        float es = 0.f;
#pragma unroll 2
        for (int j = p; j < N; j += TPR) {
            const double2 v = Gf[gfrag<N>(i, j)];
            const float2 y = fmul(make_float2((float)v.x, (float)v.y), x0[j]);   // (B X_0)_ij, i != j
            float2 c = fmul(make_float2(-xi.x, -xi.y), y);
            if (j == i) c = xi;
            else {
                s += fabs(v.x) + fabs(v.y);
                es += fabsf(y.x) + fabsf(y.y);
            }
            const int f = cfrag<N>(i, j);
            Cf[f] = __uint_as_float(tf32(c.x));
            Cf[f + 2] = __uint_as_float(tf32(c.y));
        }
        part[tid] = dmk(s, (double)es);
    }
    __syncthreads();
    float ek = 0.f;
    if (tid < N) {
        double2 s = part[tid];
        for (int p = 1; p < TPR; ++p) s = cadd(s, part[p * N + tid]);
        rowabs[tid] = s.x;
        ek = (float)s.y;
        if (!(ek == ek)) ek = INFINITY;
    }
    if (__syncthreads_or(!(ek * ek <= kGrpNsTol))) group_inverse<N, NW>(gr_raw, Gw, nl);
    if (tid < 32) {
        tc05::fence_after();
        tc05::tmem_free(*slot, ns::NsSmem<N>::tmem_cols);
    }

    // ---- this warp's q: 8 consecutive ones of the group; no barrier from here on
    const int ql0 = warp * 8;
    if (ql0 >= nvalid) return;
    const double2* Dl = Dq + (ql0 + g) * LDD;    // this lane's rows of D and dD
    const float2* El = Eq + (ql0 + g) * LDE;
    const float4* Cl = reinterpret_cast<const float4*>(Cf) + lane;
    const double2* Gl = Gf + lane;

    // v <- C v (TF32); v[n][e] is element nu = 8 n + 2 t + e of q = g; the tiles' rows 8..15 are zero
    auto apply = [&](float2 (&v)[T8][2]) {
        uint32_t ar[T8][4], ai[T8][4];
#pragma unroll
        for (int n = 0; n < T8; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                ar[n][2 * e] = tf32(v[n][e].x);
                ai[n][2 * e] = tf32(v[n][e].y);
                ar[n][2 * e + 1] = ai[n][2 * e + 1] = 0u;
            }
#pragma unroll
        for (int n = 0; n < T8; ++n) {
            float dre[4] = {0.f, 0.f, 0.f, 0.f}, dim[4] = {0.f, 0.f, 0.f, 0.f}, dni[4] = {0.f, 0.f, 0.f, 0.f},
                  di2[4] = {0.f, 0.f, 0.f, 0.f};   // four chains: an accumulator's next use is 3 tiles away
#pragma unroll
            for (int k = 0; k < T8; ++k) {
                const float4 c = Cl[(n * T8 + k) * 32];
                const uint32_t r0 = __float_as_uint(c.x), r1 = __float_as_uint(c.y);
                const uint32_t i0 = __float_as_uint(c.z), i1 = __float_as_uint(c.w);
                mma_tf32(dre, ar[k], r0, r1);
                mma_tf32(dni, ai[k], i0, i1);
                mma_tf32(dim, ar[k], i0, i1);
                mma_tf32(di2, ai[k], r0, r1);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) v[n][e] = make_float2(dre[e] - dni[e], dim[e] + di2[e]);
        }
    };
    // v <- (I - C dD + (C dD)^2) C v
    auto correct = [&](float2 (&v)[T8][2]) {
        apply(v);
        float2 z[T8][2];
#pragma unroll
        for (int n = 0; n < T8; ++n)
#pragma unroll
            for (int e = 0; e < 2; ++e) z[n][e] = v[n][e];
#pragma unroll 1
        for (int o = 0; o < 2; ++o) {      // rolled: unrolled, the compiler keeps dD of both orders and spills
#pragma unroll
            for (int n = 0; n < T8; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) z[n][e] = fmul(El[8 * n + 2 * t + e], z[n][e]);
            apply(z);
            const float sg = o ? 1.f : -1.f;
#pragma unroll
            for (int n = 0; n < T8; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    v[n][e].x = fmaf(sg, z[n][e].x, v[n][e].x);
                    v[n][e].y = fmaf(sg, z[n][e].y, v[n][e].y);
                }
        }
    };

    double rown = 0.0, berr = 0.0;
    bool conv = ql0 + g >= nvalid;
    double2 x[T8][2];
    float2 rr[T8][2];
#pragma unroll
    for (int n = 0; n < T8; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int i = 8 * n + 2 * t + e;
            const double2 gd = Gf[gfrag<N>(i, i)], d = Dl[i];
            rown = fmax(rown, rowabs[i] + fabs(gd.x + d.x) + fabs(gd.y + d.y));
            rr[n][e] = make_float2(i < nl ? 1.f : 0.f, 0.f);
        }
    rown = fmax(rown, __shfl_xor_sync(0xffffffffu, rown, 1));
    rown = fmax(rown, __shfl_xor_sync(0xffffffffu, rown, 2));
    correct(rr);
#pragma unroll
    for (int n = 0; n < T8; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) x[n][e] = dmk((double)rr[n][e].x, (double)rr[n][e].y);

    int passes = 0;
    for (int it = 0;; ++it) {
        // r = 1 - (Gamma^T + D) x: three real tile products per complex tile (Karatsuba)
        double res = 0.0, xn = 0.0;
#pragma unroll
        for (int n = 0; n < T8; ++n) {
            double t1[2] = {0.0, 0.0}, t2[2] = {0.0, 0.0}, t3[2] = {0.0, 0.0};
#pragma unroll
            for (int k = 0; k < T8; ++k)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const double2 b = Gl[(n * 2 * T8 + 2 * k + e) * 32], xv = x[k][e];
                    mma_f64(t1, xv.x, b.x);
                    mma_f64(t2, xv.y, b.y);
                    mma_f64(t3, xv.x + xv.y, b.x + b.y);
                }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int i = 8 * n + 2 * t + e;
                const double2 xv = x[n][e], dx = cmul(Dl[i], xv);
                const double rx = (i < nl ? 1.0 : 0.0) - (t1[e] - t2[e] + dx.x);
                const double ry = -(t3[e] - t1[e] - t2[e] + dx.y);
                res = fmax(res, fabs(rx) + fabs(ry));
                xn = fmax(xn, fabs(xv.x) + fabs(xv.y));
                rr[n][e] = make_float2((float)rx, (float)ry);
            }
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            res = fmax(res, __shfl_xor_sync(0xffffffffu, res, o));
            xn = fmax(xn, __shfl_xor_sync(0xffffffffu, xn, o));
        }
        if (!conv) berr = res / (rown * xn + 1.0);
        conv = conv || berr <= kGrpStop;
        passes = it + 1;
        if (__all_sync(0xffffffffu, conv) || it >= a.max_sweeps) break;
        correct(rr);
        if (!conv) {
#pragma unroll
            for (int n = 0; n < T8; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    x[n][e].x += (double)rr[n][e].x;
                    x[n][e].y += (double)rr[n][e].y;
                }
        }
    }
    if (a.stats && lane == 0) {
        atomicAdd(&a.stats[0], (unsigned long long)passes);
        atomicAdd(&a.stats[1], 1ull);
    }

    // ---- chi, gamma = x / (chi0 (1 + s U chi)), flag (a q above the bound goes to the pivoted solve)
    double sx = 0.0;
#pragma unroll
    for (int n = 0; n < T8; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) sx += x[n][e].x;      // padding rows of x are 0
    sx += __shfl_xor_sync(0xffffffffu, sx, 1);
    sx += __shfl_xor_sync(0xffffffffu, sx, 2);
    const int ql = ql0 + g;
    if (ql >= nvalid) return;
    const int q = pw[ql];
    const double chi = sx / (a.beta * a.beta);
    const bool good = isfinite(chi) && isfinite(berr) && berr <= kGrpTol;
    if (t == 0) {
        a.chi[(size_t)q + (size_t)a.nq * w] = chi;
        a.flags[(size_t)q + (size_t)a.nq * w] = good ? 0 : 1;
        if (!good && a.fail_list) a.fail_list[atomicAdd(a.fail_count, 1)] = q + a.nq * w;
    }
    const double rf = 1.0 / (1.0 + a.s * a.U * chi);
#pragma unroll
    for (int n = 0; n < T8; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int i = 8 * n + 2 * t + e;
            if (i < nl) a.gam[(size_t)q + (size_t)a.nq * (i + (size_t)nl * w)] = cscale(cmul(x[n][e], Dl[i]), rf);
        }
}

template <int N, int NW>
int launch_group(ldga_ctx* ctx, const BseArgs& a, const BseArgs* ad) {
    using S = GrpSmem<N, NW>;
    auto kern = k_bse_group<N, NW>;
    LDGA_CUDA(ctx, set_smem(ctx, kern, S::bytes));
    StageTimer st_(ctx, LDGA_STAGE_BSE);
    const int qo = bse_ensure_qorder(ctx, a, a.nnu);
    if (qo != LDGA_OK) return qo;
    // As few groups as QC allows, of about the same number of q each: more and smaller groups took more rounds
    // on the SMs at the same time per CTA (2D 64^2, Nnu = 60: 64 q per CTA 497 us, 47 q 551 us).  Groups of 32 where
    // one channel's have an SM each and the launch takes no more rounds than with groups of 64: with four
    // warps, one per sub-partition, a CTA has 0.77 of the time of eight, and narrower groups need fewer sweeps.  One
    // channel, random / RPA-like vertex, groups of 64 against 32: 153 q x 7 w 231 / 150 us against 126 / 116, 153 q x 17 w
    // 228 / 147 against 126 / 115, 91 q x 17 w 286 / 156 against 194 / 115; a round more loses (both channels, 153 q x
    // 17 w, RPA-like, 173 us against 201; one channel, 325 q x 17 w, 164 / 151 against 172 / 188).  The line depends on the whole
    // range of w, so a matrix has the same group, and bits, in a shard; one channel and both may differ by it.
    const int z = ad ? 2 : 1;
    auto rounds = [](long ctas) { return (ctas + 147) / 148; };
    const long c32 = (long)((a.nq + 31) / 32) * ctx->Nw, c64 = (long)((a.nq + 63) / 64) * ctx->Nw;
    const int per = c32 <= 148 && rounds(z * c32) <= rounds(z * c64) ? 32 : S::QC;
    const int nct = (a.nq + per - 1) / per, qpc = (a.nq + nct - 1) / nct;
    dim3 grid((a.nq + qpc - 1) / qpc, a.nw, z);
    kern<<<grid, S::NT, S::bytes, ctx->stream>>>(a, ad ? *ad : a, qpc, ctx->d_qperm);
    LDGA_LAUNCHED(ctx, "k_bse_group");
    return LDGA_OK;
}

}  // namespace

int run_bse_group(ldga_ctx* ctx, const BseArgs& a, const BseArgs* ad) {
    constexpr int N = 64;
    if (!ctx->d_qperm) return ctx_fail(ctx, LDGA_ERR_ARG, "preconditioned BSE: q order buffer missing");
    if (a.nnu > N || a.nnu <= N - 8) return ctx_fail(ctx, LDGA_ERR_ARG, "preconditioned BSE: tile and box size");
    return launch_group<N, 8>(ctx, a, ad);
}
