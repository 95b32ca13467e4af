// Symmetry-reduced k-space transform S on the irreducible wedge, computed by one CTA for a batch of
// independent vectors held in shared memory.
//
// For f even in every axis and symmetric under axis permutations (all G, K and products of them
// in the ladder path are: they live on the point-group-reduced grid and are expanded from it),
//     S(f)(q) = sum_{R in full grid} f(R) exp(-2 pi i q.R/N) = sum_{R in [0,N/2]^d} prod_a T[q_a][R_a] f(R),
// and S(f) is again such a function, so only wedge inputs and wedge outputs are needed.  The sum is
// evaluated axis by axis (x, then y, then z), keeping after each stage only the index ranges later
// stages read (M = N/2+1 rows of (M+1)M/2 columns, M of M^2 with qy <= qx, then qz <= qy), and no data
// ever leaves shared memory between stages.
//
// The convolution theorem used by the reference's conv_fft! / conv_tmp_add! then reads
//     (1/N_k) sum_k A(k) B(k+q) = S(S(A) S(B))(q) / N_k^2.
#pragma once

#include <type_traits>

#include "ldga_internal.cuh"

namespace ldga {

__device__ __forceinline__ void decode_pair(int j, int& b, int& c) {
    int bb = (int)((sqrtf(8.0f * (float)j + 1.0f) - 1.0f) * 0.5f);
    while (bb * (bb + 1) / 2 > j) --bb;
    while ((bb + 1) * (bb + 2) / 2 <= j) ++bb;
    b = bb;
    c = j - bb * (bb + 1) / 2;
}

// Shared-memory words (double2) needed per vector: input/stage-2 buffer and stage-1 buffer.
template <int DIM, int M>
struct TransformSmem {
    static constexpr int P2 = M * (M + 1) / 2;
    static constexpr int NQ = DIM == 2 ? P2 : M * (M + 1) * (M + 2) / 6;
    static constexpr int BUF_A = DIM == 2 ? NQ : (NQ > P2 * M ? NQ : P2 * M);   // in, then stage-2
    static constexpr int BUF_B = DIM == 2 ? M * M : M * P2;                     // stage-1
};

// ------------------------------------------------------------------------------------------------
// CUDA-core form.  One work item is one REAL column of a stage (the transform is real, so the real
// and imaginary parts are independent): a thread reads the column's M values once, folds them, and
// forms every row the later stages need.  The parts of a complex column sit in adjacent lanes, which
// keeps the accesses of the interleaved (re, im) layout contiguous.
//
// The fold.  A column e_0 .. e_{n/2} of period n (n even) with the rows
//     row(q) = e_0 + sum_{0<m<n/2} 2 cos(2 pi q m / n) e_m + cos(pi q) e_{n/2}
// splits by cos(2 pi q (n/2 - m) / n) = (-1)^q cos(2 pi q m / n):
//     odd q:   f_0 + sum_{0<m<n/4} 2 cos(2 pi q m / n) f_m,  f_m = e_m - e_{n/2-m},
//     even q:  row q/2 of the column e'_m = e_m + e_{n/2-m} of period n/2 (e'_{n/4} = 2 e_{n/4}),
// and so on until the period is odd.  All levels' f and the last column are M values again.  For
// N = 32 the 17 rows take 70 multiply-adds and 31 additions instead of 289, for N = 64 309 and 63 instead of 1089, and the
// cosines are N/4 - 1 constants, which stay in registers: with the 17 x 17 matrix as an operand every
// FP64 instruction needed its own constant load.
//
// What bounds it: shared-memory column reads and writes (260 KB per 3D 32^3 vector), then the
// barriers and loads of a CTA, which the other CTAs of its SM overlap.
// Within a stage the items are ordered by the number of rows they need (stage y: qx, stage z: qy),
// so a warp's lanes agree on their row loop; a second round over the items runs backwards, so a thread
// that had few rows first has many then.
// ------------------------------------------------------------------------------------------------
template <int N>
struct CosTab {
    static constexpr int NC = N % 2 ? N / 2 + 1 : N / 4 + 1;
    double c[NC];        // 2 cos(2 pi j / N)
};

// the levels of the fold: level l < K holds the f of period N >> l, level K the last column
template <int N>
struct FoldPlan {
    static constexpr int levels() {
        int k = 0;
        while ((N >> k) % 2 == 0) ++k;
        return k;
    }
    static constexpr int K = levels();
    static constexpr int len(int l) {
        const int n = N >> l;
        return l == K ? n / 2 + 1 : ((n / 2) % 2 == 0 ? n / 4 : (n / 2 + 1) / 2);
    }
    static constexpr int off(int l) {
        int o = 0;
        for (int i = 0; i < l; ++i) o += len(i);
        return o;
    }
    static constexpr int level(int q) {      // of row q
        for (int l = 0; l < K; ++l)
            if ((q >> l) & 1) return l;
        return K;
    }
    // 2 cos(2 pi j / N) = sgn(j) c[idx(j)]
    static constexpr int fold_j(int j) { return j % N < N - j % N ? j % N : N - j % N; }
    static constexpr int idx(int j) { return N % 2 == 0 && 4 * fold_j(j) > N ? N / 2 - fold_j(j) : fold_j(j); }
    static constexpr bool neg(int j) { return N % 2 == 0 && 4 * fold_j(j) > N; }
};

template <int N, int L, int ME, int M>
__device__ __forceinline__ void fold_column(const double (&e)[ME], double (&x)[M]) {
    using F = FoldPlan<N>;
    constexpr int n = N >> L, o = F::off(L);
    if constexpr (L == F::K) {
#pragma unroll
        for (int m = 0; m < F::len(L); ++m) x[o + m] = e[m];
    } else {
        constexpr int h = n / 2;
#pragma unroll
        for (int m = 0; m < F::len(L); ++m) x[o + m] = e[m] - e[h - m];
        double s[h / 2 + 1];
#pragma unroll
        for (int m = 0; m <= h / 2; ++m) s[m] = e[m] + e[h - m];
        fold_column<N, L + 1>(s, x);
    }
}

// body(std::integral_constant<int, i>) for i = A .. B - 1
template <int A, int B, class Body>
__device__ __forceinline__ void static_for(Body&& body) {
    if constexpr (A < B) {
        body(std::integral_constant<int, A>{});
        static_for<A + 1, B>(body);
    }
}

// rows r <= lim of the folded column, CH at a time, each in increasing m
template <int N, int CH, int R0 = 0, int M, class F>
__device__ __forceinline__ void rows_real(const double (&c)[CosTab<N>::NC], const double (&x)[M], int lim, F&& f) {
    using P = FoldPlan<N>;
    if constexpr (R0 < M) {
        if (R0 > lim) return;
        constexpr int R1 = R0 + CH < M ? R0 + CH : M;
        double acc[CH];
        static_for<R0, R1>([&](auto qc) {
            constexpr int q = decltype(qc)::value, l = P::level(q), o = P::off(l);
            double y = x[o];
            static_for<1, P::len(l)>([&](auto mc) {
                constexpr int m = decltype(mc)::value, j = P::idx(q * m);
                y = fma(P::neg(q * m) ? -c[j] : c[j], x[o + m], y);
            });
            acc[q - R0] = y;
        });
#pragma unroll
        for (int i = 0; i < R1 - R0; ++i)
            if (R0 + i <= lim) f(R0 + i, acc[i]);
        rows_real<N, CH, R0 + CH>(c, x, lim, f);
    }
}

template <int DIM, int N>
struct TransformPlan {
    static constexpr int M = N / 2 + 1;
    using S = TransformSmem<DIM, M>;
    static constexpr int COLS = DIM == 2 ? M : S::P2;             // complex columns of stages x and (3D) z
    // vectors per CTA at once: the count that fills whole warps best within 320 threads
    static constexpr int pick() {
        int best = 1;
        double beff = 0.0;
        for (int np = 1; np <= 16; ++np) {
            const int items = np * 2 * COLS, nt = (items + 31) / 32 * 32;
            if (np > 1 && (nt > 320 || (size_t)np * (S::BUF_A + S::BUF_B) * 16 > 112 * 1024)) break;
            double eff = (double)items / nt;
            if (nt < 96) eff *= 0.5;
            if (eff > beff + 0.02) { beff = eff; best = np; }
        }
        return best;
    }
    static constexpr int NP = pick();
    // threads: an item of stage x each; more, up to 352, where that brings the wedge points of a thread's loads and
    // stores down to 3 (3D) or 4 (2D) (2D 64^2 would need 576 and keeps 288 threads with 8 points)
    static constexpr int LDQ = DIM == 3 ? 3 : 4;
    static constexpr int NT_I = (NP * 2 * COLS + 31) / 32 * 32, NT_L = ((NP * S::NQ + LDQ - 1) / LDQ + 31) / 32 * 32;
    static constexpr int NT = NT_L > NT_I && NT_L <= 352 ? NT_L : NT_I;
    // one vector per CTA on its own SM (the EoM inverse): threads for stage y (3D) or the loads (2D)
    static constexpr int NT_ONE_W = (DIM == 3 ? 2 * M * M + 31 : (S::NQ + 1) / 2 + 31) / 32 * 32;
    static constexpr int NT_ONE = NT_ONE_W > 640 ? 640 : (NT_ONE_W > NT ? NT_ONE_W : NT);
    static constexpr size_t SMEM1 = (size_t)(S::BUF_A + S::BUF_B) * sizeof(double2);
    // resident CTAs the register allocation must allow: a column takes 2 M registers, its cosines N/2
    static constexpr int THREADS_SM = DIM == 3 ? 704 : 640;
    static constexpr int minb() {
        int b = THREADS_SM / NT;
        const int bs = (int)((size_t)224 * 1024 / (NP * SMEM1 + 1024));
        if (b > bs) b = bs;
        if (b > 16) b = 16;
        return b < 1 ? 1 : b;
    }
    static constexpr int MINB = minb();
    // rows formed together: in stage x every row is needed; in the others only rows <= a column's limit
    static constexpr int CHX = (M + (M + 6) / 7 - 1) / ((M + 6) / 7);
    static constexpr int CHY = (M + (M + 3) / 4 - 1) / ((M + 3) / 4);
};

// body(item) for item in [0, n): round 0 forwards, round 1 backwards, ...
template <class Body>
__device__ __forceinline__ void for_items_folded(int n, Body&& body) {
    const int nt = blockDim.x;
#pragma unroll 1
    for (int k = 0, lo = 0; lo < n; ++k, lo += nt) {
        const int hi = min(lo + nt, n);
        const int it = (k & 1) ? hi - 1 - (int)threadIdx.x : lo + (int)threadIdx.x;
        if (it >= lo && it < hi) body(it);
    }
}

__host__ __device__ __forceinline__ constexpr int tri(int a) { return a * (a + 1) / 2; }
__host__ __device__ __forceinline__ constexpr int tet(int a) { return a * (a + 1) * (a + 2) / 6; }

// Apply S to `np` vectors held in bufA as [p][NQ] (wedge-indexed); returns the buffer (bufA in 2D,
// bufB in 3D) that then holds the result in the same layout.  Both buffers are overwritten.  All
// threads of the CTA must call this after a barrier behind their writes of bufA; it ends on a barrier.
template <int DIM, int N>
__device__ double2* sym_transform(int np, double2* bufA, double2* bufB, const CosTab<N>& T) {
    using P = TransformPlan<DIM, N>;
    using S = typename P::S;
    constexpr int M = P::M, P2 = S::P2, NQ = S::NQ;
    double* A = reinterpret_cast<double*>(bufA);
    double* B = reinterpret_cast<double*>(bufB);
    double c[CosTab<N>::NC];
#pragma unroll
    for (int j = 0; j < CosTab<N>::NC; ++j) {
        c[j] = T.c[j];
        asm volatile("" : "+d"(c[j]));   // a register from here on, not a constant reloaded at each use
    }
    if constexpr (DIM == 2) {
        // stage x: W1[qx][b] = sum_a T[qx][a] f(a, b)
        for_items_folded(np * M * 2, [&](int it) {
            const int part = it & 1, r = it >> 1, p = r / M, b = r - p * M;
            const double* in = A + 2 * p * NQ + part;
            const int tb = tri(b);
            double v[M], x[M];
#pragma unroll
            for (int a = 0; a < M; ++a) v[a] = in[2 * (a <= b ? tb + a : tri(a) + b)];
            fold_column<N, 0>(v, x);
            double* w = B + 2 * (p * (M * M) + b) + part;
            rows_real<N, P::CHX>(c, x, M - 1, [&](int qx, double y) { w[2 * qx * M] = y; });
        });
        __syncthreads();
        // stage y: out(qx, qy) = sum_b T[qy][b] W1[qx][b], qy <= qx; columns in order of qx
        for_items_folded(np * M * 2, [&](int it) {
            const int part = it & 1, r = it >> 1, qx = r / np, p = r - qx * np;
            const double* w = B + 2 * (p * (M * M) + qx * M) + part;
            double v[M], x[M];
#pragma unroll
            for (int b = 0; b < M; ++b) v[b] = w[2 * b];
            fold_column<N, 0>(v, x);
            double* o = A + 2 * (p * NQ + tri(qx)) + part;
            rows_real<N, P::CHY>(c, x, qx, [&](int qy, double y) { o[2 * qy] = y; });
        });
        __syncthreads();
        return bufA;
    } else {
        // stage x: W1[qx][(b,c)] = sum_a T[qx][a] f(a, b, c) for b >= c
        for_items_folded(np * P2 * 2, [&](int it) {
            const int part = it & 1, r = it >> 1, p = r / P2, j = r - p * P2;
            int b, cc;
            decode_pair(j, b, cc);
            const double* in = A + 2 * p * NQ + part;
            const int i0 = tet(b) + tri(cc), i1 = tet(b) + cc, i2 = tri(b) + cc;   // a <= c, c < a <= b, a > b
            double v[M], x[M];
#pragma unroll
            for (int a = 0; a < M; ++a) v[a] = in[2 * (a <= cc ? i0 + a : a <= b ? i1 + tri(a) : i2 + tet(a))];
            fold_column<N, 0>(v, x);
            double* w = B + 2 * (p * (M * P2) + j) + part;
            rows_real<N, P::CHX>(c, x, M - 1, [&](int qx, double y) { w[2 * qx * P2] = y; });
        });
        __syncthreads();
        // stage y: W2[(qx,qy)][c] = sum_b T[qy][b] W1[qx][(b,c)], qy <= qx (W1 symmetric in b, c)
        for_items_folded(np * M * M * 2, [&](int it) {
            const int part = it & 1, r = it >> 1, qx = r / (np * M), s = r - qx * (np * M), p = s / M, cc = s - p * M;
            const double* w = B + 2 * (p * (M * P2) + qx * P2) + part;
            const int tc = tri(cc);
            double v[M], x[M];
#pragma unroll
            for (int b = 0; b < M; ++b) v[b] = w[2 * (b <= cc ? tc + b : tri(b) + cc)];
            fold_column<N, 0>(v, x);
            double* o = A + 2 * (p * S::BUF_A + tri(qx) * M + cc) + part;
            rows_real<N, P::CHY>(c, x, qx, [&](int qy, double y) { o[2 * qy * M] = y; });
        });
        __syncthreads();
        // stage z: out(qx,qy,qz) = sum_c T[qz][c] W2[(qx,qy)][c], qz <= qy; columns by falling qy
        for_items_folded(np * P2 * 2, [&](int it) {
            const int part = it & 1, r = it >> 1, j = r / np, p = r - j * np;
            int bb, cc;
            decode_pair(j, bb, cc);
            const int qy = M - 1 - bb, qx = M - 1 - cc;
            const double* w = A + 2 * (p * S::BUF_A + (tri(qx) + qy) * M) + part;
            double v[M], x[M];
#pragma unroll
            for (int m = 0; m < M; ++m) v[m] = w[2 * m];
            fold_column<N, 0>(v, x);
            double* o = B + 2 * (p * NQ + tet(qx) + tri(qy)) + part;
            rows_real<N, P::CHY>(c, x, qy, [&](int qz, double y) { o[2 * qz] = y; });
        });
        __syncthreads();
        return bufB;
    }
}

// ------------------------------------------------------------------------------------------------
// The same transform on the FP64 tensor path.  Every stage is T times a set of columns, T fixed: with
// mma.sync.m8n8k4 (FP64 operands, FP64 accumulation) T is the A operand, kept in registers as
// fragments of its 8 x 4 tiles (rows and k padded with zeros to multiples of 8 and 4), and the
// columns -- real and imaginary parts of 4 complex columns per 8-column tile -- are the B operand,
// gathered from shared memory (lane l holds B[k = l % 4][n = l / 4], n = 2 j + part of complex column
// j).  The accumulator gives lane l the complex output of row l / 4, column l % 4 (C[g][2t], C[g][2t+1]
// are its real and imaginary parts).  Warps take 8-column tiles in turn; a tile computes only the
// row tiles its columns need (stage y: qy <= qx, stage z: qz <= qy).  One tensor instruction replaces
// 256 FP64 FMAs, and no thread holds a column in registers (the CUDA-core form keeps M complex values
// per thread), so the kernels need far fewer registers.
template <int M>
struct TFrag {
    static constexpr int RT = (M + 7) / 8, KT = (M + 3) / 4;
    double a[RT][KT];
};

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

template <int M>
__device__ __forceinline__ void load_tfrag(const TMat<M>& T, TFrag<M>& F, int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int rt = 0; rt < TFrag<M>::RT; ++rt)
#pragma unroll
        for (int kt = 0; kt < TFrag<M>::KT; ++kt) {
            const int r = rt * 8 + g, k = kt * 4 + t;
            F.a[rt][kt] = (r < M && k < M) ? T.t[r * M + k] : 0.0;
        }
}

// One stage over `ncol` complex columns.  colB(j, k) returns column j's k-th input (k < M, j < ncol);
// rows(j) the largest output row column j needs (< M); out(j, r, v) receives row r of column j for every
// r <= rows(j).
template <int M, class ColB, class Rows, class Out>
__device__ __forceinline__ void tc_stage(const TFrag<M>& F, int ncol, ColB&& colB, Rows&& rows, Out&& out) {
    constexpr int RT = TFrag<M>::RT, KT = TFrag<M>::KT;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int ntile = (ncol + 3) / 4;
    for (int ct = warp; ct < ntile; ct += nwarp) {
        const int jb = ct * 4 + (g >> 1), part = g & 1;
        double b[KT];
#pragma unroll
        for (int kt = 0; kt < KT; ++kt) {
            const int k = kt * 4 + t;
            double v = 0.0;
            if (jb < ncol && k < M) {
                const double2 z = colB(jb, k);
                v = part ? z.y : z.x;
            }
            b[kt] = v;
        }
        int rmax = -1;
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (ct * 4 + c < ncol) rmax = max(rmax, rows(ct * 4 + c));
        const int jo = ct * 4 + t;
        // the row tiles' accumulations are independent chains: interleaved over k so that consecutive
        // tensor instructions do not wait for each other (the row-tile guard is uniform over the warp)
        double acc[RT][2];
#pragma unroll
        for (int rt = 0; rt < RT; ++rt) acc[rt][0] = acc[rt][1] = 0.0;
#pragma unroll
        for (int kt = 0; kt < KT; ++kt)
#pragma unroll
            for (int rt = 0; rt < RT; ++rt)
                if (rt * 8 <= rmax) dmma(acc[rt], F.a[rt][kt], b[kt]);
#pragma unroll
        for (int rt = 0; rt < RT; ++rt) {
            const int r = rt * 8 + g;
            if (rt * 8 <= rmax && jo < ncol && r <= rows(jo)) out(jo, r, make_double2(acc[rt][0], acc[rt][1]));
        }
    }
}

// sym_transform's interface and buffers on the tensor path.
template <int DIM, int M>
__device__ double2* sym_transform_tc(int np, double2* bufA, double2* bufB, const TMat<M>& T) {
    using S = TransformSmem<DIM, M>;
    constexpr int P2 = S::P2;
    constexpr int NQ = S::NQ;
    TFrag<M> F;
    load_tfrag<M>(T, F, threadIdx.x & 31);
    if constexpr (DIM == 2) {
        // stage x: W1[qx][b] = sum_a T[qx][a] f(a, b); column j = (p, b)
        tc_stage<M>(F, np * M,
            [&](int j, int k) { const int p = j / M, b = j - p * M; return bufA[p * NQ + sidx2(k, b)]; },
            [&](int) { return M - 1; },
            [&](int j, int r, double2 v) { const int p = j / M, b = j - p * M; bufB[p * (M * M) + r * M + b] = v; });
        __syncthreads();
        // stage y: out(qx, qy) = sum_b T[qy][b] W1[qx][b], qy <= qx; column j = (p, qx)
        tc_stage<M>(F, np * M,
            [&](int j, int k) { const int p = j / M, qx = j - p * M; return bufB[p * (M * M) + qx * M + k]; },
            [&](int j) { return j % M; },
            [&](int j, int r, double2 v) { const int p = j / M, qx = j - p * M; bufA[p * NQ + widx2(qx, r)] = v; });
        __syncthreads();
        return bufA;
    } else {
        // stage x: W1[qx][(b, c)] = sum_a T[qx][a] f(a, b, c), b >= c; column j = (p, pair)
        tc_stage<M>(F, np * P2,
            [&](int j, int k) {
                const int p = j / P2, pr = j - p * P2;
                int b, c;
                decode_pair(pr, b, c);
                return bufA[p * NQ + sidx3(k, b, c)];
            },
            [&](int) { return M - 1; },
            [&](int j, int r, double2 v) { const int p = j / P2, pr = j - p * P2; bufB[p * (M * P2) + r * P2 + pr] = v; });
        __syncthreads();
        // stage y: W2[(qx, qy)][c] = sum_b T[qy][b] W1[qx][(b, c)], qy <= qx; column j = (p, qx, c)
        tc_stage<M>(F, np * M * M,
            [&](int j, int k) {
                const int p = j / (M * M), rr = j - p * (M * M), qx = rr / M, c = rr - qx * M;
                return bufB[p * (M * P2) + qx * P2 + sidx2(k, c)];
            },
            [&](int j) { return (j % (M * M)) / M; },
            [&](int j, int r, double2 v) {
                const int p = j / (M * M), rr = j - p * (M * M), qx = rr / M, c = rr - qx * M;
                bufA[p * S::BUF_A + widx2(qx, r) * M + c] = v;
            });
        __syncthreads();
        // stage z: out(qx, qy, qz) = sum_c T[qz][c] W2[(qx, qy)][c], qz <= qy; column j = (p, pair)
        tc_stage<M>(F, np * P2,
            [&](int j, int k) { const int p = j / P2, pq = j - p * P2; return bufA[p * S::BUF_A + pq * M + k]; },
            [&](int j) {
                int qx, qy;
                decode_pair(j % P2, qx, qy);
                return qy;
            },
            [&](int j, int r, double2 v) {
                const int p = j / P2, pq = j - p * P2;
                int qx, qy;
                decode_pair(pq, qx, qy);
                bufB[p * NQ + widx3(qx, qy, r)] = v;
            });
        __syncthreads();
        return bufB;
    }
}

// the CUDA-core or the tensor-path form, chosen at compile time, and its coefficient operand
template <int N, bool TC>
using TransformCoef = std::conditional_t<TC, TMat<N / 2 + 1>, CosTab<N>>;

template <int DIM, int N, bool TC>
__device__ __forceinline__ double2* sym_transform_any(int np, double2* bufA, double2* bufB,
                                                      const TransformCoef<N, TC>& T) {
    if constexpr (TC) return sym_transform_tc<DIM, N / 2 + 1>(np, bufA, bufB, T);
    else return sym_transform<DIM, N>(np, bufA, bufB, T);
}

}  // namespace ldga

// Instantiation list: the k-grid sizes N per dimension the library is built for (N = 1: the one-point
// grid of the local quantities).
#define LDGA_FOR_EACH_GRID(X)                                                                          \
    X(2, 1) X(3, 1) X(2, 2) X(2, 4) X(2, 6) X(2, 8) X(2, 10) X(2, 12) X(2, 16) X(2, 20) X(2, 24) X(2, 32) \
    X(2, 40) X(2, 48) X(2, 64) X(2, 3) X(2, 5) X(2, 7) X(2, 9) X(2, 11) X(2, 13) X(2, 17) X(2, 21)        \
    X(2, 25) X(2, 33) X(2, 41) X(2, 49)                                                                \
    X(3, 2) X(3, 4) X(3, 6) X(3, 8) X(3, 10) X(3, 12) X(3, 16) X(3, 20) X(3, 24) X(3, 32) X(3, 3) X(3, 5) \
    X(3, 7) X(3, 9) X(3, 11) X(3, 13) X(3, 17) X(3, 21) X(3, 25) X(3, 33)
