// Shared by the BSE kernels' translation units: the arguments of one channel's batched solve.
#pragma once

#include "ldga_internal.cuh"

struct BseArgs {
    int nq, nnu, nw, qchunk;
    double beta, U;
    int s;                  // -1 for d, +1 for m
    const double2* Gamma;   // [Nnu, Nnu, Nw]
    const double2* chi0;    // [Nq, Nnu, Nw]
    double* chi;            // [Nq, Nw]
    double2* gam;           // [Nq, Nnu, Nw]
    int32_t* flags;         // [Nq, Nw]
    unsigned long long* stats = nullptr;   // [2] residual passes and warps of 8 q (may be null)
    // a flagged matrix is also appended (q + Nq w) to fail_list at atomicAdd(fail_count)
    int32_t* fail_list = nullptr;
    int32_t* fail_count = nullptr;
    int max_sweeps = 40;    // residual sweeps of an iteration before a q is flagged
    // k_bse_iter<..., ADJ = true>: right-hand sides [Nq, NL, Nw] instead of ones; the conjugate of the
    // solution goes to gam (which may be rhs itself), chi is not written
    const double2* rhs = nullptr;
};


// q order of the preconditioned solves (k_bse_qorder), computed once per chi0; nnu: the box size
int bse_ensure_qorder(ldga_ctx* ctx, const BseArgs& a, int nnu);
// The grouped preconditioned iteration (kernels_bse_group.cu) on tiles of 64 rows (boxes of 57..64); ad: the
// second channel in the same launch, or null.
int run_bse_group(ldga_ctx* ctx, const BseArgs& a, const BseArgs* ad);
