// adjoint_args.hpp -- the arguments of the adjoint kernels.
#pragma once

#include "build_device.cuh"
#include "eval_device.cuh"

namespace ddcb {

struct AdjointArgs
{
    SolveTables t;          // factorisation of A^T
    RhsMap r;
    int64_t nlines;
    int nct;
    int tile_req;           // Builder::tile_req
    const double* gc;       // cotangents of the coefficients (size rows)
    Lines lgc;
    double* gv;             // cotangents of the samples (npoints rows)
    Lines lgv;
    double* gdlo;           // cotangents of the lower / upper Hermite derivatives (nbv rows), or NULL
    Lines lglo;
    double* gdhi;
    Lines lghi;
    int pair_in;            // g_coefs: adjacent line pairs 16-byte aligned and contiguous
    int pair_out;           // g_vals: the same
};

struct EvalAdjointArgs
{
    EvalBasis eb;
    int ex_lo, ex_hi;
    int64_t nlines;
    int size;               // coefficient rows
    const double* coords;
    Lines lx;
    const double* coefs;    // needed for g_coords only
    Lines lc;
    int coef_pairs;         // coefs: adjacent line pairs 16-byte aligned and contiguous
    const double* gy;       // cotangents of the evaluated values
    Lines lgy;
    double* gc;             // out: cotangents of the coefficients (standalone kernel)
    Lines lgc;
    double* gx;             // out: cotangents of the coordinates, or NULL
    Lines lgx;
};

// Backward of build + evaluate over the register solve; false where it does not cover the plan.
bool launch_reg_adjoint(AdjointArgs const& a, EvalAdjointArgs const& ea, int order, cudaStream_t s);

} // namespace ddcb
