// fused_eval.hpp -- what the fused build + evaluate kernels need to know of the evaluation.
#pragma once

#include "build_device.cuh"
#include "eval_device.cuh"

namespace ddcb {

struct FusedEval
{
    EvalBasis eb;
    int ex_lo, ex_hi;
    const double* coords;
    Lines lx;
    double* out;
    Lines lo;
    // FEET kernels (the advection step): point q of line b is at pts[q] - dt * v(b), with
    // v(b) = velocity[b / v_div] (velocity == NULL: v_const); lx.n is the point count
    const double* pts;
    const double* velocity;
    double v_const, dt;
    int64_t v_div;
};

bool launch_reg_fused(BuildArgs const& args, FusedEval const& fe, int order, bool feet, cudaStream_t s);

} // namespace ddcb
