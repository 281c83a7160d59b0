// reg_fused_kernels.cu -- build + evaluate, and the advection step, in one kernel over the register
// solve (reg_solve.cuh): the solved tile goes to shared memory in coefficient order, leaves from
// there or from the registers, and is evaluated in place. Uniform bases, as in fused_kernels.cu,
// which keeps the plans the register solve does not take.
#include <algorithm>

#include "fused_eval.hpp"
#include "reg_io.cuh"

namespace ddcb {

namespace {

template <int K, int MINLEN, int D, int ORDER, bool FEET>
__global__ void __launch_bounds__(512, 1) reg_build_eval_kernel(const __grid_constant__ BuildArgs args, const __grid_constant__ RegIo io,
                                                                const __grid_constant__ FusedEval fe)
{
    extern __shared__ __align__(16) double smem[];
    SolveTables const& t = args.t;
    int const P = 1 << io.lp, TL = 2 * P;
    int const p = threadIdx.x & (P - 1);
    int const c = threadIdx.x >> io.lp;
    int const nthr = blockDim.x >> io.lp;
    RegSmem const sm = reg_smem<K>(t, P, smem);
    double* const raw = sm.end;
    double* const tile = raw + t.k * TL;
    int a, len;
    chunk_rows(t, min(c, t.nchunk - 1), a, len);
    int64_t const tiles = (args.nlines + TL - 1) >> (io.lp + 1);
    // evaluation: a thread takes every nct-th point of line l
    int const l = threadIdx.x & (TL - 1);
    int const q0 = threadIdx.x / TL;
    int const nct = blockDim.x / TL;
    int const m = int(fe.lx.n);
    reg_load_tables<K>(t, sm);
    for (int64_t ti = blockIdx.x; ti < tiles; ti += gridDim.x) {
        int64_t const line0 = ti << (io.lp + 1);
        reg_fill(args, io, line0, tile, raw);
        cp_async_wait_all();
        __syncthreads();
        {
            double2 x[kRegRows];
            reg_load(io, tile, a, len, p, x);
            if (t.k > 0) reg_border_rhs(args, sm, raw, c, p, P);
            __syncthreads(); // the tile has been read
            reg_sweeps<K, MINLEN>(t, sm, x, len, c, p, P);
            if (t.k > 0) reg_border(t, sm, x, a, len, c, p, P);
            if (c < t.nchunk) {
                reg_store_tile(args, io, tile, a, len, p, x);
                if (args.out != nullptr && args.pair16_out) reg_store(args, line0 + 2 * p, a, len, x);
            }
            for (int r = c; r < t.k; r += nthr) {
                reg_store_row(args, io, true, line0 + 2 * p, tile, t.m + r, p, sm.x2[r * P + p]);
                if (args.out != nullptr && args.pair16_out) reg_store_row(args, io, false, line0 + 2 * p, tile, t.m + r, p, sm.x2[r * P + p]);
            }
        }
        // the first coordinates are on their way while the tile is completed, and each next group
        // while the one before is evaluated
        int64_t const line = min(line0 + l, args.nlines - 1);
        int64_t const sx = fe.lx.stride * nct, so = fe.lo.stride * nct;
        const double* __restrict__ xp = FEET ? fe.pts + q0 : fe.coords + line_offset(fe.lx, line) + q0 * fe.lx.stride;
        double* __restrict__ op = fe.out + line_offset(fe.lo, line) + q0 * fe.lo.stride;
        double const shift = FEET ? fe.dt * (fe.velocity ? __ldg(fe.velocity + line / fe.v_div) : fe.v_const) : 0.0;
        CoefDirect const acc {tile + l, TL};
        constexpr int U = 8; // points of a group
        int const npt = m > q0 ? (m - q0 + nct - 1) / nct : 0;
        auto load = [&](int i, double* xs) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (FEET) xs[u] = i + u < npt ? __ldg(xp + (i + u) * nct) : 0.0;
                else xs[u] = i + u < npt ? __ldcs(xp + (i + u) * sx) : 0.0;
            }
        };
        double xs[U];
        load(0, xs);
        __syncthreads();
        if (args.out != nullptr && !args.pair16_out) reg_drain(args, io, line0, tile);
        if (line0 + l < args.nlines)
            for (int i = 0; i < npt; i += U) {
                double next[U];
                load(i + U, next);
                int j[U];
#pragma unroll
                for (int u = 0; u < U; ++u) j[u] = uniform_place<ORDER>(fe.eb, fe.ex_lo, fe.ex_hi, FEET ? xs[u] - shift : xs[u], xs[u]);
#pragma unroll
                for (int u = 0; u < U; ++u) xs[u] = uniform_at<D, ORDER>(fe.eb, j[u], xs[u], acc);
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (i + u < npt) __stcs(op + (i + u) * so, xs[u]);
#pragma unroll
                for (int u = 0; u < U; ++u) xs[u] = next[u];
            }
        __syncthreads();
    }
}

template <int K, int D, int ORDER, bool FEET>
bool launch_reg_fused_kd(BuildArgs const& args, FusedEval const& fe, cudaStream_t s)
{
    SolveTables const& t = args.t;
    if (!reg_plain_rows(args) || fe.lx.n > (int64_t(1) << 30)) return false;
    RegIo io {};
    io.v0 = args.r.periodic ? 0 : args.r.nbe_lo;
    int const optin = device_limits().optin, sms = device_limits().sms;
    auto bytes = [&] { return sizeof(double) * (reg_smem_doubles<K>(t, 1 << io.lp) + size_t(args.r.size + t.k) * size_t(2 << io.lp)); };
    auto fits = [&](int threads, int blocks) { return (t.nchunk << io.lp) <= threads && bytes() + 1024 <= (size_t(optin) + 1024) / blocks; };
    auto tiles = [&] { return (args.nlines + (int64_t(2) << io.lp) - 1) >> (io.lp + 1); };
    // Two blocks of 256 threads per SM, one's copies beside the other's evaluation, with tiles of
    // eight lines or more; else one block of 512. A batch that leaves SMs without a tile takes
    // narrower tiles down to eight lines, and 512 threads to evaluate each. Unit-stride points want eight
    // lines too, so that a warp's segments of a line are whole sectors (512 cells x 16384 lines: 117 us
    // against 163 with 16 lines), unless the lines have so few chunks that the solve would keep but a warp
    // of the block (100 cells: 61 against 40). Feet are not read: sixteen lines (Greville cubics: 95
    // against 99).
    bool const unit = !FEET && fe.lo.stride == 1 && fe.lo.inner == 1 && fe.lo.outer > 1;
    io.lp = std::min(most_pairs(args.tile_req), unit && t.nchunk >= 16 ? 2 : 4);
    while (io.lp > 2 && (!fits(256, 2) || tiles() < int64_t(sms))) --io.lp;
    int threads = 256;
    if (!fits(256, 2) || tiles() <= int64_t(sms)) threads = 512;
    if (!fits(512, 1)) return false;
    bool const full = t.nchunk > 1 && t.chunk_len >= 15;
    auto kern = full ? reg_build_eval_kernel<K, 15, D, ORDER, FEET> : reg_build_eval_kernel<K, 0, D, ORDER, FEET>;
    size_t const sm = bytes();
    allow_shared(kern, sm);
    // resident blocks: 512 threads of 128 registers an SM, and the shared memory
    int64_t const per_sm = std::max<int64_t>(1, std::min<int64_t>(512 / threads, (optin + 1024) / int64_t(sm + 1024)));
    int64_t const grid = std::min<int64_t>(tiles(), per_sm * sms);
    kern<<<dim3((unsigned)grid), dim3((unsigned)threads), sm, s>>>(args, io, fe);
    DDCB_CUDA_CHECK(cudaGetLastError());
    return true;
}

template <int K, int D>
bool launch_reg_fused_d(BuildArgs const& args, FusedEval const& fe, int order, bool feet, cudaStream_t s)
{
    if (feet) return launch_reg_fused_kd<K, D, 0, true>(args, fe, s);
    if (order == 0) return launch_reg_fused_kd<K, D, 0, false>(args, fe, s);
    if (order == 1) return launch_reg_fused_kd<K, D, 1, false>(args, fe, s);
    return false;
}

} // namespace

bool launch_reg_fused(BuildArgs const& args, FusedEval const& fe, int order, bool feet, cudaStream_t s)
{
    if (args.t.rmax == 0 || fe.eb.b.uniform == 0) return false;
    // the bands of uniform meshes: one row either side up to degree 3, two up to degree 5
    switch (args.t.kl * 8 + fe.eb.b.degree) {
    case 9: return launch_reg_fused_d<1, 1>(args, fe, order, feet, s);
    case 10: return launch_reg_fused_d<1, 2>(args, fe, order, feet, s);
    case 11: return launch_reg_fused_d<1, 3>(args, fe, order, feet, s);
    case 20: return launch_reg_fused_d<2, 4>(args, fe, order, feet, s);
    case 21: return launch_reg_fused_d<2, 5>(args, fe, order, feet, s);
    default: return false;
    }
}

} // namespace ddcb
