// reg_adjoint_kernels.cu -- the backward of build + evaluate (adjoint_kernels.cu) on uniform bases in
// one pass over the points, with the transposed solve in registers (reg_solve.cuh).
//
// The two-pass kernel reads every point twice, once for the coordinate cotangents against the
// coefficient tile and once for the scatter into the tile that replaces it. Here both tiles are in
// shared memory (1024 rows of eight lines: 2 x 66 KB and the solve's tables, one block of 512
// threads per SM), so a point is located once, its degree D and D - 1 values come from one recurrence, and
// the coordinates and cotangents of the next points are on their way meanwhile. The coefficients of
// the block's next tile are copied during the solve.
#include <algorithm>

#include "adjoint_args.hpp"
#include "reg_io.cuh"

namespace ddcb {

namespace {

// Starts the copy of the coefficient tile: row r of line l at tile[r * TL + l].
__device__ __forceinline__ void coef_fill(EvalAdjointArgs const& ea, int lp, int64_t line0, double* tile)
{
    int const TL = 2 << lp;
    if (ea.coef_pairs) {
        int const p = threadIdx.x & ((1 << lp) - 1);
        int const step = blockDim.x >> lp;
        int64_t const line = min(line0 + 2 * p, ea.nlines - 2);
        int r = threadIdx.x >> lp;
        const double* g = ea.coefs + r * ea.lc.stride + line_offset(ea.lc, line);
        for (; r < ea.size; r += step) {
            cp_async16(tile + r * TL + 2 * p, g);
            g += step * ea.lc.stride;
        }
        return;
    }
    int const l = threadIdx.x & (TL - 1);
    int const step = blockDim.x / TL;
    int64_t const line = min(line0 + l, ea.nlines - 1);
    int r = threadIdx.x / TL;
    const double* g = ea.coefs + r * ea.lc.stride + line_offset(ea.lc, line);
    for (; r < ea.size; r += step) {
        cp_async8(tile + r * TL + l, g);
        g += step * ea.lc.stride;
    }
}

// Weights dy/dc (times `scale`, multiplied into w by the caller's cotangent) and dy/dx of a point.
// Returns the first B-spline, or -1 where y is identically 0.
template <int D, int ORDER>
__device__ __forceinline__ int adjoint_point(EvalAdjointArgs const& ea, double x, const double* C, int TL, bool want_dx, double* w,
                                             double& scale, double& dydx)
{
    if constexpr (ORDER == 0) {
        bool fixed = false; // constant extrapolation: y does not move with x
        BasisDesc const& b = ea.eb.b;
        dydx = 0.0;
        if (b.periodic) {
            x = periodic_wrap(b, x);
        } else if (x < b.rmin || x > b.rmax) {
            if ((x < b.rmin ? ea.ex_lo : ea.ex_hi) == 1) return -1;
            fixed = true;
        }
        double off, low[D > 1 ? D : 1];
        int const j = DDCB_INDEX(uniform_cell_select(b, x, off), b.ncells);
        uniform_values_raw2<D>(off, w, low);
        scale = factorial_inverse(D);
        if (want_dx && !fixed) {
            double y = 0.0, cp = C[j * TL];
#pragma unroll
            for (int i = 1; i <= D; ++i) {
                double const ci = C[(j + i) * TL];
                y = fma(ci - cp, low[i - 1], y);
                cp = ci;
            }
            dydx = y * (b.inv_step * factorial_inverse(D - 1));
        }
        return j;
    } else {
        scale = 1.0;
        return point_adjoint<D, ORDER, true>(ea.eb, ea.ex_lo, ea.ex_hi, x, CoefDirect {C, TL}, want_dx, w, dydx);
    }
}

// Rows [a, a + len) of the transposed solve to the sample cotangents they belong to (samples
// a + first ..).
__device__ __forceinline__ void reg_store_samples(AdjointArgs const& a, int64_t line, int first, int len, const double2* x)
{
    if (line >= a.nlines) return;
    int64_t const st = a.lgv.stride;
    double* g = a.gv + first * st + line_offset(a.lgv, line);
    [[maybe_unused]] double* const base = a.gv + line_offset(a.lgv, line);
    if (a.pair_out) {
#pragma unroll
        for (int s = 0; s < kRegRows; ++s) {
            if (s < len) __stcs(reinterpret_cast<double2*>(DDCB_ROW(g, base, first + s, a.r.npoints, st)), x[s]);
            g += st;
        }
        return;
    }
    bool const two = line + 1 < a.nlines;
    int64_t const next = two ? line_offset(a.lgv, line + 1) - line_offset(a.lgv, line) : 0;
#pragma unroll
    for (int s = 0; s < kRegRows; ++s) {
        if (s < len) {
            double* const to = DDCB_ROW(g, base, first + s, a.r.npoints, st);
            __stcs(to, x[s].x);
            if (two) __stcs(to + next, x[s].y);
        }
        g += st;
    }
}

// Border row (system row sr) of one line: a sample, or a Hermite derivative times its dx^k.
__device__ __forceinline__ void store_border(AdjointArgs const& a, int sr, int64_t line, double g)
{
    RhsMap const& R = a.r;
    int const n = a.t.n;
    if (line >= a.nlines) return;
    int const v0 = R.periodic ? 0 : R.nbe_lo, v1 = R.periodic ? n : R.nbe_lo + R.npoints;
    if (sr >= v0 && sr < v1) {
        a.gv[(int64_t)(sr - v0) * a.lgv.stride + line_offset(a.lgv, line)] = g;
    } else if (sr < v0) {
        if (sr < R.nbv_lo && a.gdlo) a.gdlo[sr * a.lglo.stride + line_offset(a.lglo, line)] = g * R.dxpow_lo[sr];
    } else {
        int const q = sr - (n - R.nbe_hi);
        if (q < R.nbv_hi && a.gdhi) a.gdhi[q * a.lghi.stride + line_offset(a.lghi, line)] = g * R.dxpow_hi[q];
    }
}

template <int K, int MINLEN, int D, int ORDER>
__global__ void __launch_bounds__(512, 1) reg_adjoint_kernel(const __grid_constant__ AdjointArgs args,
                                                             const __grid_constant__ EvalAdjointArgs ea, int lp)
{
    extern __shared__ __align__(16) double smem[];
    SolveTables const& t = args.t;
    int const P = 1 << lp, TL = 2 * P;
    int const p = threadIdx.x & (P - 1);
    int const c = threadIdx.x >> lp;
    int const nthr = blockDim.x >> lp;
    RegSmem const sm = reg_smem<K>(t, P, smem);
    double* const T = sm.end;                  // n rows: cotangents, then the solve's right-hand side
    double* const C = T + (size_t)t.n * TL;    // size rows: coefficients (gx only)
    bool const want = ea.gx != nullptr;
    int a, len;
    chunk_rows(t, min(c, t.nchunk - 1), a, len);
    int64_t const tiles = (args.nlines + TL - 1) >> (lp + 1);
    int const l = threadIdx.x & (TL - 1);
    int const q0 = threadIdx.x / TL;
    int const nct = blockDim.x / TL;
    int const m = int(ea.lx.n);
    int const npt = m > q0 ? (m - q0 + nct - 1) / nct : 0;
    int const v0 = args.r.periodic ? 0 : args.r.nbe_lo;
    reg_load_tables<K>(t, sm);
    if (want) coef_fill(ea, lp, (int64_t)blockIdx.x << (lp + 1), C);
    double2* const T2 = reinterpret_cast<double2*>(T);
    for (int i = threadIdx.x; i < t.n * P; i += blockDim.x) T2[i] = make_double2(0.0, 0.0);
    for (int64_t ti = blockIdx.x; ti < tiles; ti += gridDim.x) {
        int64_t const line0 = ti << (lp + 1);
        {
            int64_t const line = min(line0 + l, args.nlines - 1);
            bool const live = line0 + l < args.nlines;
            const double* __restrict__ xp = ea.coords + line_offset(ea.lx, line) + q0 * ea.lx.stride;
            const double* __restrict__ gp = ea.gy + line_offset(ea.lgy, line) + q0 * ea.lgy.stride;
            double* __restrict__ ox = want ? ea.gx + line_offset(ea.lgx, line) + q0 * ea.lgx.stride : nullptr;
            int64_t const sx = ea.lx.stride * nct, sg = ea.lgy.stride * nct, so = want ? ea.lgx.stride * nct : 0;
            constexpr int U = 4; // points of a group
            auto load = [&](int i, double* xs, double* gs) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    xs[u] = i + u < npt ? __ldcs(xp + (i + u) * sx) : 0.0;
                    gs[u] = i + u < npt ? __ldcs(gp + (i + u) * sg) : 0.0;
                }
            };
            double xs[U], gs[U];
            load(0, xs, gs);
            cp_async_wait_all();
            __syncthreads();
            if (live)
                for (int i = 0; i < npt; i += U) {
                    double xn[U], gn[U];
                    load(i + U, xn, gn);
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (i + u >= npt) continue;
                        double w[D + 1], scale, dydx = 0.0;
                        int const j = adjoint_point<D, ORDER>(ea, xs[u], C + l, TL, want, w, scale, dydx);
                        if (want) __stcs(ox + (i + u) * so, gs[u] * dydx);
                        if (j >= 0) {
                            double const g = gs[u] * scale;
                            int r = j - args.r.srot;
                            r += r < 0 ? t.n : 0;
                            r -= r >= t.n ? t.n : 0;
#pragma unroll
                            for (int k = 0; k < D + 1; ++k) {
                                int const q = r + k - (r + k >= t.n ? t.n : 0);
                                atomicAdd(T + DDCB_INDEX(q, t.n) * TL + l, g * w[k]);
                            }
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        xs[u] = xn[u];
                        gs[u] = gn[u];
                    }
                }
        }
        __syncthreads();
        if (want && ti + gridDim.x < tiles) coef_fill(ea, lp, (ti + gridDim.x) << (lp + 1), C);
        double2 x[kRegRows];
#pragma unroll
        for (int s = 0; s < kRegRows; ++s) x[s] = s < len ? T2[(a + s) * P + p] : make_double2(0.0, 0.0);
        for (int r = c; r < t.k; r += nthr) sm.b2[r * P + p] = T2[(t.m + r) * P + p];
        __syncthreads(); // the right-hand side has been read
        if (ti + gridDim.x < tiles)
            for (int i = threadIdx.x; i < t.n * P; i += blockDim.x) T2[i] = make_double2(0.0, 0.0);
        reg_sweeps<K, MINLEN>(t, sm, x, len, c, p, P);
        if (t.k > 0) reg_border(t, sm, x, a, len, c, p, P);
        int64_t const line = line0 + 2 * p;
        if (c < t.nchunk) reg_store_samples(args, line, a + args.r.lrot - v0, len, x);
        for (int r = c; r < t.k; r += nthr) {
            int sr = t.m + r + args.r.lrot;
            sr -= sr >= t.n ? t.n : 0;
            double2 const g = sm.x2[r * P + p];
            store_border(args, sr, line, g.x);
            store_border(args, sr, line + 1, g.y);
        }
    }
}

template <int K, int D, int ORDER>
bool launch_kd(AdjointArgs const& a, EvalAdjointArgs const& ea, cudaStream_t s)
{
    SolveTables const& t = a.t;
    int const v0 = a.r.periodic ? 0 : a.r.nbe_lo, v1 = a.r.periodic ? t.n : a.r.nbe_lo + a.r.npoints;
    if (a.r.lrot < v0 || a.r.lrot + t.m > v1 || ea.lx.n > (int64_t(1) << 30)) return false;
    int const optin = device_limits().optin, sms = device_limits().sms;
    int lp = std::min(most_pairs(a.tile_req), 3);
    auto bytes = [&] { return sizeof(double) * (reg_smem_doubles<K>(t, 1 << lp) + size_t(t.n + ea.size) * size_t(2 << lp)); };
    auto fits = [&](int threads, int blocks) { return (t.nchunk << lp) <= threads && bytes() + 1024 <= (size_t(optin) + 1024) / blocks; };
    auto tiles = [&] { return (a.nlines + (int64_t(2) << lp) - 1) >> (lp + 1); };
    // sixteen lines or eight; two blocks of 256 threads where they fit, else one of 512
    while (lp > 2 && (!fits(512, 1) || tiles() < int64_t(sms))) --lp;
    int const threads = fits(256, 2) && tiles() > int64_t(sms) ? 256 : 512;
    if (!fits(512, 1)) return false;
    bool const full = t.nchunk > 1 && t.chunk_len >= 15;
    auto kern = full ? reg_adjoint_kernel<K, 15, D, ORDER> : reg_adjoint_kernel<K, 0, D, ORDER>;
    size_t const sm = bytes();
    allow_shared(kern, sm);
    // resident blocks: 512 threads of 128 registers an SM, and the shared memory
    int64_t const per_sm = std::max<int64_t>(1, std::min<int64_t>(512 / threads, (optin + 1024) / int64_t(sm + 1024)));
    int64_t const grid = std::min<int64_t>(tiles(), per_sm * sms);
    kern<<<dim3((unsigned)grid), dim3((unsigned)threads), sm, s>>>(a, ea, lp);
    DDCB_CUDA_CHECK(cudaGetLastError());
    return true;
}

template <int K, int D>
bool launch_d(AdjointArgs const& a, EvalAdjointArgs const& ea, int order, cudaStream_t s)
{
    if (order == 0) return launch_kd<K, D, 0>(a, ea, s);
    if (order == 1) return launch_kd<K, D, 1>(a, ea, s);
    return false;
}

} // namespace

bool launch_reg_adjoint(AdjointArgs const& a, EvalAdjointArgs const& ea, int order, cudaStream_t s)
{
    if (a.t.rmax == 0 || ea.eb.b.uniform == 0) return false;
    // the bands of uniform meshes: one row either side up to degree 3, two up to degree 5
    switch (a.t.kl * 8 + ea.eb.b.degree) {
    case 9: return launch_d<1, 1>(a, ea, order, s);
    case 10: return launch_d<1, 2>(a, ea, order, s);
    case 11: return launch_d<1, 3>(a, ea, order, s);
    case 20: return launch_d<2, 4>(a, ea, order, s);
    case 21: return launch_d<2, 5>(a, ea, order, s);
    default: return false;
    }
}

} // namespace ddcb
