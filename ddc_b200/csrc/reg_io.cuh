// reg_io.cuh -- how the register solve's rows come from the inputs and go to the coefficients.
//
// Inputs pass through a shared-memory tile (row r of line l at tile[r * TL + l]), filled by
// asynchronous copies while the previous tile is being solved: 16-byte copies of line pairs where the
// layout allows, else 8-byte ones. Coefficients of lines with the batch contiguous are written
// straight from the registers of the thread that owns the rows: lanes next to each other hold lines
// next to each other. Unit-stride lines would scatter those stores over one sector per lane; their
// coefficients go back through the tile and leave in whole sectors.
//
// The width of the tile matters more than anything else here: copying 1029 rows of 65536 lines
// through such tiles, and nothing more, takes 570 us with 4 lines (32-byte row segments), 250 us with
// 8, 205 us with 16 and 193 us with 32.
#pragma once

#include "reg_solve.cuh"

namespace ddcb {

struct RegIo
{
    int lp;         // log2 of the line pairs per block
    int stage_out;  // unit-stride coefficients: through the tile
    int v0;         // row 0 of Q is system row lrot, sample lrot - v0 (the rows of Q are all samples)
};

// Whether every row of Q is a sample, one after the other (row 0 being sample lrot - v0).
inline bool reg_plain_rows(BuildArgs const& args)
{
    bool const all = args.raw || args.r.periodic;
    int const v0 = all ? 0 : args.r.nbe_lo, v1 = all ? args.t.n : args.r.nbe_lo + args.r.npoints;
    return args.r.lrot >= v0 && args.r.lrot + args.t.m <= v1;
}

// The source of border row r (tile row m + r) of a line: a sample, a Hermite derivative, or none
// (homogeneous conditions), and the power of dx that scales it.
__device__ __forceinline__ const double* border_source(BuildArgs const& args, int r, int64_t line)
{
    RhsMap const& R = args.r;
    int const n = args.t.n;
    bool const all = args.raw || R.periodic;
    int const v0 = all ? 0 : R.nbe_lo, v1 = all ? n : R.nbe_lo + R.npoints;
    int sr = args.t.m + r + R.lrot;
    sr -= (sr >= n) ? n : 0;
    if (sr >= v0 && sr < v1) return args.vals + (int64_t)DDCB_INDEX(sr - v0, v1 - v0) * args.lv.stride + line_offset(args.lv, line);
    if (sr < R.nbe_lo) return sr < R.nbv_lo ? args.dlo + sr * args.llo.stride + line_offset(args.llo, line) : nullptr;
    int const i = sr - (n - R.nbe_hi);
    return i < R.nbv_hi ? args.dhi + i * args.lhi.stride + line_offset(args.lhi, line) : nullptr;
}

__device__ __forceinline__ double border_scale(BuildArgs const& args, int r)
{
    RhsMap const& R = args.r;
    int const n = args.t.n;
    if (args.raw || R.periodic) return 1.0;
    int sr = args.t.m + r + R.lrot;
    sr -= (sr >= n) ? n : 0;
    if (sr < R.nbe_lo) return R.dxpow_lo[sr];
    int const i = sr - (n - R.nbe_hi);
    return i >= 0 ? R.dxpow_hi[i] : 1.0;
}

// Starts the copies of a tile: the rows of Q of lines line0 .. into `tile`, and the border rows as
// they are (unscaled) into `raw`. Lines past the end repeat the last one (the last pair).
__device__ __forceinline__ void reg_fill(BuildArgs const& args, RegIo const& io, int64_t line0, double* tile, double* raw)
{
    int const TL = 2 << io.lp;
    int const m = args.t.m;
    int64_t const st = args.lv.stride;
    int const first = args.r.lrot - io.v0; // the sample of row 0
    const double* const vals = args.vals + (int64_t)first * st;
    [[maybe_unused]] int const samples = args.raw ? args.t.n : args.r.npoints;
    if (args.pair16) {
        int const P = 1 << io.lp;
        int const p = threadIdx.x & (P - 1);
        int const step = blockDim.x >> io.lp;
        int const r0 = threadIdx.x >> io.lp;
        int64_t const line = min(line0 + 2 * p, args.nlines - 2);
        const double* g = vals + r0 * st + line_offset(args.lv, line);
        int64_t const gs = step * st;
        double* s = tile + r0 * TL + 2 * p;
        for (int r = r0; r < m; r += step) {
            cp_async16(s, DDCB_ROW(g, args.vals + line_offset(args.lv, line), first + r, samples, st));
            g += gs;
            s += step * TL;
        }
    }
    int const l = threadIdx.x & (TL - 1);
    int const step = blockDim.x / TL;
    int const r0 = threadIdx.x / TL;
    int64_t const line = min(line0 + l, args.nlines - 1);
    if (!args.pair16) {
        const double* g = vals + r0 * st + line_offset(args.lv, line);
        int64_t const gs = step * st;
        double* s = tile + r0 * TL + l;
        for (int r = r0; r < m; r += step) {
            cp_async8(s, DDCB_ROW(g, args.vals + line_offset(args.lv, line), first + r, samples, st));
            g += gs;
            s += step * TL;
        }
    }
    for (int r = r0; r < args.t.k; r += step) {
        const double* const g = border_source(args, r, line);
        if (g) cp_async8(raw + r * TL + l, g);
        else raw[r * TL + l] = 0.0;
    }
}

// The rows [a, a + len) of pair p from the tile into x (zero beyond len).
__device__ __forceinline__ void reg_load(RegIo const& io, const double* tile, int a, int len, int p, double2* x)
{
    int const TL = 2 << io.lp;
    const double* const s0 = tile + a * TL + 2 * p;
#pragma unroll
    for (int s = 0; s < kRegRows; ++s) x[s] = s < len ? *reinterpret_cast<const double2*>(s0 + s * TL) : make_double2(0.0, 0.0);
}

// b2 of pair p from the raw border rows.
__device__ __forceinline__ void reg_border_rhs(BuildArgs const& args, RegSmem const& sm, const double* raw, int c, int p, int P)
{
    int const nthr = blockDim.x / P;
    for (int r = c; r < args.t.k; r += nthr) sm.b2[r * P + p] = mul2(*reinterpret_cast<const double2*>(raw + r * (2 * P) + 2 * p), border_scale(args, r));
}

// One border row of the solution (tile order) of a pair to its coefficient row and to the row a
// period further that repeats it: in the tile, or in the coefficients of lines `line`, `line` + 1.
__device__ __forceinline__ void reg_store_row(BuildArgs const& args, RegIo const& io, bool to_tile, int64_t line, double* tile, int row,
                                              int p, double2 v)
{
    int const n = args.t.n;
    int const rows = args.raw ? n : args.r.size;
    int o = row + args.r.srot;
    o -= (o >= n) ? n : 0;
    o += (o < 0) ? n : 0;
    for (o = DDCB_INDEX(o, n); o < rows; o += n) {
        if (to_tile) {
            *reinterpret_cast<double2*>(tile + o * (2 << io.lp) + 2 * p) = v;
        } else if (line < args.nlines) {
            double* const g = args.out + (int64_t)o * args.lo.stride;
            __stcs(g + line_offset(args.lo, line), v.x);
            if (line + 1 < args.nlines) __stcs(g + line_offset(args.lo, line + 1), v.y);
        }
    }
}

// The rows [a, a + len) of the solution to the tile, in coefficient order: rows a + srot .., from n on
// those from 0 on (the wrap of a periodic basis); rows below `dup` are repeated n rows further.
__device__ __forceinline__ void reg_store_tile(BuildArgs const& args, RegIo const& io, double* tile, int a, int len, int p,
                                               const double2* x)
{
    int const n = args.t.n;
    int const dup = (args.raw ? n : args.r.size) - n;
    int o = a + args.r.srot;
    o += (o < 0) ? n : 0;
    int const TL = 2 << io.lp;
    double* const t0 = tile + 2 * p;
#pragma unroll
    for (int s = 0; s < kRegRows; ++s)
        if (s < len) {
            int const q = DDCB_INDEX(o + s - (o + s >= n ? n : 0), n);
            *reinterpret_cast<double2*>(t0 + q * TL) = x[s];
            if (q < dup) *reinterpret_cast<double2*>(t0 + (q + n) * TL) = x[s];
        }
}

// The same rows to the coefficients of lines `line`, `line` + 1. Only the chunks at the ends wrap or
// repeat, so the others are spared it.
__device__ __forceinline__ void reg_store(BuildArgs const& args, int64_t line, int a, int len, const double2* x)
{
    constexpr int R = kRegRows;
    int const n = args.t.n;
    int const dup = (args.raw ? n : args.r.size) - n;
    int o = a + args.r.srot;
    o += (o < 0) ? n : 0;
    if (line >= args.nlines) return;
    int64_t const st = args.lo.stride;
    double* const base = args.out + line_offset(args.lo, line);
    bool const two = line + 1 < args.nlines;
    int64_t const next = two ? line_offset(args.lo, line + 1) - line_offset(args.lo, line) : 0;
    if (o >= dup && o + len <= n) {
        double* g = base + (int64_t)o * st;
        if (args.pair16_out) {
#pragma unroll
            for (int s = 0; s < R; ++s) {
                if (s < len) __stcs(reinterpret_cast<double2*>(DDCB_ROW(g, base, o + s, n, st)), x[s]);
                g += st;
            }
        } else {
#pragma unroll
            for (int s = 0; s < R; ++s) {
                if (s < len) {
                    double* const to = DDCB_ROW(g, base, o + s, n, st);
                    __stcs(to, x[s].x);
                    if (two) __stcs(to + next, x[s].y);
                }
                g += st;
            }
        }
        return;
    }
#pragma unroll
    for (int s = 0; s < R; ++s)
        if (s < len) {
            int const q = DDCB_INDEX(o + s - (o + s >= n ? n : 0), n);
            double* const g = base + (int64_t)q * st;
            double* const g2 = q < dup ? g + n * st : g;
            if (args.pair16_out) {
                __stcs(reinterpret_cast<double2*>(g), x[s]);
                if (q < dup) __stcs(reinterpret_cast<double2*>(g2), x[s]);
            } else {
                __stcs(g, x[s].x);
                if (q < dup) __stcs(g2, x[s].x);
                if (two) __stcs(g + next, x[s].y);
                if (two && q < dup) __stcs(g2 + next, x[s].y);
            }
        }
}

// The tile's rows (coefficient order) to the coefficients.
__device__ __forceinline__ void reg_drain(BuildArgs const& args, RegIo const& io, int64_t line0, const double* tile)
{
    int const TL = 2 << io.lp;
    int const rows = args.raw ? args.t.n : args.r.size;
    int const l = threadIdx.x & (TL - 1);
    int const step = blockDim.x / TL;
    if (line0 + l >= args.nlines) return;
    int64_t const st = args.lo.stride;
    double* g = args.out + line_offset(args.lo, line0 + l);
    for (int r = threadIdx.x / TL; r < rows; r += step) __stcs(g + r * st, tile[r * TL + l]);
}

} // namespace ddcb
