// reg_solve.cuh -- the banded solve of build_device.cuh with the rows of a chunk in registers.
//
// A thread owns one chunk (at most kRegRows = 17 rows) of a pair of lines and runs all four sweeps
// on registers; only the carries between chunks (one barrier per direction) and the few rows that
// the border touches go through shared memory. Against sweeps over a shared-memory tile this
// removes the eight passes over the tile and most of the index arithmetic around them. The factor
// rows, the transfer matrices and the border's tables are copied to shared memory once per block
// (RegRecord), and blocks stay for many tiles: read through L1 instead, the tables of a 1024-cell
// irregular mesh missed often enough that the kernel took as long as the one it replaces (quintic,
// 65536 lines: 0.70 ms).
//
// The code of a tile is kept short on purpose (the sweeps are unrolled over the rows, everything
// else is loops): a warp runs it once per tile, and rarely taken unrolled paths cost the
// instruction cache more than they save.
//
// Why 17 rows and pairs: 17 rows of two lines are 68 registers, which with a window and the factor
// loads in flight fits 128 registers a thread, i.e. 16 warps per SM, each with two independent
// chains (the lines). A chunk this long lets the carries decay below rounding within two to four
// chunks up to degree 5. More rows spill; fewer spend their time on carries.
//
// The operations on a row are those of solve_in_tile in the same order, so both give the same bits.
#pragma once

#include "build_device.cuh"

namespace ddcb {

// W factor entries at p (16-byte aligned where W > 1).
template <int W>
__device__ __forceinline__ void load_factors(const double* p, double* f)
{
    if constexpr (W % 2 == 0) {
#pragma unroll
        for (int q = 0; q < W; q += 2) {
            double2 const v = *reinterpret_cast<const double2*>(p + q);
            f[q] = v.x;
            f[q + 1] = v.y;
        }
    } else {
        static_assert(W == 1, "records are padded to 16-byte vectors");
        f[0] = *p;
    }
}

// The first row and the row count of chunk c (c < nchunk).
__device__ __forceinline__ void chunk_rows(SolveTables const& t, int c, int& a, int& len)
{
    a = c * t.chunk_len + 2 * max(0, c - t.chunk_split);
    len = (c == t.nchunk - 1 ? t.m : a + t.chunk_len + (c >= t.chunk_split ? 2 : 0)) - a;
}

// Shared memory of the solve for P line pairs, in doubles: the records, the border block, the
// forward and backward carries, the rows lambda reads, b2 and x2.
template <int K>
__host__ __device__ inline size_t reg_smem_doubles(SolveTables const& t, int P)
{
    constexpr RegRecord L(K);
    return size_t(t.nchunk) * L.size + size_t(reg_border_size(t))
           + size_t(2 * P) * (size_t(t.nchunk) * (2 * K) + size_t(t.lam_lo + t.lam_hi + 2 * t.k));
}

struct RegSmem
{
    double* rec;     // nchunk records
    double* bord;    // the border block
    double2* carry;  // forward, then backward carries: nchunk * K * P each
    double2* ends;   // the rows lambda reads, P pairs each
    double2* b2;     // k rows
    double2* x2;     // k rows
    double* end;
};

template <int K>
__device__ __forceinline__ RegSmem reg_smem(SolveTables const& t, int P, double* smem)
{
    constexpr RegRecord L(K);
    RegSmem s;
    s.rec = smem;
    s.bord = smem + t.nchunk * L.size;
    s.carry = reinterpret_cast<double2*>(s.bord + reg_border_size(t));
    s.ends = s.carry + t.nchunk * (2 * K) * P;
    s.b2 = s.ends + (t.lam_lo + t.lam_hi) * P;
    s.x2 = s.b2 + t.k * P;
    s.end = reinterpret_cast<double*>(s.x2 + t.k * P);
    return s;
}

// Starts the copy of the records and the border block (the caller waits for it).
template <int K>
__device__ __forceinline__ void reg_load_tables(SolveTables const& t, RegSmem const& sm)
{
    constexpr RegRecord L(K);
    for (int i = threadIdx.x; i < t.nchunk * (L.size / 2); i += blockDim.x) cp_async16(sm.rec + 2 * i, t.reg + 2 * i);
    for (int i = threadIdx.x; i < reg_border_size(t) / 2; i += blockDim.x) cp_async16(sm.bord + 2 * i, t.regb + 2 * i);
}

// Forward and backward sweeps of chunk c (thread-owned rows x[0 .. len-1], zero beyond) of line pair
// p of P. Threads beyond the last chunk (c >= nchunk) run along on a copy of the last one: they take
// part in the barriers and write nothing. MINLEN: 15 where no chunk is shorter, so only the last two
// steps need a test; 0 for any chunks. Every thread of the block calls it. Ends without a barrier:
// x holds the solution of Q x' = b.
template <int K, int MINLEN>
__device__ __forceinline__ void reg_sweeps(SolveTables const& t, RegSmem const& sm, double2* x, int len, int c, int p, int P)
{
    constexpr int R = kRegRows;
    constexpr RegRecord L(K);
    constexpr int LW = L.LW, UW = L.UW;
    int const NC = t.nchunk;
    int const cc = min(c, NC - 1);
    const double* const rl = sm.rec + cc * L.size;
    const double* const ru = rl + L.U;
    double2* const cf = sm.carry + p;
    double2* const cb = sm.carry + (size_t)NC * K * P + p;
    double2 const zero = make_double2(0.0, 0.0);
    if (NC > 1) {
        double2 w[K + 1];
#pragma unroll
        for (int q = 0; q < K; ++q) w[q] = x[q];
#pragma unroll
        for (int s = 0; s < R; ++s) {
            if (MINLEN > 0 ? (s == MINLEN && len <= s) : s >= len) break;
            double f[LW];
            load_factors<LW>(rl + s * LW, f);
            w[K] = s + K < R ? x[s + K] : zero;
            double2 const y = w[0];
#pragma unroll
            for (int q = 1; q <= K; ++q) w[q - 1] = fma2(-f[q - 1], y, w[q]);
        }
        if (c < NC) {
#pragma unroll
            for (int q = 0; q < K; ++q) cf[(c * K + q) * P] = w[q];
        }
        __syncthreads();
        if (c > 0) {
            double2 in[K];
            carry_direct<double2, K, K, true>([&](int b, int e) { return sm.rec[b * L.size + L.F + e]; }, cf, P, t.ndep_f, NC, cc - 1, in);
#pragma unroll
            for (int q = 0; q < K; ++q) x[q] = add2(x[q], in[q]);
        }
    }
#pragma unroll
    for (int s = 0; s < R; ++s) {
        if (MINLEN > 0 ? (s == MINLEN && len <= s) : s >= len) break;
        double f[LW];
        load_factors<LW>(rl + s * LW, f);
#pragma unroll
        for (int q = 1; q <= K; ++q)
            if (s + q < R) x[s + q] = fma2(-f[q - 1], x[s], x[s + q]);
    }
    double2 z[K];
#pragma unroll
    for (int q = 0; q < K; ++q) z[q] = zero;
    auto back = [&](int s) { // row s: the solution given the K rows after it
        double f[UW];
        load_factors<UW>(ru + s * UW, f);
        double2 v = x[s];
#pragma unroll
        for (int q = K; q >= 1; --q) v = fma2(-f[q], z[q - 1], v);
#pragma unroll
        for (int q = K - 1; q >= 1; --q) z[q] = z[q - 1];
        z[0] = mul2(v, f[0]);
    };
    constexpr int TOP = MINLEN > 0 ? MINLEN : R;
    if (NC > 1) {
        if (MINLEN > 0 && len > MINLEN) {
#pragma unroll
            for (int s = R - 1; s >= TOP; --s) back(s);
        }
#pragma unroll
        for (int s = TOP - 1; s >= 0; --s)
            if (MINLEN > 0 || s < len) back(s);
        if (c < NC) {
#pragma unroll
            for (int q = 0; q < K; ++q) cb[(c * K + q) * P] = z[q];
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < K; ++q) z[q] = zero;
        if (cc + 1 < NC)
            carry_direct<double2, K, K, false>([&](int b, int e) { return sm.rec[b * L.size + L.B + e]; }, cb, P, t.ndep_b, NC, cc + 1, z);
    }
    if (MINLEN > 0 && len > MINLEN) {
#pragma unroll
        for (int s = R - 1; s >= TOP; --s) {
            back(s);
            x[s] = z[0];
        }
    }
#pragma unroll
    for (int s = TOP - 1; s >= 0; --s)
        if (MINLEN > 0 || s < len) {
            back(s);
            x[s] = z[0];
        }
}

// Border: x2 = S^-1 (b2 - lambda x'), x1 = x' - (Q^-1 gamma) x2. The owners of the rows that lambda
// reads hand them over through shared memory, b2 is there already (written before one of the
// barriers of reg_sweeps, or before this call). Eight lanes of one warp compute a pair's x2, so its
// two steps need no block barrier, and the owners correct their rows in registers, row by row of x2
// as solve_in_tile does. The tables come from shared memory: these short chains would wait for the
// L2 at every step. On return x holds the solution, and x2 (all k rows) is complete.
__device__ __forceinline__ void reg_border(SolveTables const& t, RegSmem const& sm, double2* x, int a, int len, int c, int p, int P)
{
    int const k = t.k, nc = t.cor_lo + t.cor_hi;
    int const lo = t.lam_lo, hi0 = t.m - t.lam_hi;
    constexpr int W = kRegRows + 1;
    if (c < t.nchunk && (a < lo || a + len > hi0)) {
        double2* const E = sm.ends + p;
#pragma unroll
        for (int s = 0; s < kRegRows; ++s) {
            if (a + s >= lo || s >= len) break;
            E[DDCB_INDEX(a + s, lo + t.lam_hi) * P] = x[s];
        }
#pragma unroll
        for (int s = kRegRows - 1; s >= 0; --s) {
            if (s >= len) continue;
            if (a + s < hi0) break;
            if (a + s >= lo) E[DDCB_INDEX(lo + a + s - hi0, lo + t.lam_hi) * P] = x[s];
        }
    }
    __syncthreads();
    const double* const Sinv = sm.bord + nc * k * W;
    unsigned const lanes = P >= 4 ? 0xffffffffu : (1u << (kRegMaxBorder * P)) - 1u; // whole warps, or part of one
    for (int u = threadIdx.x; u < kRegMaxBorder * P; u += blockDim.x) {
        int const q = u / kRegMaxBorder, r = u % kRegMaxBorder;
        const double* const lam = Sinv + k * k;
        const int* const lam_row = reinterpret_cast<const int*>(lam + t.lam_nnz);
        const int* const lam_end = lam_row + k + 1;
        double2* const b2 = sm.b2 + q;
        if (r < k) {
            double2 s = b2[r * P];
            int const j1 = lam_row[r + 1];
#pragma unroll 4
            for (int j = lam_row[r]; j < j1; ++j) s = fma2(-lam[j], sm.ends[DDCB_INDEX(lam_end[j], t.lam_lo + t.lam_hi) * P + q], s);
            b2[r * P] = s;
        }
        __syncwarp(lanes);
        if (r < k) {
            double2 s = make_double2(0.0, 0.0);
#pragma unroll 4
            for (int j = 0; j < k; ++j) s = fma2(Sinv[r * k + j], b2[j * P], s);
            sm.x2[r * P + q] = s;
        }
    }
    __syncthreads();
    int const e = c < t.cor_lo ? c : c - (t.nchunk - nc);
    if (c < t.nchunk && (c < t.cor_lo || c >= t.nchunk - t.cor_hi)) {
        const double* g = sm.bord + DDCB_INDEX(e, nc) * k * W;
#pragma unroll 1
        for (int r = 0; r < k; ++r, g += W) {
            double2 const v = sm.x2[r * P + p];
#pragma unroll
            for (int s = 0; s < kRegRows; s += 2) {
                double2 const f = *reinterpret_cast<const double2*>(g + s);
                x[s] = fma2(-f.x, v, x[s]);
                if (s + 1 < kRegRows) x[s + 1] = fma2(-f.y, v, x[s + 1]);
            }
        }
    }
}

} // namespace ddcb
