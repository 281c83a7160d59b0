// tensor_items.cuh -- how the evaluators of two and more dimensions share out their work: items are
// (point, column) pairs, a column being one field or, where the layout allows 16-byte accesses, two
// neighbouring fields. Items are numbered point by point, so that few fields fill a warp with several
// points.
#pragma once

#include <algorithm>

#include "ddcb_internal.hpp"

namespace ddcb {

constexpr int kItemThreads = 256;
constexpr int kMostItems = 512; // of a block

// A block takes ppb consecutive points of hs of the H columns.
struct ItemGrid
{
    int ppb, H, hs;
    dim3 grid;
};

// Some 32 fields a block, so that the blocks in flight gather from as many: all 64 quintic fields of
// 512^2 do not fit the L2 (30000 points, each field its own: 343 us with 16 columns, 520 with 32). A
// thread takes one item until every SM has eight blocks, then two. In blocks of 2048 items, whatever
// the batch, one cubic field of 48^3 at 7000 points took 49 us (13 now) and 64 fields of 512^2 at
// a displaced mesh 162 (154).
inline ItemGrid item_grid(int64_t m, int64_t B, bool pair)
{
    ItemGrid g;
    g.H = int(pair ? B / 2 : B);
    int const most = pair && g.H <= 16 * 65535 ? 16 : 32; // (the grid's second dimension ends there)
    int const groups = std::max(1, (g.H + most / 2 - 1) / most); // equal ones: 33 columns are one group, not 32 and 1
    g.hs = (g.H + groups - 1) / groups;
    int64_t const each = (m * g.H + 8 * device_limits().sms - 1) / (8 * device_limits().sms);
    int64_t const items = std::min<int64_t>(kMostItems, std::max<int64_t>(1, (each + kItemThreads - 1) / kItemThreads) * kItemThreads);
    g.ppb = int(items) / g.hs;
    g.grid = dim3((unsigned)((m + g.ppb - 1) / g.ppb), (unsigned)((g.H + g.hs - 1) / g.hs));
    return g;
}

#if defined(__CUDACC__)

// f(point, column) for every item of the block. WARPS: for whole warps, f(live, point, column), with
// the lanes beyond the last item (live false) at some item of the block.
template <bool WARPS, class F>
__device__ __forceinline__ void for_items(int64_t m, int ppb, int H, int hs, F f)
{
    int const h0 = blockIdx.y * hs;
    hs = min(hs, H - h0);
    int64_t const p0 = (int64_t)blockIdx.x * ppb;
    int const np = int(min((int64_t)ppb, m - p0));
    int q = threadIdx.x / hs, h = threadIdx.x - q * hs;
    int const dq = kItemThreads / hs, dh = kItemThreads - dq * hs;
    while (WARPS ? __any_sync(0xffffffffu, q < np) : q < np) {
        if constexpr (WARPS) f(q < np, p0 + (q < np ? q : 0), h0 + h);
        else f(p0 + q, h0 + h);
        q += dq;
        h += dh;
        if (h >= hs) {
            h -= hs;
            ++q;
        }
    }
}

// The items of a warp over pairs of fields. Where all pairs share their point, a lane takes a pair: one
// basis, 16-byte loads. Where not, neighbouring lanes take the two fields of a pair, half of the warp's
// pairs after the other, so that a request still reads neighbouring fields. `at`: where the pair's first
// value goes; `shared`: whether its points coincide; one(to, field), both(at, column). UNROLL: the two
// halves' code side by side, 2 where its registers allow (uniform cubics: 64 fields on a displaced mesh
// of their own 207 us against 215, on a shared one 147 against 155; but irregular cubics, 64 fields at
// 30000 shared points, 55 against 45).
template <int UNROLL, class Both, class One>
__device__ __forceinline__ void pair_items(bool live, int64_t at, int h, bool shared, Both both, One one)
{
    constexpr unsigned kAll = 0xffffffffu;
    if (__all_sync(kAll, shared || !live)) {
        if (live) both(at, h);
        return;
    }
    int const lane = threadIdx.x & 31;
    at = live ? at : -1;
#pragma unroll UNROLL
    for (int half = 0; half < 32; half += 16) {
        int64_t const to = __shfl_sync(kAll, at, half + lane / 2);
        int const c = __shfl_sync(kAll, h, half + lane / 2);
        if (to >= 0) one(to + (lane & 1), 2 * c + (lane & 1));
    }
}

#endif

} // namespace ddcb
