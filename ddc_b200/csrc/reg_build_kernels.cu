// reg_build_kernels.cu -- the batched builder with its solve in registers (reg_solve.cuh): blocks of
// 2 P lines, P chosen by the chunk count and the batch. A block stays for several tiles of lines: its
// copy of the factor records is paid once, and the copies of the next tile run while it solves.
#include <algorithm>

#include "reg_io.cuh"

namespace ddcb {

namespace {

// At most 512 threads of 128 registers per SM.
template <int K, int MINLEN>
__global__ void __launch_bounds__(512, 1) reg_build_kernel(const __grid_constant__ BuildArgs args, const __grid_constant__ RegIo io)
{
    extern __shared__ __align__(16) double smem[];
    SolveTables const& t = args.t;
    int const P = 1 << io.lp, TL = 2 * P;
    int const p = threadIdx.x & (P - 1);
    int const c = threadIdx.x >> io.lp;
    int const nthr = blockDim.x >> io.lp;
    RegSmem const sm = reg_smem<K>(t, P, smem);
    double* const raw = sm.end; // border rows
    double* const tile = raw + t.k * TL;
    int a, len;
    chunk_rows(t, min(c, t.nchunk - 1), a, len);
    int64_t const tiles = (args.nlines + TL - 1) >> (io.lp + 1);
    reg_load_tables<K>(t, sm);
    reg_fill(args, io, (int64_t)blockIdx.x << (io.lp + 1), tile, raw);
    for (int64_t ti = blockIdx.x; ti < tiles; ti += gridDim.x) {
        int64_t const line0 = ti << (io.lp + 1);
        int64_t const line = line0 + 2 * p;
        cp_async_wait_all();
        __syncthreads();
        double2 x[kRegRows];
        reg_load(io, tile, a, len, p, x);
        if (t.k > 0) reg_border_rhs(args, sm, raw, c, p, P);
        __syncthreads(); // the tile has been read
        if (!io.stage_out && ti + gridDim.x < tiles)
            reg_fill(args, io, (ti + gridDim.x) << (io.lp + 1), tile, raw);
        reg_sweeps<K, MINLEN>(t, sm, x, len, c, p, P);
        if (t.k > 0) reg_border(t, sm, x, a, len, c, p, P);
        if (c < t.nchunk) {
            if (io.stage_out) reg_store_tile(args, io, tile, a, len, p, x);
            else reg_store(args, line, a, len, x);
        }
        for (int r = c; r < t.k; r += nthr) reg_store_row(args, io, io.stage_out, line, tile, t.m + r, p, sm.x2[r * P + p]);
        if (io.stage_out) {
            __syncthreads();
            reg_drain(args, io, line0, tile);
            __syncthreads();
            if (ti + gridDim.x < tiles) reg_fill(args, io, (ti + gridDim.x) << (io.lp + 1), tile, raw);
        }
    }
}

template <int K>
size_t reg_bytes(BuildArgs const& args, RegIo const& io)
{
    int const P = 1 << io.lp;
    SolveTables const& t = args.t;
    size_t const rows = size_t(io.stage_out ? std::max(t.n, args.raw ? 0 : args.r.size) : t.m);
    return sizeof(double) * (reg_smem_doubles<K>(t, P) + (rows + size_t(t.k)) * size_t(2 * P));
}

template <int K>
bool launch_reg(BuildArgs const& args, cudaStream_t s)
{
    SolveTables const& t = args.t;
    if (!reg_plain_rows(args)) return false;
    RegIo io {};
    io.v0 = (args.raw || args.r.periodic) ? 0 : args.r.nbe_lo;
    int const optin = device_limits().optin, sms = device_limits().sms;
    io.stage_out = args.lo.stride == 1 && args.lo.inner == 1 && args.lo.outer > 1;
    auto tiles = [&] { return (args.nlines + (int64_t(2) << io.lp) - 1) >> (io.lp + 1); };
    auto fits = [&](int threads, int blocks) {
        return (t.nchunk << io.lp) <= threads && reg_bytes<K>(args, io) + 1024 <= (size_t(optin) + 1024) / blocks;
    };
    // Two blocks of up to 256 threads per SM where their tiles still hold 16 lines or more, one's
    // loads and stores beside the other's sweeps (513 rows x 32768 lines: 63 us against 78 in one
    // block of 32 lines); else one block of up to 512 threads with the widest tile (1027 rows x
    // 65536 lines: 241 us with 16 lines against 320 in two blocks of 8).
    // Unit-stride lines read the same segments with any width: two blocks of eight lines; of sixteen
    // where eight would leave most of a warp without a chunk, or with a border to wait for (Greville
    // cubics x 65536 lines, 32 cells in 2 chunks: 37 us against 41; x 16384 lines, 100 cells in 6 chunks
    // and 4 border rows: 21 against 27; but without a border, 64 cells in 4 chunks: 33 against 27).
    bool const staged = io.stage_out || (args.lv.stride == 1 && args.lv.inner == 1 && args.lv.outer > 1);
    int const most = most_pairs(args.tile_req);
    io.lp = std::min(most, !staged ? 5 : (t.nchunk <= 2 || (t.nchunk <= 6 && t.k >= 4) ? 3 : 2));
    while (io.lp > 3 && !fits(256, 2)) --io.lp;
    if (!fits(256, 2)) {
        io.lp = most;
        while (io.lp > 0 && !fits(512, 1)) --io.lp;
    }
    while (io.lp > 1 && tiles() < int64_t(sms)) --io.lp; // at least a block for every SM
    size_t const bytes = reg_bytes<K>(args, io);
    if (!fits(512, 1)) return false;
    int const whole = std::max(32, 2 << io.lp); // whole warps, and whole rows of the tile
    int const threads = ((t.nchunk << io.lp) + whole - 1) / whole * whole;
    // no chunk shorter than 15 rows: tests on the last two steps only
    bool const full = t.nchunk > 1 && t.chunk_len >= 15;
    auto kern = full ? reg_build_kernel<K, 15> : reg_build_kernel<K, 0>;
    allow_shared(kern, bytes);
    // resident blocks: 512 threads of 128 registers an SM, and the shared memory
    int64_t const per_sm = std::max<int64_t>(1, std::min<int64_t>(512 / threads, (optin + 1024) / int64_t(bytes + 1024)));
    int64_t const grid = std::min<int64_t>(tiles(), per_sm * sms);
    kern<<<dim3((unsigned)grid), dim3((unsigned)threads), bytes, s>>>(args, io);
    DDCB_CUDA_CHECK(cudaGetLastError());
    return true;
}

} // namespace

// Returns false when the register solve does not cover this plan (the caller then takes the
// shared-memory tile).
bool launch_reg_build(BuildArgs const& args, cudaStream_t s)
{
    if (args.t.rmax == 0) return false;
    switch (args.t.kl) {
    case 1: return launch_reg<1>(args, s);
    case 2: return launch_reg<2>(args, s);
    case 3: return launch_reg<3>(args, s);
    case 4: return launch_reg<4>(args, s);
    default: return false;
    }
}

} // namespace ddcb
