// batch.cu -- many independent joins in one persistent launch.
//
// A serving stream is dominated in count by small and medium joins (a few
// thousand to a few million build rows).  Run one at a time, each pays a
// dozen launches, host round trips and grids too small to fill 152 SMs.
// Here n joins share every launch:
//   1. k_bt_hist     tiles of up to 4096 rows of every join's build and
//                    probe side, found by binary search in their prefix:
//                    each join's rows are counted per radix partition (the
//                    top bits of intHash64, src/Hash.h:18-25; enough bits for
//                    about 1024 build rows a partition, at most 11), and the
//                    tiles' descriptors are written;
//   2. scan_u32      the counts of all joins' partitions -> offsets;
//   3. k_bt_scatter  the partition passes' tile scatter (scatter.cuh) over
//                    the same tiles: ranked in shared memory, one
//                    reservation per tile and partition, written in
//                    partition order (src/RadixPartition.cpp:316-393);
//   4. k_bt_join     ONE persistent launch whose CTAs pop (join, partition)
//                    work items from a device queue (one atomic counter):
//                    the partition's build rows go into a shared-memory
//                    table with its next-chain (src/HashTable.h,
//                    src/BlockStore.h), then each warp on its own takes
//                    chunks of 128 probe rows: lookups, one reservation of
//                    output rows a chunk in the join's output, projection
//                    (key, build payloads, probe payloads:
//                    src/JoinOps.h:52-196).  A partition with more build
//                    rows than the shared table holds is built and probed
//                    in pieces.
// The chain (counter clears, the three kernels and the scan) reads no size back to the host: the join count and the joins'
// prefix arrays and descriptors are uploaded in one copy into a workspace
// the context keeps, the kernels read the count from there, and the chain
// is captured once into a CUDA graph at the workspace's capacity and
// replayed for every later batch that fits (option "batch_graph"; 0
// launches the same chain at the batch's own sizes, with each kernel timed).
// Each join's output is sized for one row per probe row; a join with more
// (repeated build keys) is counted exactly, flagged, and run again alone.
// Output multisets equal those of the single-join entry points; the order
// of the rows is not fixed.
#include "internal.h"
#include "piece.cuh"
#include "scatter.cuh"

#include <cstring>

namespace phjg
{
namespace
{
constexpr int kJNT = 256;              // threads of the join kernel
constexpr uint32_t kPieceRows = 2048;  // build rows a shared table holds
constexpr uint32_t kPieceSlots = 4096; // its slots (load <= 1/2)

struct BatchJoin
{
    Cols build, probe;  // inputs
    ProbeSides part;    // partitioned copies, output
    uint64_t build_rows, probe_rows;
    uint32_t bits;      // radix bits
    uint32_t part_base; // index of its first partition among all joins'
    uint32_t aligned_b, aligned_p; // every input column starts on a 16-byte boundary
};

// Index j with pre[j] <= t < pre[j+1] (pre non-decreasing, pre[0] = 0).
__device__ __forceinline__ uint32_t find_join(const uint64_t * __restrict__ pre, uint32_t n, uint64_t t)
{
    uint32_t lo = 0, hi = n; // pre[lo] <= t < pre[hi]
    while (hi - lo > 1)
    {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(pre + mid) <= t)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

__device__ __forceinline__ uint32_t part_of(uint64_t key, uint32_t bits)
{
    return bits ? (uint32_t)(int_hash64(key) >> (64u - bits)) : 0u;
}

// Tile descriptors for the scatter: bit 31 of aux is the side, the rest the
// join.
constexpr uint32_t kProbeSide = 0x80000000u;

// Each CTA counts a contiguous range of tiles (the build sides' tiles, then
// the probe sides'), adding its histogram to the counts of the join's side
// when that changes, and writes the tiles' descriptors.
template <int RPT>
__global__ void __launch_bounds__(kNT) k_bt_hist(const BatchJoin * __restrict__ d, const uint32_t * __restrict__ d_n,
                                                 const uint64_t * __restrict__ tb, const uint64_t * __restrict__ tp,
                                                 uint32_t * __restrict__ cnt_b, uint32_t * __restrict__ cnt_p, uint4 * __restrict__ desc,
                                                 uint32_t * __restrict__ d_tiles)
{
    constexpr uint32_t kT = kNT * RPT;
    __shared__ uint32_t h[1u << kMaxPassBits];
    const uint32_t n = *d_n;
    const uint64_t nb = tb[n], n_tiles = nb + tp[n];
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *d_tiles = (uint32_t)n_tiles;
    const uint64_t t0 = n_tiles * blockIdx.x / gridDim.x, t1 = n_tiles * (blockIdx.x + 1) / gridDim.x;
    for (uint32_t q = threadIdx.x; q < (1u << kMaxPassBits); q += kNT)
        h[q] = 0;
    __syncthreads();
    uint64_t t = t0;
    while (t < t1)
    {
        const bool build = t < nb;
        const uint64_t * pre = build ? tb : tp;
        const uint64_t u0 = build ? t : t - nb;
        const uint32_t j = find_join(pre, n, u0);
        const BatchJoin & J = d[j];
        const uint64_t rows = build ? J.build_rows : J.probe_rows;
        const uint64_t * keys = build ? J.build.keys : J.probe.keys;
        const uint32_t bits = J.bits, base = J.part_base;
        // this side's tiles of the CTA's range
        const uint64_t n_side = min(t1 - t, pre[j + 1] - u0);
        for (uint64_t u = u0; u < u0 + n_side; ++u)
        {
            const uint64_t r0 = (u - pre[j]) * kT;
            const uint32_t cnt = (uint32_t)min((uint64_t)kT, rows - r0);
            if (threadIdx.x == 0)
                desc[t + (u - u0)] = make_uint4((uint32_t)r0, cnt, base, j | (build ? 0u : kProbeSide));
            uint64_t k[RPT];
#pragma unroll
            for (int i = 0; i < RPT; ++i)
            {
                const uint32_t r = i * kNT + threadIdx.x;
                k[i] = r < cnt ? keys[r0 + r] : 0;
            }
#pragma unroll
            for (int i = 0; i < RPT; ++i)
                if (i * kNT + threadIdx.x < cnt)
                    atomicAdd(&h[part_of(k[i], bits)], 1u);
        }
        t += n_side;
        __syncthreads();
        uint32_t * cnt = (build ? cnt_b : cnt_p) + base;
        for (uint32_t q = threadIdx.x; q < (1u << bits); q += kNT)
            if (h[q])
            {
                atomicAdd(cnt + q, h[q]);
                h[q] = 0;
            }
        __syncthreads();
    }
}

// The batch's tiles for scatter_tiles: CTA c takes tiles c, c + grid, ...
struct BatchTiles
{
    const BatchJoin * d;
    const uint4 * desc;
    const uint32_t *off_b, *off_p;
    uint32_t *cnt_b, *cnt_p;
    uint32_t my_tiles;

    __device__ __forceinline__ uint32_t n() const { return my_tiles; }
    __device__ __forceinline__ ScatterTile tile(uint32_t k) const
    {
        const uint4 x = __ldg(desc + blockIdx.x + (uint64_t)k * gridDim.x);
        return ScatterTile{x.x, x.y, x.z, x.w};
    }
    __device__ __forceinline__ const BatchJoin & join(const ScatterTile & t) const { return d[t.aux & ~kProbeSide]; }
    __device__ __forceinline__ const Cols & in(const ScatterTile & t) const { return t.aux & kProbeSide ? join(t).probe : join(t).build; }
    __device__ __forceinline__ const Cols & out(const ScatterTile & t) const { return t.aux & kProbeSide ? join(t).part.probe : join(t).part.build; }
    __device__ __forceinline__ bool widened(const ScatterTile &) const { return false; }
    __device__ __forceinline__ bool aligned(const ScatterTile & t) const { return t.aux & kProbeSide ? join(t).aligned_p : join(t).aligned_b; }
    __device__ __forceinline__ uint32_t shift(const ScatterTile & t) const { return join(t).bits ? 64u - join(t).bits : 0u; }
    __device__ __forceinline__ uint32_t bits(const ScatterTile & t) const { return join(t).bits; }
    __device__ __forceinline__ const uint32_t * offs(const ScatterTile & t) const { return t.aux & kProbeSide ? off_p : off_b; }
    __device__ __forceinline__ uint32_t * counts(const ScatterTile & t) const { return t.aux & kProbeSide ? cnt_p : cnt_b; }
    __device__ __forceinline__ uint32_t first(const ScatterTile & t) const { return __ldg(offs(t) + t.bucket0); }
};

// (Each thread copying its rows one by one, column by column, to scattered
// places took 1,835 us for 64 joins of 4K-256K build rows, 77M rows in all.)
template <int RPT>
__global__ void __launch_bounds__(kNT, 2) k_bt_scatter(const BatchJoin * __restrict__ d, const uint4 * __restrict__ desc,
                                                       const uint32_t * __restrict__ d_tiles, const uint32_t * __restrict__ off_b,
                                                       const uint32_t * __restrict__ off_p, uint32_t * __restrict__ cnt_b,
                                                       uint32_t * __restrict__ cnt_p, uint32_t stages, uint32_t buf_bytes, uint32_t nb_max,
                                                       int * __restrict__ err)
{
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ __align__(8) uint64_t bar[kMaxStages];
    const uint32_t n_tiles = *d_tiles;
    const BatchTiles s{d, desc, off_b, off_p, cnt_b, cnt_p, blockIdx.x < n_tiles ? (n_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u};
    scatter_tiles<RPT>(s, smem, bar, stages, buf_bytes, nb_max, err);
}

// The CTA's warps probe rows [p0, p1) of the partition, 128 a warp at a time.
template <Repeats kRepeats>
__device__ __forceinline__ void probe_part(const ProbeSides & J, uint32_t p0, uint32_t p1, uint32_t c0, const PieceTable<kPieceRows> & tab,
                                           unsigned long long * out_cur, int * over)
{
    probe_piece<kRepeats, 4>(J, p0 + (threadIdx.x >> 5) * 128, kJNT / 32 * 128, p1, c0, tab, out_cur, over);
}
// (out of line, so that its registers do not weigh on the unique-key form)
__device__ __noinline__ void probe_part_dup(const ProbeSides & J, uint32_t p0, uint32_t p1, uint32_t c0, const PieceTable<kPieceRows> tab,
                                            unsigned long long * out_cur, int * over)
{
    probe_part<kLaneWrites>(J, p0, p1, c0, tab, out_cur, over);
}

// The persistent join: CTAs pop (join, partition) items until the queue is
// empty.  out_cur[j] counts join j's output rows (also past its capacity,
// where nothing is written and over[j] is set).
//
// A piece's table is 4096 slots of 4 bytes (hash bits and row), its keys
// and its next-chain: 36 KB, filled with 32-bit compare-and-swaps, so four
// 256-thread CTAs share a SM.  Warps probe without block barriers: a chunk
// is a chain of a key load, lookups, a reservation and the payload loads,
// and 32 warps a SM keep enough chains in flight.  (512-thread CTAs in
// steps of 512 probe rows with a block scan each, and 16-byte cells with
// 128-bit compare-and-swaps, took 1,575 us for 64 joins of 73M probe rows
// in all.)
__global__ void __launch_bounds__(kJNT, 4) k_bt_join(const BatchJoin * __restrict__ d, const uint32_t * __restrict__ d_n,
                                                     const uint64_t * __restrict__ parts,
                                                     const uint32_t * __restrict__ off_b, const uint32_t * __restrict__ off_p,
                                                     unsigned int * __restrict__ next_item, unsigned long long * __restrict__ out_cur,
                                                     int * __restrict__ over, const int * __restrict__ err, int * __restrict__ err_out)
{
    __shared__ __align__(16) uint32_t slots[kPieceSlots];
    __shared__ uint64_t bkeys[kPieceRows];
    __shared__ uint16_t nxt[kPieceRows];
    __shared__ BatchJoin J; // the item's join
    __shared__ uint32_t s_item;
    __shared__ int s_linked;
    const uint32_t n = *d_n;
    const uint64_t n_items = parts[n];
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *err_out = *err; // a copy of the scatter that gave up: read back with the row counts
    for (;;)
    {
        __syncthreads(); // the last item's table and s_item are no longer read
        if (threadIdx.x == 0)
            s_item = atomicAdd(next_item, 1u);
        __syncthreads();
        const uint64_t item = s_item;
        if (item >= n_items)
            return;
        const uint32_t j = find_join(parts, n, item);
        static_assert(sizeof(BatchJoin) % 8 == 0 && sizeof(BatchJoin) / 8 <= kJNT, "one 8-byte word a thread");
        if (threadIdx.x < sizeof(BatchJoin) / 8)
            reinterpret_cast<uint64_t *>(&J)[threadIdx.x] = reinterpret_cast<const uint64_t *>(d + j)[threadIdx.x];
        __syncthreads();
        const uint32_t g = J.part_base + (uint32_t)(item - parts[j]);
        const uint32_t b0 = off_b[g] - off_b[J.part_base], b1 = off_b[g + 1] - off_b[J.part_base];
        const uint32_t p0 = off_p[g] - off_p[J.part_base], p1 = off_p[g + 1] - off_p[J.part_base];
        if (b1 == b0 || p1 == p0)
            continue;
        // the partition's build rows, a piece at a time
        for (uint32_t c0 = b0; c0 < b1; c0 += kPieceRows)
        {
            const uint32_t rows = min(kPieceRows, b1 - c0);
            const uint32_t cap = max(4u, min(kPieceSlots, (uint32_t)bit_ceil64(3ull * rows))), mask = cap - 1;
            if (c0 != b0)
                __syncthreads(); // the last piece is no longer probed
            build_piece<kPieceRows, kJNT, false>(J.part.build.keys + c0, rows, slots, bkeys, nxt, mask, &s_linked);
            const PieceTable<kPieceRows> tab{slots, bkeys, nxt, mask};
            if (s_linked)
                probe_part_dup(J.part, p0, p1, c0, tab, out_cur + j, over + j);
            else
                probe_part<kUnique>(J.part, p0, p1, c0, tab, out_cur + j, over + j);
        }
    }
}

uint32_t partition_bits(uint64_t build_rows)
{
    uint32_t b = 0;
    while (b < 11 && (build_rows >> b) > 1024)
        ++b;
    return b;
}

size_t round_up(size_t x, size_t a)
{
    return (x + a - 1) / a * a;
}
} // namespace

// The chain's workspace, kept by the context across batches at fixed
// addresses, so that one captured graph of the chain replays for every
// batch of at most n_cap joins, q_cap partitions and t_cap tiles in all,
// rows of at most row_cap bytes and bits_cap radix bits a join.  Device
// block: the upload region (join count, the three prefix arrays, the join
// descriptors), then the per-join output counters and overflow flags
// (adjacent: one download), the item counter and the partitions' counts
// (with them: one clear), the partitions' offsets, the scan's carry space
// and the tile descriptors.  Pinned host block: the upload staging at the
// same offsets, then the download staging.
struct BatchGraph
{
    uint32_t n_cap = 0;
    uint64_t q_cap = 0, t_cap = 0;
    uint32_t row_cap = 0, bits_cap = 0;
    uint32_t rpt = 0, stages = 0, buf_bytes = 0; // the scatter's tile for row_cap and bits_cap
    size_t smem = 0;
    uint8_t * dev = nullptr;
    uint8_t * host = nullptr;
    size_t o_tb = 0, o_tp = 0, o_parts = 0, o_desc = 0, o_out = 0, o_next = 0, o_cnt = 0, o_off = 0, o_carry = 0, o_tile = 0, bytes = 0;
    cudaGraphExec_t exec = nullptr;
    uint64_t kernels = 0; // kernel launches in one replay
};

void free_batch_graph(phj_ctx * ctx)
{
    BatchGraph * W = ctx->batch_ws;
    if (!W)
        return;
    if (W->exec)
        cudaGraphExecDestroy(W->exec);
    if (W->dev)
        cudaFree(W->dev);
    if (W->host)
        cudaFreeHost(W->host);
    delete W;
    ctx->batch_ws = nullptr;
}

namespace
{
struct Chain
{
    const uint8_t * base;
    const BatchGraph * W;
    uint32_t * n() const { return (uint32_t *)base; }
    uint64_t * tb() const { return (uint64_t *)(base + W->o_tb); }
    uint64_t * tp() const { return (uint64_t *)(base + W->o_tp); }
    uint64_t * parts() const { return (uint64_t *)(base + W->o_parts); }
    BatchJoin * desc() const { return (BatchJoin *)(base + W->o_desc); }
    unsigned long long * out_cur() const { return (unsigned long long *)(base + W->o_out); }
    int * over() const { return (int *)(base + W->o_out + 8ull * W->n_cap); }
    unsigned int * next() const { return (unsigned int *)(base + W->o_next); }
    uint32_t * n_tiles() const { return (uint32_t *)(base + W->o_next) + 1; }
    uint32_t * cnt() const { return (uint32_t *)(base + W->o_cnt); } // build sides' partitions, then (from q_cap) the probe sides'
    uint32_t * off() const { return (uint32_t *)(base + W->o_off); } // offsets over the same array
    uint32_t * carry() const { return (uint32_t *)(base + W->o_carry); }
    uint4 * tiles() const { return (uint4 *)(base + W->o_tile); }
};

// The scatter tile for rows of row_cap bytes in up to kMaxCols + 1 columns:
// the most rows a tile with which two CTAs fit on a SM, else one CTA.
void choose_tile(const phj_ctx * ctx, BatchGraph & W)
{
    const size_t most = ctx->smem_optin - 2048, half = (ctx->smem_optin + 1024) / 2 - 1024 - 64;
    for (size_t limit : {half, most})
        for (uint32_t r = kMaxRPT; r >= 2; r /= 2)
            for (uint32_t st = 2; st >= 1; --st)
            {
                const uint32_t buf = (kNT * r * W.row_cap + 32 * (kMaxCols + 1) + 127) & ~127u;
                const size_t need = scatter_smem(kNT * r, st, buf, W.bits_cap);
                if (need > limit)
                    continue;
                W.rpt = r;
                W.stages = st;
                W.buf_bytes = buf;
                W.smem = need;
                return;
            }
    throw Error(PHJ_ERR_UNSUPPORTED, "row too wide for the shared-memory tile of the batched partition");
}

// The workspace for a batch of n joins, nq partitions, rows of at most
// row_bytes and at most `bits` radix bits a join.  Tiles are counted once
// its tile is known: the caller asks again with nt tiles.
BatchGraph & batch_workspace(phj_ctx * ctx, uint32_t n, uint64_t nq, uint64_t nt, uint32_t row_bytes, uint32_t bits)
{
    BatchGraph * W = ctx->batch_ws;
    if (W && n <= W->n_cap && nq <= W->q_cap && nt <= W->t_cap && row_bytes <= W->row_cap && bits <= W->bits_cap)
        return *W;
    uint32_t n_cap = W ? W->n_cap : 16;
    uint64_t q_cap = W ? W->q_cap : 4096, t_cap = W ? W->t_cap : 4096;
    const uint32_t row_cap = std::max(W ? W->row_cap : 20u, row_bytes), bits_cap = std::max(W ? W->bits_cap : 8u, bits);
    while (n_cap < n)
        n_cap *= 2;
    while (q_cap < nq)
        q_cap *= 2;
    while (t_cap < nt)
        t_cap *= 2;
    PHJ_CUDA(cudaStreamSynchronize(ctx->stream));
    free_batch_graph(ctx);
    W = new BatchGraph;
    ctx->batch_ws = W;
    W->n_cap = n_cap;
    W->q_cap = q_cap;
    W->t_cap = t_cap;
    W->row_cap = row_cap;
    W->bits_cap = bits_cap;
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at = round_up(at + bytes, 256);
        return o;
    };
    take(sizeof(uint32_t));
    W->o_tb = take(8ull * (n_cap + 1));
    W->o_tp = take(8ull * (n_cap + 1));
    W->o_parts = take(8ull * (n_cap + 1));
    W->o_desc = take(sizeof(BatchJoin) * n_cap);
    W->o_out = take(12ull * n_cap + 4);
    W->o_next = take(2 * sizeof(unsigned int));
    W->o_cnt = take(2 * 4ull * q_cap);
    W->o_off = take(4ull * (2 * q_cap + 1));
    W->o_carry = take(4ull * std::max<uint64_t>(scan_u32_carry(2 * q_cap), 1));
    W->o_tile = take(sizeof(uint4) * t_cap);
    W->bytes = at;
    try
    {
        choose_tile(ctx, *W);
        for (auto * k : {k_bt_scatter<8>, k_bt_scatter<4>, k_bt_scatter<2>})
            PHJ_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ctx->smem_optin - 1024));
        PHJ_CUDA(cudaMalloc(&W->dev, W->bytes));
        PHJ_CUDA(cudaMallocHost(&W->host, W->o_next));
    }
    catch (...)
    {
        free_batch_graph(ctx); // no half-made workspace for the next call
        throw;
    }
    return *W;
}

// The chain on the context's stream: counts and offsets of q_len partitions
// a side at stride q_cap (zero past the batch's own), then the three
// kernels.  With `bytes` (rows, input bytes) each kernel is timed; without,
// nothing but stream work is issued, so the chain can be captured.
void enqueue_chain(phj_ctx * ctx, const Chain & c, unsigned tgrid, unsigned jgrid, const uint64_t * bytes)
{
    cudaStream_t st = ctx->stream;
    const BatchGraph & W = *c.W;
    uint32_t *cnt_b = c.cnt(), *cnt_p = c.cnt() + W.q_cap, *off_b = c.off(), *off_p = c.off() + W.q_cap;
    PHJ_CUDA(cudaMemsetAsync(W.dev + W.o_out, 0, W.o_off - W.o_out, st)); // output counters, flags, item counter, counts
    {
        KTimer kt(ctx, bytes ? "batch_hist" : nullptr, bytes ? bytes[0] : 0, bytes ? bytes[0] * 8 : 0);
        auto kern = W.rpt == 8 ? k_bt_hist<8> : W.rpt == 4 ? k_bt_hist<4> : k_bt_hist<2>;
        kern<<<tgrid * 2, kNT, 0, st>>>(c.desc(), c.n(), c.tb(), c.tp(), cnt_b, cnt_p, c.tiles(), c.n_tiles());
        PHJ_LAUNCHED(ctx, "batch_hist");
    }
    // (32-bit offsets of both sides in one array: only differences within a
    // side are used, which a wrapped sum gives as well)
    scan_u32_into(ctx, cnt_b, off_b, 2 * W.q_cap, c.carry());
    {
        KTimer kt(ctx, bytes ? "batch_scatter" : nullptr, bytes ? bytes[0] : 0, bytes ? 2 * bytes[1] : 0);
        auto kern = W.rpt == 8 ? k_bt_scatter<8> : W.rpt == 4 ? k_bt_scatter<4> : k_bt_scatter<2>;
        kern<<<tgrid, kNT, W.smem, st>>>(c.desc(), c.tiles(), c.n_tiles(), off_b, off_p, cnt_b, cnt_p, W.stages, W.buf_bytes, 1u << W.bits_cap,
                                         ctx->d_err);
        PHJ_LAUNCHED(ctx, "batch_scatter");
    }
    {
        KTimer kt(ctx, bytes ? "batch_join" : nullptr, bytes ? bytes[2] : 0, bytes ? bytes[1] : 0);
        k_bt_join<<<jgrid, kJNT, 0, st>>>(c.desc(), c.n(), c.parts(), off_b, off_p, c.next(), c.out_cur(), c.over(), ctx->d_err,
                                          c.over() + W.n_cap);
        PHJ_LAUNCHED(ctx, "batch_join");
    }
}

unsigned join_grid(phj_ctx * ctx)
{
    int per_sm = 0;
    PHJ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bt_join, kJNT, 0));
    return (unsigned)ctx->num_sms * (unsigned)std::max(per_sm, 1);
}

// Captures the chain at the workspace's capacity (every grid at its
// largest: CTAs past the batch's tiles and partitions find no work) and
// instantiates it.
void capture_chain(phj_ctx * ctx, BatchGraph & W)
{
    const unsigned jgrid = join_grid(ctx);
    const uint64_t before = ctx->launches;
    cudaGraph_t g = nullptr;
    PHJ_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    try
    {
        enqueue_chain(ctx, Chain{W.dev, &W}, (unsigned)ctx->num_sms * 2, jgrid, nullptr);
    }
    catch (...)
    {
        cudaStreamEndCapture(ctx->stream, &g);
        if (g)
            cudaGraphDestroy(g);
        cudaGetLastError();
        ctx->launches = before;
        throw;
    }
    PHJ_CUDA(cudaStreamEndCapture(ctx->stream, &g));
    W.kernels = ctx->launches - before;
    ctx->launches = before;
    const cudaError_t e = cudaGraphInstantiate(&W.exec, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess)
        W.exec = nullptr;
    PHJ_CUDA(e);
}

void run_batch(phj_ctx * ctx, uint32_t n, const phj_table * const * builds, const phj_table * const * probes, phj_output ** outs,
               phj_batch_result * res)
{
    for (uint32_t j = 0; j < n; ++j)
    {
        if (!builds[j] || !probes[j])
            throw Error(PHJ_ERR_INVALID_ARGUMENT, "batch: null build or probe table");
        if (builds[j]->rows >= (1ull << 31) || probes[j]->rows >= (1ull << 31))
            throw Error(PHJ_ERR_UNSUPPORTED, "batch: fewer than 2^31 build rows and 2^31 probe rows per join");
    }
    begin_run(ctx);
    Scratch s(ctx);
    cudaEvent_t e0 = take_event(ctx), e1 = take_event(ctx);
    PHJ_CUDA(cudaEventRecord(e0, ctx->stream));

    std::vector<BatchJoin> h(n);
    std::vector<uint64_t> tb(n + 1, 0), tp(n + 1, 0), parts(n + 1, 0);
    uint64_t brows = 0, prows = 0, in_bytes = 0, copy_bytes = 0;
    uint32_t row_bytes = 8, most_bits = 0;
    auto side_aligned = [](const Cols & c) {
        uintptr_t x = reinterpret_cast<uintptr_t>(c.keys);
        for (uint32_t i = 0; i < c.n; ++i)
            x |= reinterpret_cast<uintptr_t>(c.col[i]);
        return (x & 15u) == 0 ? 1u : 0u;
    };
    // the partitioned copies' columns, cut from one allocation
    auto place = [&](Cols & c, const Cols & like, uint64_t rows) {
        c = like;
        c.keys = reinterpret_cast<uint64_t *>(copy_bytes);
        copy_bytes += round_up(std::max<uint64_t>(rows, 1) * 8, 256);
        for (uint32_t i = 0; i < c.n; ++i)
        {
            c.col[i] = reinterpret_cast<void *>(copy_bytes);
            copy_bytes += round_up(std::max<uint64_t>(rows, 1) * c.width[i], 256);
        }
    };
    for (uint32_t j = 0; j < n; ++j)
    {
        const phj_table & B = *builds[j];
        const phj_table & P = *probes[j];
        BatchJoin & J = h[j];
        J = BatchJoin{};
        J.build = cols_of(B);
        J.probe = cols_of(P);
        J.build_rows = B.rows;
        J.probe_rows = P.rows;
        J.bits = partition_bits(B.rows);
        J.part_base = (uint32_t)parts[j];
        J.aligned_b = side_aligned(J.build);
        J.aligned_p = side_aligned(J.probe);
        place(J.part.build, J.build, B.rows);
        place(J.part.probe, J.probe, P.rows);
        parts[j + 1] = parts[j] + (1ull << J.bits);
        most_bits = std::max(most_bits, J.bits);
        row_bytes = std::max<uint32_t>(row_bytes, 8 + (uint32_t)std::max(schema_bytes(B.schema), schema_bytes(P.schema)));
        brows += B.rows;
        prows += P.rows;
        in_bytes += B.rows * (8 + schema_bytes(B.schema)) + P.rows * (8 + schema_bytes(P.schema));
    }
    if (brows >= (1ull << 32) || prows >= (1ull << 32))
        throw Error(PHJ_ERR_UNSUPPORTED, "batch: fewer than 2^32 build rows and 2^32 probe rows in all");
    const uint64_t NQ = parts[n];
    uint8_t * copies = s.get<uint8_t>(copy_bytes);
    auto based = [&](Cols & c) {
        c.keys = reinterpret_cast<uint64_t *>(copies + reinterpret_cast<uintptr_t>(c.keys));
        for (uint32_t i = 0; i < c.n; ++i)
            c.col[i] = copies + reinterpret_cast<uintptr_t>(c.col[i]);
    };
    for (BatchJoin & J : h)
    {
        based(J.part.build);
        based(J.part.probe);
    }

    // outputs at one row per probe row (exact for unique build keys)
    std::vector<phj_output *> made(n, nullptr);
    try
    {
        for (uint32_t j = 0; j < n; ++j)
        {
            made[j] = new_output(ctx, builds[j]->schema, probes[j]->schema, probes[j]->rows);
            BatchJoin & J = h[j];
            J.part.out_keys = made[j]->keys;
            for (uint32_t c = 0; c < J.build.n; ++c)
                J.part.out_l[c] = made[j]->lcol[c];
            for (uint32_t c = 0; c < J.probe.n; ++c)
                J.part.out_r[c] = made[j]->rcol[c];
            J.part.out_cap = probes[j]->rows;
        }
        std::vector<unsigned long long> rows(n, 0);
        std::vector<int> ov(n, 0);
        if (n)
        {
            // the tiles' rows follow from the workspace's tile, then the
            // workspace has to hold that many tiles (a growth keeps the tile)
            const uint32_t kT = kNT * batch_workspace(ctx, n, NQ, 0, row_bytes, most_bits).rpt;
            for (uint32_t j = 0; j < n; ++j)
            {
                tb[j + 1] = tb[j] + ceil_div(builds[j]->rows, kT);
                tp[j + 1] = tp[j] + ceil_div(probes[j]->rows, kT);
            }
            BatchGraph & W = batch_workspace(ctx, n, NQ, tb[n] + tp[n], row_bytes, most_bits);
            // one upload: join count, prefix arrays, descriptors
            uint8_t * H = W.host;
            std::memcpy(H, &n, sizeof(uint32_t));
            std::memcpy(H + W.o_tb, tb.data(), (n + 1) * sizeof(uint64_t));
            std::memcpy(H + W.o_tp, tp.data(), (n + 1) * sizeof(uint64_t));
            std::memcpy(H + W.o_parts, parts.data(), (n + 1) * sizeof(uint64_t));
            std::memcpy(H + W.o_desc, h.data(), n * sizeof(BatchJoin));
            PHJ_CUDA(cudaMemcpyAsync(W.dev, H, W.o_desc + n * sizeof(BatchJoin), cudaMemcpyHostToDevice, ctx->stream));
            const Chain c{W.dev, &W};
            if (ctx->batch_graph)
            {
                if (!W.exec)
                    capture_chain(ctx, W);
                KTimer kt(ctx, "batch_graph", brows + prows, (brows + prows) * 8 + 3 * in_bytes);
                PHJ_CUDA(cudaGraphLaunch(W.exec, ctx->stream));
                ctx->launches += W.kernels;
            }
            else
            {
                const uint64_t n_tiles = tb[n] + tp[n];
                const unsigned tgrid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(n_tiles, (uint64_t)ctx->num_sms * 2));
                const unsigned jgrid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(NQ, join_grid(ctx)));
                const uint64_t bytes[3] = {brows + prows, in_bytes, prows};
                enqueue_chain(ctx, c, tgrid, jgrid, bytes);
            }
            uint8_t * D = H + W.o_out;
            PHJ_CUDA(cudaMemcpyAsync(D, c.out_cur(), 12ull * W.n_cap + 4, cudaMemcpyDeviceToHost, ctx->stream));
            PHJ_CUDA(cudaStreamSynchronize(ctx->stream));
            std::memcpy(rows.data(), D, n * sizeof(unsigned long long));
            std::memcpy(ov.data(), D + 8ull * W.n_cap, n * sizeof(int));
            int gave_up = 0;
            std::memcpy(&gave_up, D + 12ull * W.n_cap, sizeof(int));
            if (gave_up)
            {
                PHJ_CUDA(cudaMemsetAsync(ctx->d_err, 0, sizeof(int), ctx->stream));
                throw Error(PHJ_ERR_DEVICE_TIMEOUT, "a bounded device wait gave up (code " + std::to_string(gave_up) + ")");
            }
        }
        uint64_t out_rows = 0;
        for (uint32_t j = 0; j < n; ++j)
        {
            if (ov[j])
            {
                // more output rows than probe rows (repeated build keys):
                // this join again, alone
                free_output(ctx, made[j]);
                made[j] = nullptr;
                made[j] = join_alone(ctx, *builds[j], *probes[j]);
            }
            else
                made[j]->rows = rows[j];
            out_rows += made[j]->rows;
        }
        PHJ_CUDA(cudaEventRecord(e1, ctx->stream));
        PHJ_CUDA(cudaEventSynchronize(e1));
        if (res)
        {
            res->e2e_wall_ms = event_ms(e0, e1);
            res->n_joins = n;
            res->build_rows = brows;
            res->probe_rows = prows;
            res->output_rows = out_rows;
            res->peak_mem_bytes = ctx->peak_bytes;
        }
    }
    catch (...)
    {
        for (phj_output * o : made)
            if (o)
                free_output(ctx, o);
        throw;
    }
    for (uint32_t j = 0; j < n; ++j)
        outs[j] = made[j];
}
} // namespace
} // namespace phjg

extern "C" phj_status phj_batch_run(phj_ctx * ctx, uint32_t n, const phj_table * const * builds, const phj_table * const * probes,
                                    phj_output ** outs, phj_batch_result * result)
{
    if (!ctx || (n && (!builds || !probes || !outs)))
        return PHJ_ERR_INVALID_ARGUMENT;
    for (uint32_t j = 0; j < n; ++j)
        outs[j] = nullptr;
    return phjg::guard(ctx, [&] { phjg::run_batch(ctx, n, builds, probes, outs, result); });
}
