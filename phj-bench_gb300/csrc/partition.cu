// partition.cu -- radix partitioning on the top bits of intHash64
// (src/RadixPartition.cpp: scatterBatch :316-393, radixShuffle :546-577,
// refineToLeaves :417-539).
//
// One physical pass splits every segment of the previous pass (rows that
// share their top hash bits, stored contiguously; the first pass has one
// segment, the input) into 2^b buckets on the next b bits:
//   k_p1_hist / k_seg_hist   rows per bucket: shared-memory histograms, added
//                  to the buckets' global counts;
//   a scan         bucket counts -> bucket offsets (the first pass's last
//                  histogram CTA does it; later passes use scan_u32);
//   k_scatter      tiles of 4096 rows (one segment's each) arrive in shared
//                  memory by bulk asynchronous copies, their rows are ranked
//                  by digit, each tile reserves its rows' places with one
//                  atomic per digit on the bucket's count, and every column
//                  (key first, then payloads of 1/2/4/8/16 bytes) is written
//                  in digit order -- the column-first scatter of the
//                  reference, so that stores coalesce.
// The tiles of all CTAs in flight write next to each other in every bucket
// (one frontier a bucket, not one a bucket and CTA), and no per-tile counts
// are written, scanned and read back.  The order of the rows inside a bucket
// is not fixed, as in the reference.
#include "internal.h"
#include "scatter.cuh"

namespace phjg
{
namespace
{
// One segment's tiles of a later pass: row0, rows, first bucket.
struct PassGeom
{
    const uint32_t * seg_off;  // n_segs + 1: first row of each input segment
    const uint32_t * tile_pre; // n_segs + 1: first tile of each input segment
    uint32_t n_segs;
    uint32_t shift;            // digit = (hash >> shift) & mask
    uint32_t b;
};

// ---------------------------------------------------------------------------
// Histograms
// ---------------------------------------------------------------------------

// First pass: bucket counts, then (in the CTA that finishes last) the
// bucket offsets off[0..2^b].  `done` is zero at launch.
// With `mark` set (PHJ/BEP probe batches) the same pass also flags the
// leaves the rows hash to: a shared-memory bitmap per CTA (a bit is read
// before it is set), ORed into the global bitmap at the end.
__global__ void __launch_bounds__(kNT) k_p1_hist(const uint64_t * __restrict__ keys, uint64_t n, uint32_t shift, uint32_t b,
                                                 uint32_t * __restrict__ counts, uint32_t * __restrict__ done, uint32_t * __restrict__ off,
                                                 LeafMark mark)
{
    extern __shared__ uint32_t bins[];
    __shared__ uint32_t ws[kNT / 32];
    __shared__ uint32_t last;
    const uint32_t nb = 1u << b, mask = nb - 1;
    uint32_t * bm = bins + nb;
    for (uint32_t i = threadIdx.x; i < nb; i += kNT)
        bins[i] = 0;
    if (mark.bits)
        for (uint32_t i = threadIdx.x; i < mark.words; i += kNT)
            bm[i] = 0;
    __syncthreads();
    for (uint64_t base = (uint64_t)blockIdx.x * 8 * kNT; base < n; base += (uint64_t)gridDim.x * 8 * kNT)
    {
        uint64_t k[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
            const uint64_t row = base + j * kNT + threadIdx.x;
            k[j] = row < n ? __ldcs(keys + row) : 0;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (base + j * kNT + threadIdx.x < n)
            {
                const uint64_t h = int_hash64(k[j]);
                atomicAdd(&bins[(uint32_t)(h >> shift) & mask], 1u);
                if (mark.bits)
                {
                    const uint32_t L = (uint32_t)(h >> mark.shift);
                    if (!(bm[L >> 5] & (1u << (L & 31))))
                        atomicOr(&bm[L >> 5], 1u << (L & 31));
                }
            }
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d < nb; d += kNT)
        if (bins[d])
            atomicAdd(&counts[d], bins[d]);
    if (mark.bits)
        for (uint32_t w = threadIdx.x; w < mark.words; w += kNT)
        {
            const uint32_t v = bm[w];
            if (v && (__ldcg(mark.bits + w) & v) != v)
                atomicOr(mark.bits + w, v);
        }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last)
        return;
    __threadfence();
    constexpr uint32_t kPer = (1u << kMaxPassBits) / kNT;
    const uint32_t per = (nb + kNT - 1) / kNT, d0 = threadIdx.x * per;
    uint32_t v[kPer], acc = 0;
#pragma unroll
    for (uint32_t i = 0; i < kPer; ++i)
    {
        v[i] = i < per && d0 + i < nb ? __ldcg(counts + d0 + i) : 0u;
        acc += v[i];
    }
    uint32_t total;
    uint32_t run = block_excl_scan<kNT>(acc, ws, &total);
#pragma unroll
    for (uint32_t i = 0; i < kPer; ++i)
        if (i < per && d0 + i < nb)
        {
            off[d0 + i] = run;
            run += v[i];
        }
    if (threadIdx.x == 0)
        off[nb] = total;
}

// Later passes, one CTA: first tile of each of at most 4 * 1024 segments.
__global__ void __launch_bounds__(1024) k_seg_tiles(const uint32_t * __restrict__ seg_off, uint32_t n_segs, uint32_t tile_rows,
                                                    uint32_t * __restrict__ tile_pre)
{
    __shared__ uint32_t ws[32];
    const uint32_t per = (n_segs + 1023) / 1024, s0 = threadIdx.x * per;
    uint32_t v[4], acc = 0;
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i)
    {
        v[i] = i < per && s0 + i < n_segs ? (seg_off[s0 + i + 1] - seg_off[s0 + i] + tile_rows - 1) / tile_rows : 0u;
        acc += v[i];
    }
    uint32_t total;
    uint32_t run = block_excl_scan<1024>(acc, ws, &total);
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i)
        if (i < per && s0 + i < n_segs)
        {
            tile_pre[s0 + i] = run;
            run += v[i];
        }
    if (threadIdx.x == 0)
        tile_pre[n_segs] = total;
}

__global__ void k_tiles_per_seg(const uint32_t * __restrict__ seg_off, uint32_t n_segs, uint32_t tile_rows, uint32_t * __restrict__ nt)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n_segs)
        nt[s] = (seg_off[s + 1] - seg_off[s] + tile_rows - 1) / tile_rows;
}

// Later passes: each CTA counts a contiguous range of tiles, adding its
// histogram to the segment's buckets when the segment changes, and writes
// the tiles' descriptors {first row, rows, first bucket} for the scatter.
template <int RPT>
__global__ void __launch_bounds__(kNT) k_seg_hist(const uint64_t * __restrict__ keys, PassGeom g, uint32_t * __restrict__ counts,
                                                  uint4 * __restrict__ desc)
{
    constexpr uint32_t kT = kNT * RPT;
    extern __shared__ uint32_t bins[];
    const uint32_t nb = 1u << g.b, mask = nb - 1;
    const uint32_t n_tiles = g.tile_pre[g.n_segs];
    const uint32_t t0 = (uint32_t)((uint64_t)n_tiles * blockIdx.x / gridDim.x), t1 = (uint32_t)((uint64_t)n_tiles * (blockIdx.x + 1) / gridDim.x);
    if (t0 >= t1)
        return;
    // largest s with tile_pre[s] <= t0 (segments without tiles are skipped:
    // tile_pre[s] == tile_pre[s + 1] there)
    uint32_t seg = 0, hi = g.n_segs;
    while (hi - seg > 1)
    {
        const uint32_t mid = (seg + hi) >> 1;
        if (g.tile_pre[mid] <= t0)
            seg = mid;
        else
            hi = mid;
    }
    for (uint32_t i = threadIdx.x; i < nb; i += kNT)
        bins[i] = 0;
    __syncthreads();
    uint32_t seg_end = g.tile_pre[seg + 1];
    for (uint32_t t = t0; t < t1; ++t)
    {
        if (t >= seg_end)
        {
            // the segment's histogram so far, then the next segment
            __syncthreads();
            for (uint32_t d = threadIdx.x; d < nb; d += kNT)
                if (bins[d])
                {
                    atomicAdd(&counts[((uint64_t)seg << g.b) + d], bins[d]);
                    bins[d] = 0;
                }
            __syncthreads();
            while (t >= seg_end)
                seg_end = g.tile_pre[++seg + 1];
        }
        const uint32_t row0 = g.seg_off[seg] + (t - g.tile_pre[seg]) * kT, cnt = min(kT, g.seg_off[seg + 1] - row0);
        if (threadIdx.x == 0)
            desc[t] = make_uint4(row0, cnt, seg << g.b, 0);
        uint64_t k[RPT];
#pragma unroll
        for (int j = 0; j < RPT; ++j)
        {
            const uint32_t i = j * kNT + threadIdx.x;
            k[j] = i < cnt ? keys[row0 + i] : 0;
        }
#pragma unroll
        for (int j = 0; j < RPT; ++j)
            if (j * kNT + threadIdx.x < cnt)
                atomicAdd(&bins[(uint32_t)(int_hash64(k[j]) >> g.shift) & mask], 1u);
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d < nb; d += kNT)
        if (bins[d])
            atomicAdd(&counts[((uint64_t)seg << g.b) + d], bins[d]);
}

// ---------------------------------------------------------------------------
// Scatter (scatter.cuh)
// ---------------------------------------------------------------------------
struct ScatterGeom
{
    uint64_t n;               // rows (first pass)
    const uint4 * desc;       // later passes: tile descriptors, nullptr in the first pass
    const uint32_t * n_tiles; // later passes: number of tiles (device)
    uint32_t shift, b;
    uint32_t wave, tiles_per_cta; // tile k of CTA c: (c / wave) * wave * tiles_per_cta + k * wave + c % wave
    uint32_t stages, buf_bytes;
    int use_tma;
};

// The tiles of a pass, for scatter_tiles.
template <int RPT, bool kLater>
struct PassTiles
{
    const Cols & cin;
    const Cols & cout;
    const ScatterGeom & g;
    const uint32_t * off;
    uint32_t * cnt;
    uint64_t t_first;
    uint32_t my_tiles;

    __device__ __forceinline__ PassTiles(const Cols & i, const Cols & o, const ScatterGeom & geom, const uint32_t * offs, uint32_t * counts)
        : cin(i), cout(o), g(geom), off(offs), cnt(counts)
    {
        const uint64_t n_tiles = kLater ? *g.n_tiles : ceil_div(g.n, kNT * RPT);
        t_first = (uint64_t)(blockIdx.x / g.wave) * g.wave * g.tiles_per_cta + blockIdx.x % g.wave;
        my_tiles = t_first >= n_tiles ? 0u : (uint32_t)min((uint64_t)g.tiles_per_cta, (n_tiles - t_first + g.wave - 1) / g.wave);
    }
    __device__ __forceinline__ uint32_t n() const { return my_tiles; }
    __device__ __forceinline__ ScatterTile tile(uint32_t k) const
    {
        const uint64_t t = t_first + (uint64_t)k * g.wave;
        if (kLater)
        {
            const uint4 d = __ldg(g.desc + t);
            return ScatterTile{d.x, d.y, d.z, 0};
        }
        const uint64_t r = g.n - t * (kNT * RPT);
        return ScatterTile{(uint32_t)(t * (kNT * RPT)), r < kNT * RPT ? (uint32_t)r : kNT * RPT, 0, 0};
    }
    __device__ __forceinline__ const Cols & in(const ScatterTile &) const { return cin; }
    __device__ __forceinline__ const Cols & out(const ScatterTile &) const { return cout; }
    __device__ __forceinline__ bool widened(const ScatterTile &) const { return kLater; }
    __device__ __forceinline__ bool aligned(const ScatterTile &) const { return g.use_tma != 0; }
    __device__ __forceinline__ uint32_t shift(const ScatterTile &) const { return g.shift; }
    __device__ __forceinline__ uint32_t bits(const ScatterTile &) const { return g.b; }
    __device__ __forceinline__ const uint32_t * offs(const ScatterTile &) const { return off; }
    __device__ __forceinline__ uint32_t * counts(const ScatterTile &) const { return cnt; }
    __device__ __forceinline__ uint32_t first(const ScatterTile &) const { return 0; }
};

template <int RPT, bool kLater>
__global__ void __launch_bounds__(kNT, 2) k_scatter(const __grid_constant__ Cols in, const __grid_constant__ Cols out,
                                                    const __grid_constant__ ScatterGeom g, const uint32_t * __restrict__ offs,
                                                    uint32_t * __restrict__ counts, int * __restrict__ err)
{
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ __align__(8) uint64_t bar[kMaxStages];
    const PassTiles<RPT, kLater> s(in, out, g, offs, counts);
    scatter_tiles<RPT>(s, smem, bar, g.stages, g.buf_bytes, 1u << g.b, err);
}

// Tile shape of a scatter: rows per thread, ring depth, dynamic shared memory.
struct TileShape
{
    uint32_t rpt = 0, stages = 0, buf_bytes = 0;
    size_t smem = 0;
};

TileShape shape_of(const Cols & c, uint32_t rpt, uint32_t stages, uint32_t b)
{
    TileShape s;
    s.rpt = rpt;
    s.stages = stages;
    const uint32_t kT = kNT * rpt;
    uint32_t bytes = tile_col_bytes(kT, 8);
    for (uint32_t i = 0; i < c.n; ++i)
        bytes += tile_col_bytes(kT, c.width[i]);
    s.buf_bytes = (bytes + 127) & ~127u;
    s.smem = scatter_smem(kT, stages, s.buf_bytes, b);
    return s;
}

// The tile of the most rows (longest runs a digit) and the deepest ring of
// at most two buffers with which two CTAs fit on a SM; one CTA a SM where
// no tile leaves room for two.  Fewer rows a tile where the input would
// leave SMs without one.  Options "p1_tile_rows" and "p1_stages" pin the
// first pass's.  (32M rows of 20 bytes, 8 bits: 4096-row tiles, one buffer
// and two CTAs a SM write a pass in 256-266 us, 5.0-5.2 TB/s; 2048-row tiles
// in a ring of four and one CTA a SM took 496 us.)
TileShape choose_shape(const phj_ctx * ctx, const Cols & c, uint64_t n, uint32_t b, bool first)
{
    const uint32_t pin_rows = first ? ctx->p1_tile_rows : 0, pin_stages = first ? ctx->p1_stages : 0;
    const size_t most = ctx->smem_optin - 2048, half = (ctx->smem_optin + 1024) / 2 - 1024 - 64;
    uint32_t top = kMaxRPT;
    while (!pin_rows && top > 2 && ceil_div(n, (uint64_t)kNT * top) < (uint64_t)ctx->num_sms)
        top /= 2;
    TileShape best;
    for (int pass = 0; pass < 2 && !best.rpt; ++pass)
        for (uint32_t r = top; r >= 2 && !best.rpt; r /= 2)
            for (uint32_t st = pin_stages ? pin_stages : 2; st >= 1; --st)
            {
                if ((pin_rows && (uint32_t)kNT * r != pin_rows) || (pin_stages && st != pin_stages))
                    continue;
                const TileShape s = shape_of(c, r, st, b);
                if (s.smem <= (pass == 0 ? half : most))
                {
                    best = s;
                    break;
                }
            }
    if (!best.rpt)
        throw Error(PHJ_ERR_UNSUPPORTED, "row too wide for the shared-memory tile of the partition pass");
    return best;
}

uint64_t row_bytes_of(const Cols & c)
{
    uint64_t b = 8;
    for (uint32_t i = 0; i < c.n; ++i)
        b += c.width[i];
    return b;
}

// Launches the scatter over at most `tiles` tiles.  CTAs take a few tiles
// each and end, so that a kernel of another stream gets its turn on the
// SMs; the tiles in flight at a time are neighbours.  (Up to 8 tiles each, a
// build side of 3M rows waited for the probe side's pass of 37M again and
// again: the join took 925 us against 905 with up to 4; with 1 or 2 it takes
// 910 to 919.  Passes on their own take the same.)
void launch_scatter(phj_ctx * ctx, const Cols & src, const Cols & dst, ScatterGeom g, const TileShape & sh, uint64_t tiles, const uint32_t * offs,
                    uint32_t * counts, const char * phase, uint64_t n)
{
    g.stages = sh.stages;
    g.buf_bytes = sh.buf_bytes;
    g.wave = (uint32_t)ctx->num_sms * 2;
    g.tiles_per_cta = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(4, tiles / g.wave / 4));
    const uint64_t waves = ceil_div(tiles, (uint64_t)g.wave * g.tiles_per_cta);
    const unsigned grid = (unsigned)(waves == 1 ? std::min<uint64_t>(g.wave, tiles) : waves * g.wave);
    auto kern = g.desc ? (sh.rpt == 8 ? k_scatter<8, true> : sh.rpt == 4 ? k_scatter<4, true> : k_scatter<2, true>)
                       : (sh.rpt == 8 ? k_scatter<8, false> : sh.rpt == 4 ? k_scatter<4, false> : k_scatter<2, false>);
    KTimer kt(ctx, phase, n, 2 * n * row_bytes_of(src));
    kern<<<grid, kNT, sh.smem, ctx->stream>>>(src, dst, g, offs, counts, ctx->d_err);
    PHJ_LAUNCHED(ctx, "scatter");
}

// The first physical pass: bucket counts and offsets in one kernel, then the
// scatter.
void first_pass(phj_ctx * ctx, Scratch & s, const Cols & src, const Cols & dst, uint64_t n, uint32_t b, uint32_t * bucket_off, const char * phase)
{
    const uint32_t nb = 1u << b;
    const TileShape sh = choose_shape(ctx, src, n, b, true);
    bool aligned = (reinterpret_cast<uintptr_t>(src.keys) & 15u) == 0;
    for (uint32_t c = 0; c < src.n; ++c)
        aligned = aligned && (reinterpret_cast<uintptr_t>(src.col[c]) & 15u) == 0;
    uint32_t * counts = s.get<uint32_t>((uint64_t)nb + 1); // and the finished CTAs
    PHJ_CUDA(cudaMemsetAsync(counts, 0, ((uint64_t)nb + 1) * sizeof(uint32_t), ctx->stream));
    {
        KTimer kt(ctx, "part_hist", n, n * 8);
        // a pending leaf mark (PHJ/BEP) rides on this pass, once
        const LeafMark mark = ctx->leaf_mark;
        ctx->leaf_mark = LeafMark{};
        const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(n, 8 * kNT), (uint64_t)ctx->num_sms * 4));
        k_p1_hist<<<grid, kNT, (size_t)(nb + (mark.bits ? mark.words : 0)) * sizeof(uint32_t), ctx->stream>>>(src.keys, n, 64u - b, b, counts,
                                                                                                               counts + nb, bucket_off, mark);
        PHJ_LAUNCHED(ctx, "p1_hist");
    }
    ScatterGeom g{};
    g.n = n;
    g.shift = 64u - b;
    g.b = b;
    g.use_tma = aligned ? 1 : 0;
    launch_scatter(ctx, src, dst, g, sh, ceil_div(n, (uint64_t)kNT * sh.rpt), bucket_off, counts, phase, n);
}

// A later physical pass over n_segs segments.
void later_pass(phj_ctx * ctx, Scratch & s, const Cols & src, const Cols & dst, uint64_t n, const uint32_t * seg_off, uint32_t n_segs,
                uint32_t consumed, uint32_t b, uint32_t * next_off, const char * phase)
{
    const uint32_t nb = 1u << b;
    const uint64_t nbuckets = (uint64_t)n_segs * nb;
    const TileShape sh = choose_shape(ctx, src, n, b, false);
    const uint32_t kT = kNT * sh.rpt;
    uint32_t * tile_pre = s.get<uint32_t>((uint64_t)n_segs + 1);
    if (n_segs <= 4096)
    {
        k_seg_tiles<<<1, 1024, 0, ctx->stream>>>(seg_off, n_segs, kT, tile_pre);
        PHJ_LAUNCHED(ctx, "part_tiles");
    }
    else
    {
        uint32_t * nt = s.get<uint32_t>(n_segs);
        k_tiles_per_seg<<<(unsigned)ceil_div(n_segs, 256), 256, 0, ctx->stream>>>(seg_off, n_segs, kT, nt);
        PHJ_LAUNCHED(ctx, "part_tiles");
        scan_u32(ctx, s, nt, tile_pre, n_segs);
    }
    const uint64_t tiles_ub = ceil_div(n, kT) + std::min<uint64_t>(n_segs, n);
    uint32_t * counts = s.get<uint32_t>(nbuckets);
    PHJ_CUDA(cudaMemsetAsync(counts, 0, nbuckets * sizeof(uint32_t), ctx->stream));
    uint4 * desc = s.get<uint4>(tiles_ub);
    const PassGeom pg{seg_off, tile_pre, n_segs, 64u - consumed - b, b};
    {
        KTimer kt(ctx, "part_hist", n, n * 8);
        const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(tiles_ub, (uint64_t)ctx->num_sms * 4));
        auto kern = sh.rpt == 8 ? k_seg_hist<8> : sh.rpt == 4 ? k_seg_hist<4> : k_seg_hist<2>;
        kern<<<grid, kNT, nb * sizeof(uint32_t), ctx->stream>>>(src.keys, pg, counts, desc);
        PHJ_LAUNCHED(ctx, "part_hist");
    }
    scan_u32(ctx, s, counts, next_off, nbuckets);
    ScatterGeom g{};
    g.desc = desc;
    g.n_tiles = tile_pre + n_segs;
    g.shift = 64u - consumed - b;
    g.b = b;
    launch_scatter(ctx, src, dst, g, sh, tiles_ub, next_off, counts, phase, n);
}
} // namespace

void radix_partition(phj_ctx * ctx, Scratch & s, const Cols & in, uint64_t n, const std::vector<uint32_t> & pass_bits, const Cols & out,
                     const Cols & tmp, uint32_t * leaf_off, const char * phase)
{
    uint32_t total_bits = 0;
    std::vector<uint32_t> phys; // physical passes
    for (uint32_t b : pass_bits)
    {
        total_bits += b;
    }
    // Physical passes: the leaf ranges depend only on the total bits, so the
    // logical passes are re-split into the fewest passes of at most
    // kMaxPassBits bits (3 x 6 bits run as 9 + 9); an odd bit goes to the
    // later pass (17 bits: 8 + 9), whose tiles each serve one first-pass
    // bucket, so the first pass keeps more rows per bucket and tile
    // (32M x 128M multi-match: 8.6 -> 8.3 ms).
    {
        const uint32_t pieces = (total_bits + kMaxPassBits - 1) / kMaxPassBits;
        for (uint32_t p = 0; p < pieces; ++p)
            phys.push_back(total_bits / pieces + (pieces - 1 - p < total_bits % pieces ? 1u : 0u));
    }
    if (total_bits == 0 || total_bits > 24)
        throw Error(PHJ_ERR_UNSUPPORTED, "device radix partitioning supports 1..24 total bits");
    if (n >= (1ull << 32))
        throw Error(PHJ_ERR_UNSUPPORTED, "device radix partitioning supports < 2^32 rows per side");
    const uint64_t n_leaves = 1ull << total_bits;
    if (n == 0)
    {
        PHJ_CUDA(cudaMemsetAsync(leaf_off, 0, (n_leaves + 1) * sizeof(uint32_t), ctx->stream));
        return;
    }
    const size_t np = phys.size();
    const uint32_t * seg_off = nullptr;
    uint32_t n_segs = 1, consumed = 0;
    Cols src = in;
    for (size_t p = 0; p < np; ++p)
    {
        const uint32_t b = phys[p];
        const Cols & dst = ((np - 1 - p) % 2 == 0) ? out : tmp;
        uint32_t * next_off = (p + 1 == np) ? leaf_off : s.get<uint32_t>(((uint64_t)n_segs << b) + 1);
        if (p == 0)
            first_pass(ctx, s, src, dst, n, b, next_off, phase);
        else
            later_pass(ctx, s, src, dst, n, seg_off, n_segs, consumed, b, next_off, phase);
        seg_off = next_off;
        n_segs <<= b;
        consumed += b;
        src = dst;
    }
}

void set_partition_smem_limits(int smem_optin)
{
    for (auto * k : {k_scatter<8, false>, k_scatter<4, false>, k_scatter<2, false>, k_scatter<8, true>, k_scatter<4, true>, k_scatter<2, true>})
        PHJ_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin - 1024));
    PHJ_CUDA(cudaFuncSetAttribute(k_p1_hist, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)std::min<size_t>(((1u << kMaxPassBits) + (1u << 20) / 32) * sizeof(uint32_t), (size_t)smem_optin - 1024)));
}

} // namespace phjg
