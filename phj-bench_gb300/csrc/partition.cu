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

namespace phjg
{
namespace
{
constexpr int kNT = 512;
constexpr uint32_t kMaxPassBits = 11;  // shared-memory digit histogram <= 2048 bins
constexpr uint32_t kMaxRPT = 8;        // rows per thread of a tile: 4096-row tiles
constexpr uint32_t kMaxStages = 4;

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
// Scatter
// ---------------------------------------------------------------------------
struct TileSmem
{
    uint32_t buf_bytes;              // one tile of every column
    uint32_t col_off[kMaxCols + 1];  // byte offset of each payload column in a buffer (keys at 0)
};

struct ScatterGeom
{
    uint64_t n;               // rows (first pass)
    const uint4 * desc;       // later passes: tile descriptors, nullptr in the first pass
    const uint32_t * n_tiles; // later passes: number of tiles (device)
    uint32_t shift, b;
    uint32_t wave, tiles_per_cta; // tile k of CTA c: (c / wave) * wave * tiles_per_cta + k * wave + c % wave
    uint32_t stages;
    int use_tma;
};

template <class T, int RPT>
__device__ __forceinline__ void write_column(const uint8_t * buf, T * __restrict__ dst, const uint32_t (&src)[RPT], const uint32_t (&dest)[RPT],
                                             uint32_t cnt)
{
    const T * b = reinterpret_cast<const T *>(buf);
#pragma unroll
    for (int j = 0; j < RPT; ++j)
        if (j * kNT + threadIdx.x < cnt)
            dst[dest[j]] = b[src[j]];
}

// Bound by DRAM when enough tiles are in flight: a tile is a chain of
// dependent steps (rank with shared atomics, digit scan, reservation,
// permutation, column writes) with three block barriers, during which one
// CTA alone leaves the SM idle, so two CTAs of 512 threads share a SM (64
// registers a thread, at most half of the shared memory each) and one's
// copies and writes fill the other's barriers.  Measured (256M rows of 16
// bytes, 6 bits): 5.4 TB/s, 80% of a plain copy's rate; one CTA a SM with a
// deeper ring reached 4.0 (stalls: block barriers, then shared memory).
template <int RPT, bool kLater>
__global__ void __launch_bounds__(kNT, 2) k_scatter(const __grid_constant__ Cols in, const __grid_constant__ Cols out,
                                                    const __grid_constant__ ScatterGeom g, const __grid_constant__ TileSmem sm,
                                                    const uint32_t * __restrict__ offs, uint32_t * __restrict__ counts, int * __restrict__ err)
{
    constexpr uint32_t kT = kNT * RPT;
    constexpr uint32_t kWarps = kNT / 32;
    constexpr int kRows = (1 << kMaxPassBits) / 32 / kWarps; // 32-digit rows a warp scans
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ __align__(8) uint64_t bar[kMaxStages];
    const uint32_t nb = 1u << g.b, mask = nb - 1;
    uint32_t * perm = reinterpret_cast<uint32_t *>(smem + (size_t)g.stages * sm.buf_bytes); // tile row | digit << 12, in digit order
    uint32_t * bins = perm + kT;
    uint32_t * excl = bins + nb;
    uint32_t * delta = excl + nb; // output row of a digit's first row, less its position in the tile's digit order
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    const uint64_t n_tiles = kLater ? *g.n_tiles : ceil_div(g.n, kT);
    const uint64_t t_first = (uint64_t)(blockIdx.x / g.wave) * g.wave * g.tiles_per_cta + blockIdx.x % g.wave;
    if (t_first >= n_tiles)
        return;
    const uint32_t my_tiles = (uint32_t)min((uint64_t)g.tiles_per_cta, (n_tiles - t_first + g.wave - 1) / g.wave);
    for (uint32_t d = threadIdx.x; d < nb; d += kNT)
        bins[d] = 0;
    if (threadIdx.x == 0)
    {
        for (uint32_t i = 0; i < g.stages; ++i)
            mbar_init(&bar[i], 1);
        fence_barrier_init();
    }
    __syncthreads();

    auto tile_of = [&](uint32_t k) -> uint4 {
        const uint64_t t = t_first + (uint64_t)k * g.wave;
        if (kLater)
            return __ldg(g.desc + t);
        const uint64_t r = g.n - t * kT;
        return make_uint4((uint32_t)(t * kT), r < kT ? (uint32_t)r : kT, 0, 0);
    };
    // A first-pass tile is fetched by bulk copy when every column slice is a
    // whole number of 16-byte units (always, except a short last tile); a
    // later pass reads the library's own buffers (256-byte granules), where
    // a slice may be widened to 16-byte units on both sides.
    auto tma_ok = [&](const uint4 & t) -> bool {
        if (kLater)
            return true;
        if (!g.use_tma || ((t.y * 8u) & 15u))
            return false;
        for (uint32_t c = 0; c < in.n; ++c)
            if ((t.y * in.width[c]) & 15u)
                return false;
        return true;
    };
    auto buffer = [&](uint32_t i) -> uint8_t * { return smem + (size_t)i * sm.buf_bytes; };
    auto issue = [&](const uint4 & t, uint32_t bi) {
        auto span = [&](uint32_t w, uint64_t & a) -> uint32_t {
            a = ((uint64_t)t.x * w) & ~15ull;
            return (uint32_t)((((uint64_t)(t.x + t.y) * w + 15) & ~15ull) - a);
        };
        uint64_t a;
        uint32_t bytes = span(8, a);
        for (uint32_t c = 0; c < in.n; ++c)
            bytes += span(in.width[c], a);
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(&bar[bi], bytes);
        const uint32_t kb = span(8, a);
        bulk_copy_g2s(buffer(bi), reinterpret_cast<const uint8_t *>(in.keys) + a, kb, &bar[bi]);
        for (uint32_t c = 0; c < in.n; ++c)
        {
            const uint32_t cb = span(in.width[c], a);
            bulk_copy_g2s(buffer(bi) + sm.col_off[c], static_cast<const uint8_t *>(in.col[c]) + a, cb, &bar[bi]);
        }
    };
    // tiles in flight ahead of the one being written: stages - 1, or the
    // next one once this one's buffer is free
    const uint32_t ahead = g.stages > 1 ? g.stages - 1 : 1;
    uint32_t parity = 0; // bit i: phase of bar[i] to wait for
    if (threadIdx.x == 0)
        for (uint32_t i = 0; i < ahead && i < my_tiles; ++i)
        {
            const uint4 t = tile_of(i);
            if (tma_ok(t))
                issue(t, i);
        }

    uint32_t bi = 0;
    for (uint32_t k = 0; k < my_tiles; ++k, bi = (bi + 1 == g.stages) ? 0 : bi + 1)
    {
        const uint4 tile = tile_of(k);
        const uint32_t cnt = tile.y;
        uint8_t * buf = buffer(bi);
        bool ok = true;
        if (tma_ok(tile))
        {
            ok = mbar_wait(&bar[bi], (parity >> bi) & 1u, err, 1);
        }
        else
        {
            uint64_t * bk = reinterpret_cast<uint64_t *>(buf);
            for (uint32_t i = threadIdx.x; i < cnt; i += kNT)
                bk[i] = in.keys[tile.x + i];
            for (uint32_t c = 0; c < in.n; ++c)
                for (uint32_t i = threadIdx.x; i < cnt; i += kNT)
                    copy_elem(buf + sm.col_off[c], i, in.col[c], (uint64_t)tile.x + i, in.width[c]);
            __syncthreads();
        }
        // bytes of a column before the tile's first row in its buffer
        auto lead = [&](uint32_t w) -> uint32_t { return kLater ? (tile.x * w) & 15u : 0u; };

        // digit and rank within the digit (bins are zero here)
        const uint64_t * bk = reinterpret_cast<const uint64_t *>(buf + lead(8));
        uint32_t dr[RPT]; // digit | rank << 11
#pragma unroll
        for (int j = 0; j < RPT; ++j)
        {
            const uint32_t i = j * kNT + threadIdx.x;
            dr[j] = 0xFFFFFFFFu;
            if (i < cnt)
            {
                const uint32_t d = (uint32_t)(int_hash64(bk[i]) >> g.shift) & mask;
                dr[j] = d | atomicAdd(&bins[d], 1u) << kMaxPassBits;
            }
        }
        if (!__syncthreads_and(ok))
            break;
        if (tma_ok(tile))
            parity ^= 1u << bi;
        // every thread is past the previous tile: its buffer can be refilled
        if (g.stages > 1 && threadIdx.x == 0 && k + ahead < my_tiles)
        {
            const uint4 t = tile_of(k + ahead);
            if (tma_ok(t))
                issue(t, bi == 0 ? g.stages - 1 : bi - 1);
        }

        // each warp scans its rows of 32 digits (its prefix from the counts
        // of all rows before) and reserves the digits' output places
        uint32_t ex[kRows], place[kRows];
#pragma unroll
        for (int q = 0; q < kRows; ++q)
        {
            const uint32_t r = warp + q * kWarps;
            ex[q] = place[q] = 0;
            if (r * 32 >= nb)
                continue;
            uint32_t before = 0;
            for (uint32_t p = 0; p < r; ++p)
                before += bins[p * 32 + lane];
            const uint32_t d = r * 32 + lane;
            const uint32_t v = d < nb ? bins[d] : 0u;
            if (v)
                place[q] = __ldg(offs + tile.z + d) + atomicSub(counts + tile.z + d, v) - v;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                before += __shfl_xor_sync(0xffffffffu, before, o);
            uint32_t x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= (uint32_t)o)
                    x += y;
            }
            ex[q] = before + x - v;
            if (d < nb)
                excl[d] = ex[q];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < RPT; ++j)
            if (dr[j] != 0xFFFFFFFFu)
            {
                const uint32_t d = dr[j] & ((1u << kMaxPassBits) - 1);
                perm[excl[d] + (dr[j] >> kMaxPassBits)] = (j * kNT + threadIdx.x) | d << 12;
            }
#pragma unroll
        for (int q = 0; q < kRows; ++q)
        {
            const uint32_t d = (warp + q * kWarps) * 32 + lane;
            if (d < nb)
            {
                delta[d] = place[q] - ex[q];
                bins[d] = 0;
            }
        }
        __syncthreads();
        uint32_t src[RPT], dest[RPT];
#pragma unroll
        for (int j = 0; j < RPT; ++j)
        {
            const uint32_t pos = j * kNT + threadIdx.x;
            src[j] = dest[j] = 0;
            if (pos < cnt)
            {
                const uint32_t e = perm[pos];
                src[j] = e & 4095u;
                dest[j] = delta[e >> 12] + pos;
            }
        }
        write_column<uint64_t, RPT>(buf + lead(8), out.keys, src, dest, cnt);
        for (uint32_t c = 0; c < in.n; ++c)
        {
            const uint8_t * cb = buf + sm.col_off[c] + lead(in.width[c]);
            switch (in.width[c])
            {
                case 1: write_column<uint8_t, RPT>(cb, (uint8_t *)out.col[c], src, dest, cnt); break;
                case 2: write_column<uint16_t, RPT>(cb, (uint16_t *)out.col[c], src, dest, cnt); break;
                case 4: write_column<uint32_t, RPT>(cb, (uint32_t *)out.col[c], src, dest, cnt); break;
                case 8: write_column<uint64_t, RPT>(cb, (uint64_t *)out.col[c], src, dest, cnt); break;
                default: write_column<uint4, RPT>(cb, (uint4 *)out.col[c], src, dest, cnt); break;
            }
        }
        // The next tile's first barrier (after its ranking) comes before
        // this tile's perm, excl and delta are written again; its ranking
        // finds the counts zeroed before this tile's last barrier.  Only a
        // single buffer must be free before it is refilled.
        if (g.stages == 1 && k + 1 < my_tiles)
        {
            __syncthreads();
            if (threadIdx.x == 0)
            {
                const uint4 t = tile_of(k + 1);
                if (tma_ok(t))
                    issue(t, 0);
            }
        }
    }
    // Bulk copies still in flight (only after a timeout) must land before
    // the CTA's shared memory is released.
    if (threadIdx.x == 0 && *err)
        for (uint32_t i = 0; i < g.stages; ++i)
            (void)mbar_wait(&bar[i], (parity >> i) & 1u, err, 1);
}

// Tile shape of a scatter: rows per thread, ring depth, dynamic shared memory.
struct TileShape
{
    uint32_t rpt = 0, stages = 0;
    TileSmem sm{};
    size_t smem = 0;
};

TileShape shape_of(const Cols & c, uint32_t rpt, uint32_t stages, uint32_t b)
{
    TileShape s;
    s.rpt = rpt;
    s.stages = stages;
    const uint32_t kT = kNT * rpt;
    uint32_t off = kT * 8 + 16; // 16 more bytes a column: a slice widened to 16-byte units
    for (uint32_t i = 0; i < c.n; ++i)
    {
        s.sm.col_off[i] = off;
        off += (kT * c.width[i] + 31) & ~15u;
    }
    s.sm.buf_bytes = (off + 127) & ~127u;
    s.smem = (size_t)stages * s.sm.buf_bytes + 4ull * kT + 3 * 4ull * (1u << b);
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
// SMs; the tiles in flight at a time are neighbours.
void launch_scatter(phj_ctx * ctx, const Cols & src, const Cols & dst, ScatterGeom g, const TileShape & sh, uint64_t tiles, const uint32_t * offs,
                    uint32_t * counts, const char * phase, uint64_t n)
{
    g.stages = sh.stages;
    g.wave = (uint32_t)ctx->num_sms * 2;
    g.tiles_per_cta = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(8, tiles / g.wave / 4));
    const uint64_t waves = ceil_div(tiles, (uint64_t)g.wave * g.tiles_per_cta);
    const unsigned grid = (unsigned)(waves == 1 ? std::min<uint64_t>(g.wave, tiles) : waves * g.wave);
    auto kern = g.desc ? (sh.rpt == 8 ? k_scatter<8, true> : sh.rpt == 4 ? k_scatter<4, true> : k_scatter<2, true>)
                       : (sh.rpt == 8 ? k_scatter<8, false> : sh.rpt == 4 ? k_scatter<4, false> : k_scatter<2, false>);
    KTimer kt(ctx, phase, n, 2 * n * row_bytes_of(src));
    kern<<<grid, kNT, sh.smem, ctx->stream>>>(src, dst, g, sh.sm, offs, counts, ctx->d_err);
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
