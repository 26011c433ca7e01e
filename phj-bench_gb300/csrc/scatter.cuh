// scatter.cuh -- the tile scatter shared by the radix partition (partition.cu)
// and the batched joins (batch.cu): tiles of rows arrive in shared memory by
// bulk asynchronous copies, their rows are ranked by digit, places are
// reserved with one atomic per tile and digit, and every column is written in
// digit order.
#pragma once

#include "common.cuh"

namespace phjg
{
constexpr int kNT = 512;               // threads of a scatter CTA
constexpr uint32_t kMaxPassBits = 11;  // shared-memory digit histogram <= 2048 bins
constexpr uint32_t kMaxRPT = 8;        // rows per thread of a tile: 4096-row tiles
constexpr uint32_t kMaxStages = 4;     // tile buffers

// A tile: `cnt` rows from row0 of a source's columns, whose digits' buckets
// start at bucket0.
struct ScatterTile
{
    uint32_t row0, cnt, bucket0, aux;
};

// Bytes of one column's slice of a tile buffer (16 more: a slice widened to
// 16-byte units on both sides).
__host__ __device__ constexpr uint32_t tile_col_bytes(uint32_t tile_rows, uint32_t width)
{
    return (tile_rows * width + 31) & ~15u;
}

// Dynamic shared memory of a scatter CTA whose tile buffers hold buf_bytes.
__host__ __device__ constexpr uint64_t scatter_smem(uint32_t tile_rows, uint32_t stages, uint32_t buf_bytes, uint32_t bits)
{
    return (uint64_t)stages * buf_bytes + 4ull * tile_rows + 3 * 4ull * (1u << bits);
}

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

// The tiles of one CTA, as the source S gives them:
//   s.n()            number of tiles of this CTA
//   s.tile(k)        its k-th tile
//   s.in(t), s.out(t) the tile's source and destination columns
//   s.widened(t)     every source column is a buffer of the library's own
//                    (256-byte granules, 256-byte aligned), so a slice may be
//                    widened to 16-byte units; otherwise s.aligned(t) says
//                    whether the columns' bases lie on 16-byte boundaries
//   s.shift(t), s.bits(t)  digit = (hash >> shift) & (2^bits - 1)
//   s.offs(t), s.counts(t) bucket offsets and (counted down) bucket counts
//   s.first(t)       output row of the destination columns' first row
//
// Bound by DRAM when enough tiles are in flight: a tile is a chain of
// dependent steps (rank with shared atomics, digit scan, reservation,
// permutation, column writes) with three block barriers, during which one
// CTA alone leaves the SM idle, so two CTAs of 512 threads share a SM (64
// registers a thread, at most half of the shared memory each) and one's
// copies and writes fill the other's barriers.  Measured (256M rows of 16
// bytes, 6 bits): 5.4 TB/s, 80% of a plain copy's rate; one CTA a SM with a
// deeper ring reached 4.0 (stalls: block barriers, then shared memory).
template <int RPT, class S>
__device__ __forceinline__ void scatter_tiles(const S & s, uint8_t * smem, uint64_t * bar, uint32_t stages, uint32_t buf_bytes, uint32_t nb_max,
                                              int * __restrict__ err)
{
    constexpr uint32_t kT = kNT * RPT;
    constexpr uint32_t kWarps = kNT / 32;
    constexpr int kRows = (1 << kMaxPassBits) / 32 / kWarps; // 32-digit rows a warp scans
    uint32_t * perm = reinterpret_cast<uint32_t *>(smem + (size_t)stages * buf_bytes); // tile row | digit << 12, in digit order
    uint32_t * bins = perm + kT;
    uint32_t * excl = bins + nb_max;
    uint32_t * delta = excl + nb_max; // output row of a digit's first row, less its position in the tile's digit order
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

    const uint32_t my_tiles = s.n();
    if (my_tiles == 0)
        return;
    for (uint32_t d = threadIdx.x; d < nb_max; d += kNT)
        bins[d] = 0;
    if (threadIdx.x == 0)
    {
        for (uint32_t i = 0; i < stages; ++i)
            mbar_init(&bar[i], 1);
        fence_barrier_init();
    }
    __syncthreads();

    // Without widening, a tile is fetched by bulk copy when every column
    // slice is a whole number of 16-byte units (always, except a short last
    // tile).
    auto tma_ok = [&](const ScatterTile & t) -> bool {
        if (s.widened(t))
            return true;
        if (!s.aligned(t) || ((t.cnt * 8u) & 15u))
            return false;
        const Cols & in = s.in(t);
        for (uint32_t c = 0; c < in.n; ++c)
            if ((t.cnt * in.width[c]) & 15u)
                return false;
        return true;
    };
    auto buffer = [&](uint32_t i) -> uint8_t * { return smem + (size_t)i * buf_bytes; };
    auto issue = [&](const ScatterTile & t, uint32_t bi) {
        const Cols & in = s.in(t);
        auto span = [&](uint32_t w, uint64_t & a) -> uint32_t {
            a = ((uint64_t)t.row0 * w) & ~15ull;
            return (uint32_t)((((uint64_t)t.row0 + t.cnt) * w + 15 - a) & ~15ull);
        };
        uint64_t a;
        uint32_t bytes = span(8, a);
        for (uint32_t c = 0; c < in.n; ++c)
            bytes += span(in.width[c], a);
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(&bar[bi], bytes);
        const uint32_t kb = span(8, a);
        bulk_copy_g2s(buffer(bi), reinterpret_cast<const uint8_t *>(in.keys) + a, kb, &bar[bi]);
        uint32_t off = tile_col_bytes(kT, 8);
        for (uint32_t c = 0; c < in.n; ++c)
        {
            const uint32_t cb = span(in.width[c], a);
            bulk_copy_g2s(buffer(bi) + off, static_cast<const uint8_t *>(in.col[c]) + a, cb, &bar[bi]);
            off += tile_col_bytes(kT, in.width[c]);
        }
    };
    // tiles in flight ahead of the one being written: stages - 1, or the
    // next one once this one's buffer is free
    const uint32_t ahead = stages > 1 ? stages - 1 : 1;
    uint32_t parity = 0; // bit i: phase of bar[i] to wait for
    if (threadIdx.x == 0)
        for (uint32_t i = 0; i < ahead && i < my_tiles; ++i)
        {
            const ScatterTile t = s.tile(i);
            if (tma_ok(t))
                issue(t, i);
        }

    uint32_t bi = 0;
    for (uint32_t k = 0; k < my_tiles; ++k, bi = (bi + 1 == stages) ? 0 : bi + 1)
    {
        const ScatterTile tile = s.tile(k);
        const Cols & in = s.in(tile);
        const uint32_t cnt = tile.cnt;
        const uint32_t shift = s.shift(tile), nb = 1u << s.bits(tile), mask = nb - 1;
        uint8_t * buf = buffer(bi);
        const bool tma = tma_ok(tile);
        bool ok = true;
        if (tma)
            ok = mbar_wait(&bar[bi], (parity >> bi) & 1u, err, 1);
        else
        {
            uint64_t * bk = reinterpret_cast<uint64_t *>(buf);
            for (uint32_t i = threadIdx.x; i < cnt; i += kNT)
                bk[i] = in.keys[(uint64_t)tile.row0 + i];
            uint32_t off = tile_col_bytes(kT, 8);
            for (uint32_t c = 0; c < in.n; ++c)
            {
                for (uint32_t i = threadIdx.x; i < cnt; i += kNT)
                    copy_elem(buf + off, i, in.col[c], (uint64_t)tile.row0 + i, in.width[c]);
                off += tile_col_bytes(kT, in.width[c]);
            }
            __syncthreads();
        }
        // bytes of a column before the tile's first row in its buffer (a
        // tile that is not widened starts on a 16-byte boundary)
        const bool led = s.widened(tile);
        auto lead = [&](uint32_t w) -> uint32_t { return led ? (tile.row0 * w) & 15u : 0u; };

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
                const uint32_t d = (uint32_t)(int_hash64(bk[i]) >> shift) & mask;
                dr[j] = d | atomicAdd(&bins[d], 1u) << kMaxPassBits;
            }
        }
        if (!__syncthreads_and(ok))
            break;
        if (tma)
            parity ^= 1u << bi;
        // every thread is past the previous tile: its buffer can be refilled
        if (stages > 1 && threadIdx.x == 0 && k + ahead < my_tiles)
        {
            const ScatterTile t = s.tile(k + ahead);
            if (tma_ok(t))
                issue(t, bi == 0 ? stages - 1 : bi - 1);
        }

        // each warp scans its rows of 32 digits (its prefix from the counts
        // of all rows before) and reserves the digits' output places
        const uint32_t * offs = s.offs(tile) + tile.bucket0;
        uint32_t * counts = s.counts(tile) + tile.bucket0;
        const uint32_t first = s.first(tile);
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
                place[q] = __ldg(offs + d) + atomicSub(counts + d, v) - v - first;
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
        const Cols & out = s.out(tile);
        write_column<uint64_t, RPT>(buf + lead(8), out.keys, src, dest, cnt);
        uint32_t off = tile_col_bytes(kT, 8);
        for (uint32_t c = 0; c < in.n; ++c)
        {
            const uint32_t w = in.width[c];
            const uint8_t * cb = buf + off + lead(w);
            off += tile_col_bytes(kT, w);
            switch (w)
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
        if (stages == 1 && k + 1 < my_tiles)
        {
            __syncthreads();
            if (threadIdx.x == 0)
            {
                const ScatterTile t = s.tile(k + 1);
                if (tma_ok(t))
                    issue(t, 0);
            }
        }
    }
    // Bulk copies still in flight (only after a timeout) must land before
    // the CTA's shared memory is released.
    if (threadIdx.x == 0 && *err)
        for (uint32_t i = 0; i < stages; ++i)
            (void)mbar_wait(&bar[i], (parity >> i) & 1u, err, 1);
}
} // namespace phjg
