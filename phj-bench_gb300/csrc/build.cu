// build.cu -- hashtable build on the device.
//
// PHJ-PURE / PHJ: one JoinHashTable per leaf (src/PHJ.cpp:260-282,
// src/PHJBep.cpp:192-232).  Capacity follows JoinHashTable::reserve
// (src/HashTable.h:72-79): bit_ceil(2 * rows), i.e. load <= 1/2.  One CTA
// owns a leaf: it builds the table in shared memory with 128-bit CAS
// inserts, threads each row's previous head into the next-chain
// (BlockStore::setPrev, src/BlockStore.h:83-84; buildOneBlock,
// src/JoinOps.h:205-228), then streams the finished table to global memory.
// Leaves too large for shared memory are built in place in global memory.
//
// CHJ: one global table of 256 sub-tables selected by the top 8 hash bits
// (the mutex-free form of ChjSlottedTable, src/TwoLevelHashTable.h:57-91),
// filled by every thread of the grid with 128-bit CAS inserts.
#include "internal.h"

#include <cmath>

namespace phjg
{
namespace
{
constexpr int kBuildNT = 256;
constexpr uint32_t kSmemCellsMax = 8192; // 128 KiB of cells per CTA
constexpr uint32_t kLookers = 1024;
constexpr uint32_t kInlineLeafRows = 32; // the fewest rows a leaf, in the mean, of inline tables

// Cells of a table for r rows: the power of two at or above r * pct / 100
// (pct 200: load <= 1/2, the reference's JoinHashTable::reserve), and above r.
__host__ __device__ __forceinline__ uint64_t table_cells(uint64_t r, uint32_t pct)
{
    if (!r)
        return 0;
    const uint64_t want = (r * pct + 99) / 100;
    return bit_ceil64(want > r ? want : r + 1);
}

__global__ void k_leaf_caps(const uint32_t * __restrict__ leaf_off, uint32_t n_leaves, uint32_t pct, uint32_t * __restrict__ caps,
                            uint32_t * __restrict__ max_rows)
{
    const uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= n_leaves)
        return;
    const uint32_t r = leaf_off[l + 1] - leaf_off[l];
    caps[l] = (uint32_t)table_cells(r, pct);
    if (r)
        atomicMax(max_rows, r);
}

__device__ __forceinline__ uint32_t log2u(uint64_t x)
{
    return 63u - (uint32_t)__clzll((long long)x);
}

// Position of `key` in a finished table (the key is present).
__device__ __forceinline__ uint32_t cell_of(const Cell * tab, uint64_t cap, uint64_t h, uint64_t key)
{
    uint64_t pos = probe_start(h, cap);
    for (uint64_t step = 0; step < cap; ++step)
    {
        if (tab[pos].key == key && ref_valid(tab[pos].ref))
            return (uint32_t)pos;
        pos = (pos + 1) & (cap - 1);
    }
    return 0; // unreachable: every row's key was inserted
}

// The payloads of row `si`, to row `di`.
__device__ __forceinline__ void copy_row(const Cols & src, uint64_t si, const Cols & dst, uint64_t di)
{
    for (uint32_t c = 0; c < src.n; ++c)
        copy_elem(dst.col[c], di, src.col[c], si, src.width[c]);
}

// Tables sized by estimate: whether a leaf has more rows than its table may
// hold is found out before any is built (a hot key of 100,000 rows among 8M: a
// build of 150 us that was thrown away when the leaf's own CTA found out; now
// 45 us of CTAs that end at once).
__device__ __forceinline__ bool past_estimate(const uint32_t * __restrict__ leaf_off, uint32_t l0, uint32_t l1, uint32_t stride, uint32_t most_rows)
{
    bool over = false;
    for (uint32_t l = l0 + threadIdx.x; l < l1; l += stride)
        over |= leaf_off[l + 1] - leaf_off[l] > most_rows;
    return over;
}

__global__ void k_leaf_check(const uint32_t * __restrict__ leaf_off, uint32_t n_leaves, uint32_t most_rows, int * __restrict__ flags, int * __restrict__ stop)
{
    const uint32_t l0 = blockIdx.x * blockDim.x;
    if (past_estimate(leaf_off, l0, min(n_leaves, l0 + blockDim.x), blockDim.x, most_rows))
    {
        atomicOr(flags, kLeafOverflow);
        *stop = 1;
    }
}

// One CTA per leaf.  Tables are either uniform (every leaf 2^ulog cells at
// leaf << ulog, ulog >= 0) or sized per leaf through table_off (ulog < 0).
// The RowRefCell of a build row is {0, row}: block 0 is the whole
// leaf-partitioned build side, row its index there.
// With kGroup (every table in shared memory) a leaf whose keys repeat is
// grouped while its table is at hand: the payloads of one key's rows become
// contiguous in `dst` and the key's cell holds {row count, first row}
// (block_no, always 0 for the single partitioned build block, carries the
// count).  Nothing follows a chain then, and none is written.  33.5M rows of
// 27 bytes in 131,072 leaves, beside the probe side's pass: 1,082 us, against
// 566 for the tables and 820 for a second kernel that found every row's cell
// again in memory (the join 7,260 -> 6,990).  Bound by the latency of a
// leaf's steps.
template <int NT, bool kGroup>
__global__ void __launch_bounds__(NT) k_build_leaf(const __grid_constant__ Cols part, const __grid_constant__ Cols dst, const uint32_t * __restrict__ leaf_off,
                                                         const uint32_t * __restrict__ table_off, int ulog, const int * __restrict__ stop, uint32_t smem_cells,
                                                         Cell * __restrict__ cells, uint64_t * __restrict__ next, LeafMeta * __restrict__ meta,
                                                         int * __restrict__ any_dup)
{
    extern __shared__ __align__(16) Cell sh_cells[]; // | (kGroup) cnt[smem_cells] | place of each row[smem_cells]
    __shared__ int dup;
    __shared__ uint32_t warp_sums[NT / 32];
    const uint64_t * keys = part.keys;
    const uint32_t l = blockIdx.x;
    const uint32_t r0 = leaf_off[l], r = leaf_off[l + 1] - r0;
    const uint64_t t0 = ulog >= 0 ? ((uint64_t)l << ulog) : table_off[l];
    const uint64_t cap = ulog >= 0 ? (1ull << ulog) : table_off[l + 1] - t0;
    if (threadIdx.x == 0)
        dup = 0;
    const int stopped = stop ? __ldg(stop) : 0; // (looked at when the table is cleared)
    const Cell empty{0ull, INVALID_REF};
    if (r == 0)
    {
        for (uint64_t i = threadIdx.x; i < cap; i += NT) // uniform layout: an empty table
            reinterpret_cast<ulonglong2 *>(cells + t0)[i] = make_ulonglong2(0ull, INVALID_REF);
        if (threadIdx.x == 0)
            meta[l] = LeafMeta{t0, r0, cap ? (uint8_t)log2u(cap) : (uint8_t)0, 0, 0, 0};
        return;
    }
    // (Only where `stopped`: the bound is for the compiler.  With it this form
    // has 31 registers and no spills, 1,080 us for the workload above against
    // 1,160; the other form is better without: the table of a leaf with a key
    // of 100,000 rows takes 565 us, 1,070 with it.)
    if (kGroup && r >= cap)
        return;
    const bool in_smem = cap <= smem_cells;
    Cell * tab = in_smem ? sh_cells : cells + t0;
    for (uint64_t i = threadIdx.x; i < cap; i += NT)
        tab[i] = empty;
    __syncthreads();
    if (stopped)
        return; // some leaf is past the estimate: all are built again at the counted sizes
    bool my_dup = false;
    for (uint32_t i = threadIdx.x; i < r; i += NT)
    {
        const uint64_t k = keys[r0 + i];
        const uint64_t h = int_hash64(k);
        const uint64_t ref = make_ref(0, r0 + i);
        const uint64_t prev = in_smem ? table_insert<true>(tab, cap, h, k, ref) : table_insert<false>(tab, cap, h, k, ref);
        if constexpr (!kGroup)
            next[r0 + i] = prev;
        my_dup |= ref_valid(prev);
    }
    if (__any_sync(0xffffffffu, my_dup) && (threadIdx.x & 31) == 0)
        dup = 1;
    __syncthreads();
    if constexpr (kGroup)
        if (dup)
        {
            uint32_t * cnt = reinterpret_cast<uint32_t *>(sh_cells + smem_cells); // rows of each cell, then its first
            uint32_t * place = cnt + smem_cells;                                 // each row's cell | its rank in the cell << 13
            static_assert(kSmemCellsMax <= 1u << 13, "a cell and a rank in 32 bits");
            const uint32_t c_n = (uint32_t)cap;
            for (uint32_t i = threadIdx.x; i < c_n; i += NT)
                cnt[i] = 0;
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < r; i += NT)
            {
                const uint64_t k = keys[r0 + i];
                const uint32_t c = cell_of(tab, cap, int_hash64(k), k);
                place[i] = c | atomicAdd(&cnt[c], 1u) << 13;
            }
            __syncthreads();
            // one block scan: thread t owns cells [t * per, (t + 1) * per)
            const uint32_t per = (c_n + NT - 1) / NT, c0 = threadIdx.x * per;
            uint32_t local = 0;
            for (uint32_t j = 0; j < per; ++j)
                if (c0 + j < c_n)
                    local += cnt[c0 + j];
            uint32_t tot;
            uint32_t run = block_excl_scan<NT>(local, warp_sums, &tot);
            for (uint32_t j = 0; j < per; ++j)
                if (c0 + j < c_n)
                {
                    const uint32_t v = cnt[c0 + j];
                    cnt[c0 + j] = run;
                    if (v)
                        tab[c0 + j].ref = make_ref(v, r0 + run);
                    run += v;
                }
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < r; i += NT)
                copy_row(part, r0 + i, dst, (uint64_t)r0 + cnt[place[i] & (kSmemCellsMax - 1u)] + (place[i] >> 13));
        }
    if (in_smem)
    {
        ulonglong2 * dst = reinterpret_cast<ulonglong2 *>(cells + t0);
        const ulonglong2 * src = reinterpret_cast<const ulonglong2 *>(sh_cells);
        for (uint64_t i = threadIdx.x; i < cap; i += NT)
            dst[i] = src[i];
    }
    if (threadIdx.x == 0)
    {
        meta[l] = LeafMeta{t0, r0, (uint8_t)log2u(cap), 1, (uint8_t)dup, 0};
        if (dup)
            atomicOr(any_dup, kLeafRepeats);
    }
}

// ---- inline tables (PHJ-PURE, unique keys, at most 8 payload bytes) ----------
// One CTA per leaf; a table of `cap` cells {key, packed payload} at leaf *
// cap, built in shared memory with 64-bit compare-and-swaps on the keys and
// streamed out.  An empty cell holds a key of another leaf.  A repeated key
// or a leaf of more than most_rows rows sets *bad (the table is then unusable).
// Bound by the write of the tables (16 bytes a cell, 2.2 to 2.9 cells a
// row): 3M rows in 16,384 leaves 60 us, 2.9 TB/s, where the general tables,
// their next-chain and the payload packing took 115.  kRows: shared memory
// holds the keys and their rows only (10 bytes a cell).
template <int NT, bool kRows>
__global__ void __launch_bounds__(NT, kRows ? 2 : 1) k_build_inline(const __grid_constant__ Cols part, const uint32_t * __restrict__ leaf_off,
                                                     const __grid_constant__ PackSpec pk, const __grid_constant__ InlineTables t,
                                                     uint32_t most_rows, int * __restrict__ bad)
{
    extern __shared__ __align__(16) ulonglong2 icells[]; // (kRows: keys[cap] | rows[cap])
    uint64_t * ikeys = reinterpret_cast<uint64_t *>(icells);
    uint16_t * irows = reinterpret_cast<uint16_t *>(ikeys + t.cap);
    constexpr uint32_t kStride = kRows ? 1 : 2; // 8-byte words from key to key
    const uint32_t l = blockIdx.x;
    const uint32_t r0 = leaf_off[l], r = leaf_off[l + 1] - r0;
    const uint64_t none = t.empty_key(l);
    // another leaf's build may have found the tables unusable (one thread
    // asks: every warp of 16K CTAs reading one word took 60 us)
    // (the first kLookers CTAs look through all leaves, a share each)
    if (blockIdx.x < kLookers)
    {
        const uint32_t lookers = min(gridDim.x, kLookers);
        const uint32_t l0 = (uint32_t)((uint64_t)gridDim.x * blockIdx.x / lookers), l1 = (uint32_t)((uint64_t)gridDim.x * (blockIdx.x + 1) / lookers);
        if (past_estimate(leaf_off, l0, l1, NT, most_rows))
            atomicOr(bad, kLeafOverflow);
    }
    const int stop = threadIdx.x == 0 ? *reinterpret_cast<volatile int *>(bad) : 0;
    if (r > most_rows) // (fewer than t.cap)
    {
        if (threadIdx.x == 0)
            atomicOr(bad, kLeafOverflow);
        return;
    }
    for (uint32_t i = threadIdx.x; i < t.cap; i += NT)
    {
        if constexpr (kRows)
            ikeys[i] = none;
        else
            icells[i] = make_ulonglong2(none, 0ull);
    }
    if (__syncthreads_or(stop))
        return;
    auto payload = [&](uint32_t i) -> uint64_t {
        uint64_t v = 0;
        for (uint32_t c = 0; c < part.n; ++c)
        {
            uint64_t x;
            switch (part.width[c])
            {
                case 1: x = static_cast<const uint8_t *>(part.col[c])[r0 + i]; break;
                case 2: x = static_cast<const uint16_t *>(part.col[c])[r0 + i]; break;
                case 4: x = static_cast<const uint32_t *>(part.col[c])[r0 + i]; break;
                default: x = static_cast<const uint64_t *>(part.col[c])[r0 + i]; break;
            }
            v |= x << (pk.off[c] * 8u);
        }
        return v;
    };
    bool repeats = false;
    for (uint32_t i = threadIdx.x; i < r && !repeats; i += NT)
    {
        const uint64_t k = part.keys[r0 + i];
        const uint64_t v = kRows ? 0ull : payload(i);
        uint32_t pos = t.start(int_hash64(k));
        for (;;) // fewer rows than cells: an empty one is found
        {
            const unsigned long long old = atomicCAS(reinterpret_cast<unsigned long long *>(ikeys + pos * kStride), none, k);
            if (old == none)
            {
                if constexpr (kRows)
                    irows[pos] = (uint16_t)i;
                else
                    icells[pos].y = v;
                break;
            }
            if (old == k)
            {
                repeats = true;
                break;
            }
            pos = pos + 1 == t.cap ? 0 : pos + 1;
        }
    }
    if (__syncthreads_or(repeats))
    {
        if (threadIdx.x == 0)
            atomicOr(bad, kLeafRepeats);
        return;
    }
    ulonglong2 * dst = t.cells + (uint64_t)l * t.cap;
    for (uint32_t i = threadIdx.x; i < t.cap; i += NT)
    {
        if constexpr (kRows)
        {
            const uint64_t key = ikeys[i];
            dst[i] = make_ulonglong2(key, key != none ? payload(irows[i]) : 0ull);
        }
        else
            dst[i] = icells[i];
    }
}

// ---- grouped duplicates (PHJ-PURE with repeated build keys) ----------------
// One CTA per leaf.  The payloads of one key's rows become contiguous in
// `dst`; the key's cell then holds {row count, first row} (block_no, which is
// always 0 for the single partitioned build block, carries the count).
// Leaves without repeated keys are copied unchanged.  A grouped leaf is read
// through its cells only, so neither keys nor a next-chain are written.
// For builds that did not group (LeafTables::groups): at most 11 radix bits
// (no second set of columns at hand), or tables built in place.  Bound by the latency of a leaf's steps (a row's cell, its place, its
// payloads).  33.5M rows of 27 bytes in 131,072 leaves, beside the probe
// side's pass: 946 us with keys and next-chain, 820 without.
__global__ void __launch_bounds__(kBuildNT) k_group_leaf(const __grid_constant__ Cols src, const __grid_constant__ Cols dst,
                                                         const uint32_t * __restrict__ leaf_off, const LeafMeta * __restrict__ meta,
                                                         Cell * __restrict__ cells)
{
    extern __shared__ uint32_t gsh[]; // cnt[cap] | fill[cap] | cell of each row[cap]
    __shared__ uint32_t warp_sums[kBuildNT / 32];
    const uint32_t l = blockIdx.x;
    const uint32_t r0 = leaf_off[l], r = leaf_off[l + 1] - r0;
    if (r == 0)
        return;
    const LeafMeta m = meta[l];
    if (!m.dup)
    {
        for (uint32_t i = threadIdx.x; i < r; i += kBuildNT)
            copy_row(src, r0 + i, dst, r0 + i);
        return;
    }
    const uint32_t cap = 1u << m.log2cap;
    Cell * tab = cells + m.table_off;
    uint32_t * cnt = gsh;
    uint32_t * fill = gsh + cap;
    uint32_t * rowcell = gsh + 2 * cap; // a leaf has at most cap rows
    for (uint32_t i = threadIdx.x; i < cap; i += kBuildNT)
        cnt[i] = 0;
    __syncthreads();
    // each row's cell, found once and kept for the placement below
    for (uint32_t i = threadIdx.x; i < r; i += kBuildNT)
    {
        const uint64_t k = src.keys[r0 + i];
        const uint32_t c = cell_of(tab, cap, int_hash64(k), k);
        rowcell[i] = c;
        atomicAdd(&cnt[c], 1u);
    }
    __syncthreads();
    // one block scan: thread t owns cells [t * per, (t + 1) * per)
    const uint32_t per = (cap + kBuildNT - 1) / kBuildNT;
    const uint32_t c0 = threadIdx.x * per;
    uint32_t local = 0;
    for (uint32_t j = 0; j < per; ++j)
        if (c0 + j < cap)
            local += cnt[c0 + j];
    uint32_t tot;
    uint32_t run = block_excl_scan<kBuildNT>(local, warp_sums, &tot);
    for (uint32_t j = 0; j < per; ++j)
        if (c0 + j < cap)
        {
            const uint32_t c = c0 + j, v = cnt[c];
            fill[c] = run;
            if (v)
                tab[c].ref = make_ref(v, r0 + run);
            run += v;
        }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < r; i += kBuildNT)
    {
        const uint32_t c = rowcell[i];
        const uint32_t slot = atomicAdd(&fill[c], 1u);
        copy_row(src, r0 + i, dst, (uint64_t)r0 + slot);
    }
}

// ---- CHJ --------------------------------------------------------------------

__global__ void k_slot_hist(const uint64_t * __restrict__ keys, uint64_t n, uint32_t slot_bits, uint32_t * __restrict__ counts)
{
    extern __shared__ uint32_t bins[];
    const uint32_t nb = 1u << slot_bits;
    for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x)
        bins[i] = 0;
    __syncthreads();
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        atomicAdd(&bins[int_hash64(keys[i]) >> (64 - slot_bits)], 1u);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x)
        if (bins[i])
            atomicAdd(&counts[i], bins[i]);
}

// Rows of each of 2^slot_bits (at most 1024) sub-tables, and by the last CTA
// to finish the tables themselves: their cells (as table_cells) laid end to
// end in meta, the sum in counts[nb + 1] (counts[nb] counts CTAs; all zero
// before).  Bound by the keys' latency and one global atomic a CTA and
// sub-table: one CTA of 1024 threads a SM, four loads in flight (669K rows
// 10.7 us; 1,216 CTAs of 256 threads, a load at a time, 16.4).
__global__ void __launch_bounds__(1024) k_slot_plan(const uint64_t * __restrict__ keys, uint64_t n, uint32_t slot_bits, uint32_t * __restrict__ counts,
                                                    LeafMeta * __restrict__ meta)
{
    __shared__ uint32_t bins[1024];
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t s_last;
    const uint32_t nb = 1u << slot_bits, t = threadIdx.x;
    bins[t] = 0;
    __syncthreads();
    const uint64_t stride = (uint64_t)gridDim.x * 1024;
    for (uint64_t i = (uint64_t)blockIdx.x * 1024 + t; i < n; i += 4 * stride)
    {
        uint64_t k[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            k[u] = i + u * stride < n ? keys[i + u * stride] : 0ull;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i + u * stride < n)
                atomicAdd(&bins[int_hash64(k[u]) >> (64 - slot_bits)], 1u);
    }
    __syncthreads();
    if (t < nb && bins[t])
        atomicAdd(&counts[t], bins[t]);
    __threadfence();
    __syncthreads();
    if (t == 0)
        s_last = atomicAdd(&counts[nb], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last)
        return;
    __threadfence();
    const uint32_t r = t < nb ? __ldcg(counts + t) : 0u;
    const uint32_t cap = (uint32_t)table_cells(r, 200);
    uint32_t total;
    const uint32_t off = block_excl_scan<1024>(cap, warp_sums, &total);
    if (t < nb)
        meta[t] = LeafMeta{off, 0u, cap ? (uint8_t)log2u(cap) : (uint8_t)0, (uint8_t)(r != 0), 0, 0};
    if (t == 0)
        counts[nb + 1] = total;
}

__global__ void k_slot_meta(const uint32_t * __restrict__ counts, const uint32_t * __restrict__ table_off, uint32_t n_slots, LeafMeta * __restrict__ meta)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n_slots)
        return;
    const uint64_t cap = table_off[s + 1] - table_off[s];
    meta[s] = LeafMeta{table_off[s], 0u, cap ? (uint8_t)log2u(cap) : (uint8_t)0, (uint8_t)(counts[s] != 0), 0, 0};
}

// n cells, or *n_dev.
__global__ void k_fill_empty(Cell * __restrict__ cells, uint64_t n, const uint32_t * __restrict__ n_dev)
{
    if (n_dev)
        n = *n_dev;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        reinterpret_cast<ulonglong2 *>(cells)[i] = make_ulonglong2(0ull, INVALID_REF);
}

__device__ __forceinline__ uint32_t block_of_row(uint64_t g, const uint64_t * __restrict__ block_off, uint32_t n_blocks, uint32_t uniform)
{
    if (uniform)
        return (uint32_t)(g / uniform);
    uint32_t lo = 0, hi = n_blocks; // block_off[lo] <= g < block_off[hi]
    while (hi - lo > 1)
    {
        const uint32_t mid = (lo + hi) >> 1;
        if (block_off[mid] <= g)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

__global__ void k_chj_insert(const uint64_t * __restrict__ keys, uint64_t n, uint32_t slot_bits, const uint64_t * __restrict__ block_off,
                             uint32_t n_blocks, uint32_t uniform, Cell * __restrict__ cells, LeafMeta * __restrict__ meta, uint64_t * __restrict__ next,
                             int * __restrict__ any_dup)
{
    for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n; g += (uint64_t)gridDim.x * blockDim.x)
    {
        const uint64_t k = keys[g];
        const uint64_t h = int_hash64(k);
        const uint32_t s = (uint32_t)(h >> (64 - slot_bits));
        const uint32_t b = block_of_row(g, block_off, n_blocks, uniform);
        const uint32_t row = (uint32_t)(g - block_off[b]);
        const LeafMeta m = meta[s];
        const uint64_t prev = table_insert<false>(cells + m.table_off, 1ull << m.log2cap, h, k, make_ref(b, row));
        next[g] = prev;
        // flags read before they are written: a repeated key must not make
        // every thread store to the same two addresses
        if (ref_valid(prev))
        {
            if (!*reinterpret_cast<volatile uint8_t *>(&meta[s].dup))
                meta[s].dup = 1;
            if (!*reinterpret_cast<volatile int *>(any_dup))
                *any_dup = 1;
        }
    }
}

// The leaves without repeated keys of a build that grouped the others: their
// payloads in the same order, a warp per leaf.
__global__ void k_copy_leaves(const __grid_constant__ Cols src, const __grid_constant__ Cols dst, const uint32_t * __restrict__ leaf_off, uint32_t n_leaves,
                              const LeafMeta * __restrict__ meta)
{
    const uint32_t l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (l >= n_leaves || meta[l].dup)
        return;
    for (uint32_t i = leaf_off[l] + (threadIdx.x & 31); i < leaf_off[l + 1]; i += 32)
        copy_row(src, i, dst, i);
}
} // namespace

// Rows of the largest leaf, with a margin of six standard deviations of a
// uniform hash (and eight rows): a join whose keys spread evenly stays
// within it, one that does not is found out by the build itself.
static uint64_t leaf_rows_estimate(uint64_t rows, uint64_t n_leaves)
{
    const double m = (double)rows / (double)n_leaves;
    return (uint64_t)(m + 6.0 * std::sqrt(m) + 8.0);
}

// Cells a leaf of an inline table that holds `est` rows at the load.
static uint64_t inline_cells(uint64_t est, uint32_t pct)
{
    return (std::max(est * pct / 100, est + 1) + 1) & ~1ull;
}

// Whether general tables of `est` rows a leaf are sized by that estimate: up
// to 9 cells a row at the default load.  Leaves of 390 rows have 5.2 then, and
// 2.6 by their count: 100K x 800K rows of 12 payload bytes 104 us against 150,
// 900K x 7.2M 231 and 292, 7M x 56M 1,322 and 1,466, 14M x 64M 1,825 and 1,957;
// 28M x 64M 2,713 and 2,581.
static bool estimate_fits(uint64_t rows, uint64_t n_leaves, uint64_t est, uint32_t pct)
{
    return n_leaves * table_cells(est, pct) * 200 <= 9 * rows * pct;
}

uint64_t estimated_table_bytes(uint64_t rows, uint32_t total_bits, uint64_t payload_bytes, bool unique)
{
    constexpr uint32_t kPct = 200;
    const uint64_t n_leaves = 1ull << total_bits, est = leaf_rows_estimate(rows, n_leaves);
    uint64_t bytes = 0;
    const bool in_cells = payload_bytes <= 8 && rows >> total_bits >= kInlineLeafRows;
    if (in_cells)
        bytes = n_leaves * inline_cells(est, kPct) * sizeof(Cell);
    if (!(in_cells && unique) && estimate_fits(rows, n_leaves, est, kPct))
        bytes = std::max(bytes, n_leaves * table_cells(est, kPct) * sizeof(Cell) + rows * 8);
    return bytes;
}

// Rows that a table of `cells` may hold at the load the option allows.
static uint32_t rows_at_load(uint64_t cells, uint32_t pct)
{
    return (uint32_t)std::min<uint64_t>(std::min(cells - 1, cells * 100 / pct), 0xFFFFFFFFu);
}

bool build_inline_tables(phj_ctx * ctx, Scratch & s, const Cols & part, uint64_t rows, const uint32_t * leaf_off, uint32_t total_bits,
                         const PackSpec & pk, InlineTables & t, int * bad)
{
    const uint64_t n_leaves = 1ull << total_bits;
    // fewer rows a leaf: the margin would make the tables sparse
    if (rows >> total_bits < kInlineLeafRows)
        return false;
    const uint64_t est = leaf_rows_estimate(rows, n_leaves);
    t.cap = (uint32_t)std::min<uint64_t>(inline_cells(est, ctx->table_cap_pct), 1u << 30);
    const size_t smem = (size_t)t.cap * 16;
    if (smem + 2048 > ctx->smem_optin || ctx->table_cap_pct < 125)
        return false;
    t.leaf_shift = 64u - total_bits;
    // a key of the lower and of the upper half of the leaves
    for (uint64_t k = 1, have = 0; have != 3; ++k)
    {
        const uint32_t top = (uint32_t)(int_hash64(k) >> 63);
        if (!(have >> top & 1u))
            t.half_key[top] = k;
        have |= 1ull << top;
    }
    t.half_shift = total_bits - 1;
    t.cells = reinterpret_cast<ulonglong2 *>(s.get<Cell>(n_leaves * t.cap));
    KTimer kt(ctx, "build_inline", rows, rows * 16 + n_leaves * t.cap * 16);
    // leaves of more than 1024 rows get 1024 threads; where two such CTAs do
    // not fit on a SM with cells in shared memory, keys and rows are held
    // there and the payloads are read as the cells go out (256 leaves of
    // 4096 rows: 24 us against 28, in one wave of CTAs)
    const uint32_t most = rows_at_load(t.cap, ctx->table_cap_pct);
    const size_t lean = (size_t)t.cap * 10, two = (ctx->smem_optin + 1024) / 2 - 2048;
    if (est > 1024 && smem > two && lean <= two)
        k_build_inline<1024, true><<<(unsigned)n_leaves, 1024, lean, ctx->stream>>>(part, leaf_off, pk, t, most, bad);
    else if (est > 1024)
        k_build_inline<1024, false><<<(unsigned)n_leaves, 1024, smem, ctx->stream>>>(part, leaf_off, pk, t, most, bad);
    else
        k_build_inline<kBuildNT, false><<<(unsigned)n_leaves, kBuildNT, smem, ctx->stream>>>(part, leaf_off, pk, t, most, bad);
    PHJ_LAUNCHED(ctx, "build_inline");
    return true;
}

void set_build_smem_limits(int smem_optin)
{
    for (const auto kernel : {k_build_inline<kBuildNT, false>, k_build_inline<1024, false>, k_build_inline<1024, true>})
        PHJ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin - 1024));
    const size_t need = (size_t)kSmemCellsMax * sizeof(Cell);
    for (const auto kernel : {k_build_leaf<kBuildNT, false>, k_build_leaf<1024, false>, k_build_leaf<kBuildNT, true>, k_build_leaf<1024, true>})
        PHJ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)std::min<size_t>(need + need / 2, (size_t)smem_optin - 1024)));
    PHJ_CUDA(cudaFuncSetAttribute(k_group_leaf, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)std::min<size_t>((size_t)kSmemCellsMax * 12, (size_t)smem_optin - 1024)));
}

bool group_leaf_duplicates(phj_ctx * ctx, const Cols & src, const Cols & dst, const uint32_t * leaf_off, uint32_t n_leaves, const LeafTables & lt)
{
    const uint64_t max_cap = lt.max_rows ? table_cells(lt.max_rows, ctx->table_cap_pct) : 1;
    if (!lt.any_dup || max_cap > kSmemCellsMax || lt.state)
        return false;
    KTimer kt(ctx, "group_leaf", 0, 0);
    if (lt.groups)
    {
        k_copy_leaves<<<(unsigned)ceil_div(n_leaves, 8), 256, 0, ctx->stream>>>(src, dst, leaf_off, n_leaves, lt.meta);
        PHJ_LAUNCHED(ctx, "copy_leaves");
        return true;
    }
    k_group_leaf<<<n_leaves, kBuildNT, (size_t)max_cap * 12, ctx->stream>>>(src, dst, leaf_off, lt.meta, lt.cells);
    PHJ_LAUNCHED(ctx, "group_leaf");
    return true;
}

// Lazy layout (PHJ/BEP): the directory says where each leaf's table lives;
// the cells are built on first use by the probe (state NOT_BUILT).
__global__ void k_leaf_plan(const uint32_t * __restrict__ leaf_off, const uint32_t * __restrict__ table_off, int ulog, uint32_t n_leaves,
                            LeafMeta * __restrict__ meta)
{
    const uint32_t l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= n_leaves)
        return;
    const uint32_t r0 = leaf_off[l], r = leaf_off[l + 1] - r0;
    const uint64_t t0 = ulog >= 0 ? ((uint64_t)l << ulog) : table_off[l];
    const uint64_t cap = ulog >= 0 ? (1ull << ulog) : table_off[l + 1] - t0;
    (void)r;
    meta[l] = LeafMeta{t0, r0, cap ? (uint8_t)log2u(cap) : (uint8_t)0, (uint8_t)(cap != 0), 1, 0};
}

void build_leaf_tables(phj_ctx * ctx, Scratch & s, const Cols & build_part, const uint32_t * leaf_off, uint32_t n_leaves, LeafTables & lt,
                       bool lazy, uint64_t estimate_rows, const Cols * group_dst)
{
    uint32_t * table_off = nullptr;
    uint32_t * small = s.get<uint32_t>(4); // [0] max rows, [1] flags (kLeafRepeats, kLeafOverflow), [2] a leaf is past the estimate
    PHJ_CUDA(cudaMemsetAsync(small, 0, 4 * sizeof(uint32_t), ctx->stream));
    lt.flags = reinterpret_cast<int *>(small + 1);
    uint64_t max_cap;
    const uint64_t est = estimate_rows ? leaf_rows_estimate(estimate_rows, n_leaves) : 0;
    lt.estimated = est && estimate_fits(estimate_rows, n_leaves, est, ctx->table_cap_pct);
    if (lt.estimated)
    {
        // uniform tables at the estimated size: no size is read back before
        // the build
        lt.max_rows = (uint32_t)est;
        max_cap = table_cells(est, ctx->table_cap_pct);
        lt.uniform_log2cap = (int)(63 - __builtin_clzll(max_cap));
        lt.total_cells = (uint64_t)n_leaves * max_cap;
    }
    else
    {
        uint32_t * caps = s.get<uint32_t>(n_leaves + 1);
        table_off = s.get<uint32_t>(n_leaves + 1);
        k_leaf_caps<<<(unsigned)ceil_div(n_leaves, 256), 256, 0, ctx->stream>>>(leaf_off, n_leaves, ctx->table_cap_pct, caps, small);
        PHJ_LAUNCHED(ctx, "leaf_caps");
        scan_u32(ctx, s, caps, table_off, n_leaves);
        uint32_t host[2] = {0, 0};
        read_small(ctx, {{&host[0], small, sizeof(uint32_t)}, {&host[1], table_off + n_leaves, sizeof(uint32_t)}});
        lt.max_rows = host[0];
        // at least one aligned cell pair: the probe's first load reads two cells
        max_cap = lt.max_rows ? table_cells(lt.max_rows, ctx->table_cap_pct) : 2;
        // Uniform capacity (the largest leaf's) lets the probe compute a table's
        // address from the leaf id alone; it is used unless it costs more than
        // 1.5x the cells of per-leaf sizing.
        const uint64_t uniform_cells = (uint64_t)n_leaves * max_cap;
        const bool uniform = uniform_cells <= (3 * (uint64_t)host[1]) / 2 + n_leaves;
        lt.uniform_log2cap = uniform ? (int)(63 - __builtin_clzll(max_cap)) : -1;
        lt.total_cells = uniform ? uniform_cells : host[1];
    }
    lt.max_cells = max_cap;
    lt.meta = s.get<LeafMeta>(n_leaves);
    lt.cells = s.get<Cell>(lt.total_cells);
    if (lazy)
    {
        lt.state = s.get<uint32_t>(n_leaves);
        PHJ_CUDA(cudaMemsetAsync(lt.state, 0, (size_t)n_leaves * sizeof(uint32_t), ctx->stream));
        k_leaf_plan<<<(unsigned)ceil_div(n_leaves, 256), 256, 0, ctx->stream>>>(leaf_off, table_off, lt.uniform_log2cap, n_leaves, lt.meta);
        PHJ_LAUNCHED(ctx, "leaf_plan");
        lt.any_dup = 1; // unknown until the tables are built: chains are followed
        return;
    }
    // Tables are built in shared memory and copied out when two CTAs fit
    // on an SM; larger ones (one resident CTA per SM would leave the SMs
    // idling through each leaf's copy-out) are built in place, in global
    // memory that stays in L2 (1M x 8M, 256 leaves of 8192 cells: 0.310 ->
    // 0.304 ms a join).
    const uint32_t smem_cells =
        max_cap * sizeof(Cell) * 2 <= ctx->smem_optin ? (uint32_t)std::min<uint64_t>(max_cap, kSmemCellsMax) : 0u;
    {
        KTimer kt(ctx, "build_leaf_tables", 0, 0);
        int * stop = reinterpret_cast<int *>(small + 2);
        if (lt.estimated)
        {
            k_leaf_check<<<(unsigned)ceil_div(n_leaves, 256), 256, 0, ctx->stream>>>(leaf_off, n_leaves, rows_at_load(max_cap, ctx->table_cap_pct), lt.flags, stop);
            PHJ_LAUNCHED(ctx, "leaf_check");
        }
        // leaves of more than 1024 rows get 1024 threads
        const bool large = lt.max_rows > 1024;
        lt.groups = group_dst && smem_cells && smem_cells == max_cap;
        const auto kb = lt.groups ? (large ? k_build_leaf<1024, true> : k_build_leaf<kBuildNT, true>)
                                  : (large ? k_build_leaf<1024, false> : k_build_leaf<kBuildNT, false>);
        kb<<<n_leaves, large ? 1024 : kBuildNT, (size_t)smem_cells * (lt.groups ? sizeof(Cell) + 8 : sizeof(Cell)), ctx->stream>>>(
            build_part, group_dst ? *group_dst : Cols{}, leaf_off, table_off, lt.uniform_log2cap, lt.estimated ? stop : nullptr, smem_cells, lt.cells, lt.next, lt.meta, lt.flags);
        PHJ_LAUNCHED(ctx, "build_leaf");
    }
    lt.any_dup = 0; // unknown until the flags are read
    if (!lt.estimated)
        read_small(ctx, {{&lt.any_dup, lt.flags, sizeof(int)}});
}

void build_global_table(phj_ctx * ctx, Scratch & s, const phj_table & build, uint32_t slot_bits, LeafTables & lt)
{
    const uint32_t n_slots = 1u << slot_bits;
    const uint64_t n = build.rows;
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(n, 256), (uint64_t)ctx->num_sms * 8));
    uint32_t * counts = s.get<uint32_t>(n_slots + 3); // and the plan's CTA count and total; the repeated-key flag
    int * any_dup = reinterpret_cast<int *>(counts + n_slots + 2);
    PHJ_CUDA(cudaMemsetAsync(counts, 0, (n_slots + 3) * sizeof(uint32_t), ctx->stream));
    lt.meta = s.get<LeafMeta>(n_slots);
    // Up to 16M rows the cells are allocated at the most they can be (four a
    // row, 1 GiB), so their number is not read back and one launch counts and
    // plans: the tables' fill starts 12 us after the count did instead of 47
    // (342K x 3.6M rows: 208 -> 170 us a join, 669K x 2.7M 213 -> 177).  More
    // rows are counted first: the exact size is then worth the round trip.
    const bool plan = n <= (16u << 20) && n_slots <= 1024 && !ctx->lean;
    if (plan)
    {
        lt.total_cells = std::max<uint64_t>(4 * n, 2);
        lt.cells = s.get<Cell>(lt.total_cells);
        KTimer kt(ctx, "chj_slot_hist", n, n * 8);
        k_slot_plan<<<(unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(n, 4096), (uint64_t)ctx->num_sms)), 1024, 0, ctx->stream>>>(
            build.keys, n, slot_bits, counts, lt.meta);
        PHJ_LAUNCHED(ctx, "chj_slot_hist");
    }
    else
    {
        uint32_t * caps = s.get<uint32_t>(n_slots + 1);
        uint32_t * table_off = s.get<uint32_t>(n_slots + 1);
        {
            KTimer kt(ctx, "chj_slot_hist", n, n * 8);
            k_slot_hist<<<grid, 256, n_slots * sizeof(uint32_t), ctx->stream>>>(build.keys, n, slot_bits, counts);
            PHJ_LAUNCHED(ctx, "chj_slot_hist");
        }
        uint32_t * max_rows = s.get<uint32_t>(1);
        PHJ_CUDA(cudaMemsetAsync(max_rows, 0, sizeof(uint32_t), ctx->stream));
        // counts -> capacities -> offsets: the offsets of leaf_off-style caps
        // reuse k_leaf_caps on a prefix of the counts.
        uint32_t * cnt_off = s.get<uint32_t>(n_slots + 1);
        scan_u32(ctx, s, counts, cnt_off, n_slots);
        k_leaf_caps<<<(unsigned)ceil_div(n_slots, 256), 256, 0, ctx->stream>>>(cnt_off, n_slots, 200u, caps, max_rows);
        PHJ_LAUNCHED(ctx, "chj_caps");
        scan_u32(ctx, s, caps, table_off, n_slots);
        uint32_t total = 0;
        read_small(ctx, {{&total, table_off + n_slots, sizeof(uint32_t)}});
        lt.total_cells = total;
        lt.cells = s.get<Cell>(total);
        k_slot_meta<<<(unsigned)ceil_div(n_slots, 256), 256, 0, ctx->stream>>>(counts, table_off, n_slots, lt.meta);
        PHJ_LAUNCHED(ctx, "chj_meta");
    }
    {
        KTimer kt(ctx, "chj_fill", 0, plan ? 0 : lt.total_cells * 16ull);
        k_fill_empty<<<(unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(lt.total_cells, 256), (uint64_t)ctx->num_sms * 16)), 256, 0,
                       ctx->stream>>>(lt.cells, lt.total_cells, plan ? counts + n_slots + 1 : nullptr);
        PHJ_LAUNCHED(ctx, "chj_fill");
    }
    {
        KTimer kt(ctx, "chj_insert", n, n * 16);
        k_chj_insert<<<grid, 256, 0, ctx->stream>>>(build.keys, n, slot_bits, build.block_off, build.n_blocks, build.uniform_block_rows, lt.cells,
                                                   lt.meta, lt.next, any_dup);
        PHJ_LAUNCHED(ctx, "chj_insert");
    }
    read_small(ctx, {{&lt.any_dup, any_dup, sizeof(int)}});
}

} // namespace phjg
