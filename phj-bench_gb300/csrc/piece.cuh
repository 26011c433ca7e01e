// piece.cuh -- joins against a table in shared memory, shared by the batched
// joins (batch.cu) and the small joins (small.cu): a CTA builds the table of
// a piece of the build side, its warps then probe on their own, without
// block barriers.
#pragma once

#include "common.cuh"

namespace phjg
{
// A lane's kU values of a payload column of at most 8 bytes, in 64-bit registers.
template <int kU>
__device__ __forceinline__ void load_rows(uint64_t (&v)[kU], const void * src, uint32_t width, const uint32_t (&idx)[kU], uint32_t one)
{
    switch (width)
    {
#define PHJ_LOAD4(W, T)                                                                                                                              \
    case W:                                                                                                                                          \
        _Pragma("unroll") for (int u = 0; u < kU; ++u) if (one >> u & 1u) v[u] = static_cast<const T *>(src)[idx[u]];                                 \
        break;
        PHJ_LOAD4(1, uint8_t)
        PHJ_LOAD4(2, uint16_t)
        PHJ_LOAD4(4, uint32_t)
        default: PHJ_LOAD4(8, uint64_t)
#undef PHJ_LOAD4
    }
}

template <int kU>
__device__ __forceinline__ void store_rows(const uint64_t (&v)[kU], void * dst, uint32_t width, uint64_t base, const uint32_t (&rel)[kU], uint32_t one)
{
    switch (width)
    {
#define PHJ_STORE4(W, T)                                                                                                                             \
    case W:                                                                                                                                          \
        _Pragma("unroll") for (int u = 0; u < kU; ++u) if (one >> u & 1u) __stcs(static_cast<T *>(dst) + base + rel[u], (T)v[u]);                     \
        break;
        PHJ_STORE4(1, uint8_t)
        PHJ_STORE4(2, uint16_t)
        PHJ_STORE4(4, uint32_t)
        default: PHJ_STORE4(8, uint64_t)
#undef PHJ_STORE4
    }
}

// A piece of at most kRows (a power of two) build rows has a table of slots
// {hash bits, row of the piece}: log2(kRows) bits of row, hash bits above
// them up to bit 30, kEmptySlot when free.
constexpr uint32_t kEmptySlot = 0xFFFFFFFFu;
constexpr uint32_t kNil = 0xFFFFu; // no row; end of a chain

// A slot's hash bits, in place (its group of slots is chosen by lower ones).
template <uint32_t kRows>
__device__ __forceinline__ uint32_t slot_tag(uint64_t h)
{
    return (uint32_t)(h >> 1) & 0x7FFFFFFFu & ~(kRows - 1);
}

// A piece's table in shared memory.
template <uint32_t kRows>
struct PieceTable
{
    const uint32_t * slots;
    const uint64_t * keys;
    const uint16_t * nxt;
    uint32_t mask;

    // The piece's row that heads `key`'s chain, kNil when the key is absent:
    // groups of four slots are filled from their first slot on, so a group
    // with an empty slot ends the search.
    __device__ __forceinline__ uint32_t find(uint64_t key) const
    {
        const uint64_t h = int_hash64(key);
        const uint32_t tag = slot_tag<kRows>(h);
        for (uint32_t pos = (uint32_t)h & mask & ~3u;; pos = (pos + 4) & mask) // some group has an empty slot
        {
            const uint4 s = *reinterpret_cast<const uint4 *>(slots + pos);
            const uint32_t v[4] = {s.x, s.y, s.z, s.w};
            // the group's last slot with the key's hash bits, without branches
            uint32_t row = kNil;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                row = (v[i] ^ tag) < kRows ? v[i] ^ tag : row;
            if (row != kNil)
            {
                if (keys[row] == key)
                    return row;
                // other keys with the same hash bits: one by one
                for (int i = 0; i < 4; ++i)
                    if ((v[i] ^ tag) < kRows && keys[v[i] ^ tag] == key)
                        return v[i] ^ tag;
            }
            if (s.w == kEmptySlot)
                return kNil;
        }
    }
};

__device__ __forceinline__ void prefetch_l2(const void * p)
{
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// Builds the table of `rows` build keys (`keys`, in memory) with all NT
// threads of the CTA: mask + 1 slots (a power of two, at least 4, more than
// the rows).  *linked (shared): 0 when no key repeats, otherwise 1 or, with
// kCount, the rows whose key was there already.  Ends with a barrier.
template <uint32_t kRows, int NT, bool kCount>
__device__ __forceinline__ void build_piece(const uint64_t * __restrict__ keys, uint32_t rows, uint32_t * slots, uint64_t * skeys, uint16_t * nxt,
                                            uint32_t mask, int * linked)
{
    if (threadIdx.x == 0)
        *linked = 0;
    for (uint32_t i = threadIdx.x; i <= mask; i += NT)
        slots[i] = kEmptySlot;
    for (uint32_t i = threadIdx.x; i < rows; i += NT)
        skeys[i] = keys[i];
    __syncthreads();
    int mine_linked = 0;
    for (uint32_t i = threadIdx.x; i < rows; i += NT)
    {
        const uint64_t k = skeys[i];
        const uint64_t h = int_hash64(k);
        const uint32_t tag = slot_tag<kRows>(h), mine = tag | i;
        uint32_t pos = (uint32_t)h & mask & ~3u, link = kNil;
        for (;; pos = (pos + 1) & mask) // fewer rows than slots: an empty one is found
        {
            uint32_t old = slots[pos];
            if (old == kEmptySlot)
                old = atomicCAS(&slots[pos], kEmptySlot, mine);
            if (old == kEmptySlot)
                break;
            if ((old ^ tag) < kRows && skeys[old ^ tag] == k)
            {
                // the key's slot, which stays the key's: this row becomes its
                // head in one exchange, whoever else does so meanwhile (with
                // compare-and-swaps 8,000 rows of one key took 6.5 ms, this
                // way 1.4)
                link = atomicExch(&slots[pos], mine) ^ tag;
                if constexpr (kCount)
                    ++mine_linked;
                else
                    *linked = 1;
                break;
            }
        }
        nxt[i] = (uint16_t)link;
    }
    if (kCount && mine_linked)
        atomicAdd(linked, mine_linked);
    __syncthreads();
}

// The columns a probe reads and writes.
struct ProbeSides
{
    Cols build, probe;
    uint64_t * out_keys;
    void * out_l[kMaxCols];
    void * out_r[kMaxCols];
    uint64_t out_cap;
};

// Four values a lane of an output column, to rows out[u].
__device__ __forceinline__ void store_at(const uint64_t (&v)[4], void * dst, uint32_t width, const uint64_t (&out)[4], uint32_t one)
{
    switch (width)
    {
#define PHJ_STORE_AT(W, T)                                                                                                                           \
    case W:                                                                                                                                          \
        _Pragma("unroll") for (int u = 0; u < 4; ++u) if (one >> u & 1u) static_cast<T *>(dst)[out[u]] = (T)v[u];                                     \
        break;
        PHJ_STORE_AT(1, uint8_t)
        PHJ_STORE_AT(2, uint16_t)
        PHJ_STORE_AT(4, uint32_t)
        default: PHJ_STORE_AT(8, uint64_t)
#undef PHJ_STORE_AT
    }
}

// The output rows of a probe row (`row`, of key `key`) whose matches are the
// chain from row b of the piece at c0 (kNil: none), o and those after it.
__device__ __forceinline__ void write_chain(const ProbeSides & J, uint64_t o, uint32_t b, uint64_t key, uint32_t row, uint32_t c0, const uint16_t * nxt)
{
    for (; b != kNil; b = nxt[b], ++o)
        if (o < J.out_cap)
        {
            J.out_keys[o] = key;
            for (uint32_t c = 0; c < J.build.n; ++c)
                copy_elem(J.out_l[c], o, J.build.col[c], c0 + b, J.build.width[c]);
            for (uint32_t c = 0; c < J.probe.n; ++c)
                copy_elem(J.out_r[c], o, J.probe.col[c], row, J.probe.width[c]);
        }
}

// The same for the 32 probe rows of a warp, one a lane, when one of them has
// more than four matches.  Every lane walks four rows of its chain; the warp
// then writes them eight chains at a time, four neighbouring lanes the four
// rows of one, at output rows that start at a multiple of four: a store fills
// sectors.  Bound by the stores and the build rows' gathers in L1.  A lane
// writing its chain alone waits for each row's loads, and its stores are
// quarters of sectors, which L2 reads back from memory when they do not meet
// (12.8M output rows, 8K build rows of 64 a key x 400K: 859 us a join of 20-byte
// rows and 1,429 of 32-byte ones, this way 200 and 300; 13.4M of 67 a key
// 1,217 and 347).
static __device__ __noinline__ void write_chains(const ProbeSides & J, uint64_t o, uint32_t b, uint64_t key, uint32_t row, uint32_t c0,
                                                 const uint16_t * nxt)
{
    const uint32_t lane = threadIdx.x & 31, e = lane & 3;
    const uint64_t out_cap = J.out_cap;
    uint32_t fifth = b;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        fifth = fifth != kNil ? nxt[fifth] : kNil;
    if (!__any_sync(0xffffffffu, fifth != kNil))
    {
        write_chain(J, o, b, key, row, c0, nxt);
        return;
    }
    uint32_t skip = (uint32_t)o & 3u; // groups of four start at multiples of four
    for (o -= skip;; o += 4, skip = 0)
    {
        uint32_t at[4];
        if (o >= out_cap)
            b = kNil;
        if (!__any_sync(0xffffffffu, b != kNil))
            return;
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k)
        {
            at[k] = k >= skip ? b : kNil;
            if (at[k] != kNil)
                b = nxt[b];
        }
        uint64_t out[4], v[4];
        uint32_t brow[4], prow[4], one = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            const int from = u * 8 + (int)(lane >> 2);
            uint32_t x = kNil;
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
            {
                const uint32_t y = __shfl_sync(0xffffffffu, at[k], from);
                x = e == k ? y : x;
            }
            brow[u] = c0 + x;
            prow[u] = __shfl_sync(0xffffffffu, row, from);
            out[u] = __shfl_sync(0xffffffffu, o, from) + e;
            v[u] = __shfl_sync(0xffffffffu, key, from);
            if (x != kNil && out[u] < out_cap)
                one |= 1u << u;
        }
        store_at(v, J.out_keys, 8, out, one);
        const uint32_t nl = J.build.n, nc = nl + J.probe.n;
#pragma unroll 1
        for (uint32_t c = 0; c < nc; ++c)
        {
            const bool left = c < nl;
            const uint32_t i = left ? c : c - nl, w = left ? J.build.width[i] : J.probe.width[i];
            const void * src = left ? J.build.col[i] : J.probe.col[i];
            void * dst = left ? J.out_l[i] : J.out_r[i];
            uint32_t idx[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                idx[u] = left ? brow[u] : prow[u];
            if (w <= 8)
            {
                load_rows(v, src, w, idx, one);
                store_at(v, dst, w, out, one);
            }
            else
            {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (one >> u & 1u)
                        static_cast<uint4 *>(dst)[out[u]] = static_cast<const uint4 *>(src)[idx[u]];
            }
        }
    }
}

// Whether a piece's keys repeat, and how a probe row's matches, a chain, are
// then written.
enum Repeats
{
    kUnique,
    kLaneWrites, // by its lane
    kWarpWrites  // by the whole warp, if a chain has more than four rows
};

// One warp probes rows first, first + step, ... of [.., p1), 32 * kU rows at
// a time, against the piece whose first build row is c0.  Output
// rows are reserved on *out_cur, a chunk at a time; rows past the capacity
// are counted and not written (and *over is set).
template <Repeats kRepeats, int kU, uint32_t kRows>
__device__ __forceinline__ void probe_piece(const ProbeSides & J, uint32_t first, uint32_t step, uint32_t p1, uint32_t c0,
                                            const PieceTable<kRows> & tab, unsigned long long * __restrict__ out_cur, int * __restrict__ over)
{
    constexpr bool kDup = kRepeats != kUnique;
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll 1
    for (uint32_t base = first; base < p1; base += step)
    {
        // the descriptor (in shared memory) is read where it is used: kept
        // out of the loop its three dozen pointers would be spilled
        asm volatile("" ::: "memory");
        const uint64_t * pkeys = J.probe.keys;
        const uint64_t out_cap = J.out_cap;
        uint64_t key[kU];
        uint32_t head[kU], rel[kU], total = 0, one = 0;
#pragma unroll
        for (int u = 0; u < kU; ++u)
        {
            const uint32_t r = base + u * 32 + lane;
            key[u] = r < p1 ? __ldcs(pkeys + r) : 0ull;
        }
        {
            // the warp's next chunk into L2, a line a lane
            const uint32_t next = base + step;
            const uint32_t rows = next < p1 ? min(32u * kU, p1 - next) : 0u;
            if (lane * 16 < rows)
                prefetch_l2(pkeys + next + lane * 16);
            for (uint32_t c = 0; c < J.probe.n; ++c)
                if (lane * 128 < rows * J.probe.width[c])
                    prefetch_l2(static_cast<const uint8_t *>(J.probe.col[c]) + (uint64_t)next * J.probe.width[c] + lane * 128);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u)
        {
            head[u] = base + u * 32 + lane < p1 ? tab.find(key[u]) : kNil;
            if (head[u] != kNil)
                one |= 1u << u;
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kU; ++u)
            if constexpr (kDup)
            {
                uint32_t cnt = 0;
                for (uint32_t b = head[u]; b != kNil; b = tab.nxt[b])
                    ++cnt;
                uint32_t x = cnt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1)
                {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= (uint32_t)o)
                        x += y;
                }
                rel[u] = total + x - cnt;
                total += __shfl_sync(0xffffffffu, x, 31);
            }
            else
            {
                const uint32_t m = __ballot_sync(0xffffffffu, one >> u & 1u);
                rel[u] = total + __popc(m & ((1u << lane) - 1u));
                total += __popc(m);
            }
        if (total == 0)
            continue;
        // the build payloads' columns, then the probe's; the first one's
        // loads go out before the reservation comes back, each next one's
        // before the last one's stores
        const uint32_t nl = J.build.n, nc = nl + J.probe.n;
        auto load_column = [&](uint32_t c, uint64_t (&v)[kU]) {
            uint32_t idx[kU];
            const bool left = c < nl;
#pragma unroll
            for (int u = 0; u < kU; ++u)
                idx[u] = left ? c0 + head[u] : base + u * 32 + lane;
            const uint32_t i = left ? c : c - nl;
            load_rows(v, left ? J.build.col[i] : J.probe.col[i], left ? J.build.width[i] : J.probe.width[i], idx, one);
        };
        unsigned long long o0 = 0;
        if (lane == 0)
        {
            o0 = atomicAdd(out_cur, (unsigned long long)total);
            if (o0 + total > out_cap)
                *over = 1;
        }
        uint64_t v[kU] = {};
        if (!kDup && nc)
            load_column(0, v);
        o0 = __shfl_sync(0xffffffffu, o0, 0);
        if constexpr (kDup)
        {
#pragma unroll
            for (int u = 0; u < kU; ++u)
                if constexpr (kRepeats == kLaneWrites)
                    write_chain(J, o0 + rel[u], head[u], key[u], base + u * 32 + lane, c0, tab.nxt);
                else
                    write_chains(J, o0 + rel[u], head[u], key[u], base + u * 32 + lane, c0, tab.nxt);
        }
        else
        {
            uint64_t * out = J.out_keys + o0;
            uint32_t fits = one;
#pragma unroll
            for (int u = 0; u < kU; ++u)
            {
                if (o0 + rel[u] >= out_cap)
                    fits &= ~(1u << u);
                if (fits >> u & 1u)
                    __stcs(out + rel[u], key[u]);
            }
#pragma unroll 1
            for (uint32_t c = 0; c < nc; ++c)
            {
                asm volatile("" ::: "memory");
                const bool left = c < nl;
                const uint32_t i = left ? c : c - nl, w = left ? J.build.width[i] : J.probe.width[i];
                void * dst = left ? J.out_l[i] : J.out_r[i];
                uint64_t nx[kU] = {};
                if (c + 1 < nc)
                    load_column(c + 1, nx);
                if (w <= 8)
                    store_rows(v, dst, w, o0, rel, fits);
                else
                {
                    const uint4 * src = static_cast<const uint4 *>(left ? J.build.col[i] : J.probe.col[i]);
#pragma unroll
                    for (int u = 0; u < kU; ++u)
                        if (fits >> u & 1u)
                            __stcs(static_cast<uint4 *>(dst) + o0 + rel[u], src[left ? c0 + head[u] : base + u * 32 + lane]);
                }
#pragma unroll
                for (int u = 0; u < kU; ++u)
                    v[u] = nx[u];
            }
        }
    }
}

} // namespace phjg
