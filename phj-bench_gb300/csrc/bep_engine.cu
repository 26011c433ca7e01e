// bep_engine.cu -- PHJ (best-effort partitioning, src/PHJBep.cpp:113-790)
// with the probe side's byte budget kept on the device.
//
// One CTA per SM is one of the reference's workers (a "CTA group") with its
// own contiguous slice of the probe input and its own share of the budget
// (bep_budget_mib / groups).  Probe rows live in fixed-size blocks of `page`
// rows (column-major inside a block) taken from one device pool through a
// free-block stack.
//
// The run alternates between two steps, S and E, until the input is through:
//   S  k_bep_scatter, a cooperative launch of the groups.  In waves separated
//      by grid-wide barriers, each group scatters the next tile of its slice
//      by the first radix pass into its private pass-1 bucket chains (the
//      reference's per-worker `unrefined` chains) and adds the tile's bytes
//      to its unrefined count.  At the per-group high water (half the
//      group's budget) it refines its largest bucket, again and again until
//      the count is below the low water (a quarter): refining a bucket
//      counts its rows by leaf (leaf_rows, the global leaf count) and
//      publishes its blocks as refined blocks of that bucket.  (The rows
//      are not moved: a leaf's rows are found in its bucket's blocks by
//      their hash when the leaf is evicted.)
//      (src/PHJBep.cpp:397-450 refinePartition, :508-528 evictAsNeeded
//      phase 1, :582-605 the main loop.)  When the global leaf bytes reach
//      the leaf high water (5/8 of the budget), or the input is through and
//      every group has refined what it held (:662-676), the launch ends; the
//      groups' state stays in memory.
//   E  the round-robin eviction cursor (next_evict_leaf) advances over the
//      leaves until the leaves it passed hold enough rows to take the global
//      count below the low water (5/8 of the high water; every leaf in the
//      final drain): k_bep_range.  Each leaf passed is claimed with a CAS on
//      its lock word and counted as an eviction when it held rows
//      (k_bep_claim); the claimed leaves whose table is NOT_BUILT are built
//      (k_bep_build of bep.cu: NOT_BUILT -> BUILDING by CAS, BUILT when
//      done; a leaf found BUILDING is waited for, bounded); then every
//      refined block's rows of the claimed leaves are probed and projected
//      (k_bep_probe), the blocks in bucket order so one bucket's leaf tables
//      stay in L2; a block whose rows are all probed goes back to the pool.
//      (src/PHJBep.cpp:453-505 tryEvictOneLeaf, :530-571 phase 2; the
//      post-probe drain, :689-727.)
// The host enqueues S and E in turn, one pair and then more at a time, and
// reads the control block between; steps past the end find nothing to do.
// The reference's cooperative end-of-slice drain (:619-655) has no separate
// form: the slices are equal and every group takes part in every E, so no
// group idles while another scatters.
//
// Counters as the reference defines them (src/PHJBep.h:13-39): evictions
// (leaves that held rows when claimed), refinements (bucket refines), peak
// (the largest global leaf bytes, seen after each wave's refines), skip
// retries (claims that found the leaf locked, and waits on a BUILDING leaf).
//
// Every wait is bounded: the grid barrier, the bulk copies and the BUILDING
// wait give up after the context's wait limit (the copies after a poll
// limit), set an error code and end the run.  A group that finds too few
// free blocks for its tile refines what it holds and the wave ends in a
// drain of every leaf (which frees every refined block); a second shortage
// right after such a drain ends the run with a capacity error.  Each group
// takes its free blocks from a cache of its own, refilled from the pool's
// stack a batch at a time.
//
// Measured (64M x 512M rows, Zipf keys, 32 MiB a group): 14.4 ms (S 5.7,
// claims and builds 1.4, probes 6.5 ms); one persistent grid of 1024-thread
// CTAs for both steps, whose refines sorted every block by leaf, took 28.1 ms
// (S 11.6, claims and builds 3.9, probes 12.3).  8M x 64M rows: 2.60 ms
// (S 1.0, 0.36, 0.87) against 6.06 ms.
#include "internal.h"
#include "list.cuh"

#include <cstdio>
#include <cstdlib>
#include <type_traits>

namespace phjg
{
namespace
{
constexpr int kENT = 1024; // threads of a group's CTA
constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kBuilt = 2, kBuiltDup = 3; // (0 NOT_BUILT, 1 BUILDING)

// error codes written to the context's error word
// (1: a bulk copy, 4: a BUILDING leaf was not there in time)
constexpr int kErrBarrier = 5; // a grid barrier was not reached in time
constexpr int kErrPool = 6;    // the block pool ran out
constexpr int kErrChain = 7;   // a bucket chain outgrew its directory

constexpr uint32_t kETile = 4096;  // most input rows of one scatter step
constexpr uint32_t kRefill = 64;   // free blocks a group takes beyond its need
constexpr uint32_t kPersistScal = 8;

struct EngineCtl
{
    unsigned int bar_count;
    unsigned int bar_gen;
    int abort;
    int evict_now;
    unsigned long long global_leaf_rows;
    unsigned long long peak_leaf_rows;
    unsigned long long cursor;   // next_evict_leaf, counted in leaves (mod n_leaves)
    unsigned long long ev_lo;    // the current E's range of cursor positions [ev_lo, ev_lo + ev_len)
    unsigned long long ev_len;
    unsigned long long out_rows; // output rows placed (the exact total, also past capacity)
    long long free_top;          // blocks on the free stack
    unsigned int work_n;
    unsigned int build_n, build_next;
    unsigned long long work_next;
    unsigned long long evictions, refinements, skip_retries, evict_phases;
    unsigned long long ns_shuffle, ns_evict, ns_probe; // group 0's time in S, E bookkeeping, E probing
    unsigned long long rows_scattered, rows_refined, rows_probed, rows_claimed; // row totals per step (checks)
    unsigned int groups_done; // groups whose slice is scattered
    int ev_mode;              // the E to come: 0 none, 1 down to the low water, 2 every leaf
    int input_done;           // the final drain is the E to come, or is done
    int finished;             // the final drain is claimed: nothing is left to do
    int started;              // an S step has run: the groups' state is in memory
    unsigned long long t_evict0, t_probe0; // start of this E, of its probes (0: none)
    int no_more_input;        // every group's slice is scattered (decided at each wave's barrier)
    unsigned int waves;       // waves so far
    int pool_low;             // a group found too few free blocks for its tile this wave
    int forced_last;          // the previous E was a drain forced by a low pool
    int any_dup;              // some leaf built so far has a repeated key
    unsigned long long forced_drains;
    unsigned long long wave_s_max, ns_s_crit; // the slowest group's S time this wave; summed over waves
    unsigned long long ns_refine0, tiles0, blocks0; // group 0: time refining, tiles scattered, blocks refined
};

static_assert(sizeof(EngineCtl) + 8 <= kSmallReadBytes, "the control block and the error word are read back in one small read");

struct EngineArgs
{
    Cols pin; // probe side in input order
    uint64_t probe_rows;
    Cols bpart; // leaf-partitioned build side (keys and payloads)
    uint32_t * state;
    LeafMeta * meta;
    Cell * cells;
    uint64_t * next;
    const uint32_t * leaf_off;
    int ulog;            // >= 0: uniform tables of 2^ulog cells at leaf << ulog
    uint32_t b1;         // first-pass bits
    uint32_t total_bits; // leaf bits
    uint32_t lb_log2;    // leaf-in-bucket bits (total_bits - b1)
    uint32_t n_leaves, n_buckets;
    // blocks of `page` rows: keys at 0, payload column c at col_off[c]
    uint8_t * pool;
    uint32_t page_log2;
    uint64_t block_bytes;
    uint32_t col_off[kMaxCols];
    uint32_t n_blocks;
    uint32_t * free_stack;
    uint32_t * blk_state; // refined and holding unprobed rows: its bucket; otherwise kNone
    uint32_t * blk_rows;
    uint32_t * blk_rem;
    uint32_t * blk_bucket; // the bucket of a refined block (kept after the block is freed)
    // the eviction cursor when the block was refined: the block's rows of
    // leaf L are probed when the cursor first passes L after that point
    unsigned long long * blk_c0;
    uint32_t * chain; // [group][bucket][maxb] block ids of the unrefined chains
    uint32_t maxb;
    uint32_t * leaf_rows; // unprobed refined rows per leaf
    uint32_t * leaf_lock;
    uint32_t * bucket_cnt;  // E: refined blocks per bucket, then their first work slot
    uint32_t * bucket_fill; // E: work slots taken per bucket
    uint32_t * work;        // E: refined blocks to probe, bucket by bucket
    uint32_t * build_queue; // E: claimed leaves to build
    // budget, bytes (src/PHJBep.cpp:186-190)
    uint64_t unref_high, unref_low, leaf_high, leaf_low;
    uint32_t rb;        // bytes of a probe row
    uint64_t tile_rows; // input rows a group scatters per wave
    uint32_t stage_rows;                 // rows of a scatter step (<= kETile)
    uint32_t stage_off[kMaxCols], stage_bytes; // a step's columns in shared memory (keys at 0)
    int use_tma;                         // the input columns start on 16-byte boundaries
    uint32_t * group_state; // per group: the words of Smem::persist
    uint32_t persist_words, bcache_words, fresh_words, half_bytes;
    // output
    uint64_t * out_keys;
    void * out_l[kMaxCols];
    void * out_r[kMaxCols];
    uint64_t out_cap;
    uint64_t wait_limit_ns;
    uint32_t test_stall_wave; // test hook: group 0 holds back from this wave's barrier (kNone: off)
    EngineCtl * ctl;
    int * err;
};

__device__ __forceinline__ uint64_t now_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint32_t ld_acquire_u32(const unsigned int * p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void fail(const EngineArgs & a, int code)
{
    atomicExch(&a.ctl->abort, code);
    atomicExch(a.err, code);
}

__device__ __forceinline__ bool aborted(const EngineArgs & a)
{
    return *reinterpret_cast<volatile int *>(&a.ctl->abort) != 0;
}

template <class T>
__device__ __forceinline__ T vload(const T * p)
{
    return *reinterpret_cast<const volatile T *>(p);
}

__device__ __forceinline__ uint64_t umin64(uint64_t x, uint64_t y) { return x < y ? x : y; }

// Element src_i of a column (written by an earlier kernel) to
// element dst_i of an output column, with a streaming store.
__device__ __forceinline__ void copy_elem_out(void * dst, uint64_t dst_i, const void * src, uint64_t src_i, uint32_t w)
{
    switch (w)
    {
        case 1: __stcs(static_cast<unsigned char *>(dst) + dst_i, __ldg(static_cast<const unsigned char *>(src) + src_i)); break;
        case 2: __stcs(static_cast<unsigned short *>(dst) + dst_i, __ldg(static_cast<const unsigned short *>(src) + src_i)); break;
        case 4: __stcs(static_cast<unsigned int *>(dst) + dst_i, __ldg(static_cast<const unsigned int *>(src) + src_i)); break;
        case 8: __stcs(static_cast<unsigned long long *>(dst) + dst_i, __ldg(static_cast<const unsigned long long *>(src) + src_i)); break;
        default: __stcs(static_cast<uint4 *>(dst) + dst_i, __ldg(static_cast<const uint4 *>(src) + src_i)); break;
    }
}

// Grid-wide barrier (every group is resident: cooperative launch).  The
// last group to arrive runs `last` before it releases the others.  A wait
// longer than the context's limit ends the grid with kErrBarrier.  Returns
// false when the grid is ending.
template <class F>
__device__ bool grid_sync(const EngineArgs & a, uint32_t & gen, F last)
{
    __syncthreads();
    if (threadIdx.x == 0)
    {
        const uint32_t target = gen + 1;
        __threadfence();
        const uint32_t arrived = atomicAdd(&a.ctl->bar_count, 1u);
        if (arrived == gridDim.x - 1)
        {
            a.ctl->bar_count = 0;
            last();
            __threadfence();
            atomicExch(&a.ctl->bar_gen, target);
        }
        else
        {
            const uint64_t t0 = now_ns();
            uint32_t spins = 0;
            while (ld_acquire_u32(&a.ctl->bar_gen) != target)
            {
                if (aborted(a))
                    break;
                if ((++spins & 255u) == 0 && now_ns() - t0 > a.wait_limit_ns)
                {
                    fail(a, kErrBarrier);
                    break;
                }
                __nanosleep(64);
            }
        }
        gen = target;
        __threadfence();
    }
    __syncthreads();
    return !aborted(a);
}

// Block-wide exclusive scan over `n` u32 bins in shared memory (in place);
// returns the total.  `ws` holds kENT/32 words.
__device__ uint32_t scan_bins(uint32_t * bins, uint32_t n, uint32_t * ws)
{
    const uint32_t per = (n + kENT - 1) / kENT;
    const uint32_t b0 = threadIdx.x * per;
    uint32_t sum = 0;
    for (uint32_t i = 0; i < per; ++i)
        if (b0 + i < n)
            sum += bins[b0 + i];
    uint32_t total;
    const uint32_t excl = block_excl_scan<kENT>(sum, ws, &total);
    uint32_t run = excl;
    for (uint32_t i = 0; i < per; ++i)
        if (b0 + i < n)
        {
            const uint32_t v = bins[b0 + i];
            bins[b0 + i] = run;
            run += v;
        }
    __syncthreads();
    return total;
}

__device__ __forceinline__ uint8_t * block_ptr(const EngineArgs & a, uint32_t blk)
{
    return a.pool + (uint64_t)blk * a.block_bytes;
}

// An S CTA scatters in two halves of 512 threads, a step each at a time.
constexpr int kHNT = kENT / 2;
constexpr int kHRows = (int)kETile / kHNT; // rows a thread of a step

// One half's shared memory.
struct Half
{
    uint8_t * stage;  // a step's rows, column-major
    uint32_t * perm;  // a step's rows in bucket order: row | bucket << 12
    uint32_t * bins;  // buckets: rows of the step
    uint32_t * off;   // buckets: first position in the step's bucket order (and the total)
    uint32_t * nb0;   // buckets: first of the step's new blocks (and the total)
    uint2 * fl;       // buckets: {rows in the chain's last block before the step - off, that block}
    uint32_t * fresh; // the step's new blocks
    uint32_t * wsum;  // the warps' sums of a scan
    uint32_t * scal;  // [0] the step's outcome, [1,2] where its new blocks come from
};

// Shared memory of an S CTA.
struct Smem
{
    Half hf;          // this thread's half's
    uint32_t * acc;   // leaves per bucket: rows a refine adds to each leaf
    uint32_t * scal;  // scalars (32 words, 8-byte aligned)
    uint32_t * list;  // buckets: refine_down_to's lists (half 0's `off`, between steps)
    // kept in memory between launches, one run of words:
    uint32_t * persist;
    uint32_t * fill;   // buckets: rows in each chain's last block (page: no block)
    uint32_t * clen;   // buckets: blocks in each chain
    uint32_t * urows;  // buckets: unrefined rows per bucket
    uint32_t * last;   // buckets: each chain's last block
    uint32_t * bcache; // the group's free blocks
    uint32_t * pscal;  // [0] blocks in bcache, [1] counted in groups_done, [2,3] next input row, [4,5] unrefined bytes
};

// Barriers of one half (hardware barrier 1 + half).
__device__ __forceinline__ void half_sync(uint32_t half)
{
    asm volatile("barrier.sync %0, %1;" ::"r"(1u + half), "n"(kHNT) : "memory");
}
__device__ __forceinline__ bool half_sync_and(uint32_t half, bool v)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %3, 0;\n\t"
        "barrier.red.and.pred q, %1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"(1u + half), "n"(kHNT), "r"((uint32_t)v)
        : "memory");
    return r != 0;
}

// ---------------------------------------------------------------------------
// S: one scatter step -- the `n` rows in a half's stage into the group's
// chains.
// ---------------------------------------------------------------------------
enum : uint32_t
{
    kTileDone = 0,
    kTileNoRoom = 1,
    kTileFailed = 2
};
// words of Smem::scal that order the halves' steps: the step whose turn it is
// to allocate, the outcome of the first step that was not taken, and which
constexpr uint32_t kTurn = 8, kStop = 9, kStopStep = 10;
constexpr uint32_t kRefineSlot = 16; // refine_down_to's words

template <class T>
__device__ __forceinline__ void block_column(const EngineArgs & a, const uint8_t * src_v, uint32_t col_off, const uint32_t (&row)[4],
                                             const uint32_t (&blk)[4], const uint32_t (&slot)[4], uint32_t live)
{
    const T * src = reinterpret_cast<const T *>(src_v);
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (live >> j & 1u)
            reinterpret_cast<T *>(block_ptr(a, blk[j]) + col_off)[slot[j]] = src[row[j]];
}

// Takes `lack` blocks and up to kRefill beyond from the pool's stack: the
// first of them in *from, their number returned (0: too few free blocks).
__device__ __forceinline__ uint32_t take_blocks(const EngineArgs & a, uint32_t lack, uint32_t * from)
{
    const uint32_t want = lack + kRefill;
    unsigned long long * top = reinterpret_cast<unsigned long long *>(&a.ctl->free_top);
    long long cur = (long long)vload(top), t;
    for (;;)
    {
        t = cur >= (long long)want ? (long long)want : (cur >= (long long)lack ? cur : 0);
        if (t == 0)
            break;
        const long long seen = (long long)atomicCAS(top, (unsigned long long)cur, (unsigned long long)(cur - t));
        if (seen == cur)
            break;
        cur = seen;
    }
    *from = (uint32_t)(cur - t);
    return (uint32_t)t;
}

// Bucket p's share of a step: c rows and nb new blocks, of them bcache[first,
// +nb); its rows start at `row` of the step's bucket order, its new blocks at
// `rb` of hf.fresh.  False: the chain outgrew its directory.
__device__ __forceinline__ bool place_bucket(const EngineArgs & a, const Smem & sm, uint32_t g, uint32_t p, uint32_t c, uint32_t nb, uint32_t row,
                                             uint32_t rb, uint32_t first)
{
    const Half & hf = sm.hf;
    const uint32_t fill = sm.fill[p], last = sm.last[p];
    hf.off[p] = row;
    hf.nb0[p] = rb;
    hf.fl[p] = make_uint2(fill - row, last);
    if (c == 0)
        return true;
    hf.bins[p] = 0;
    const uint32_t len = sm.clen[p];
    if (len + nb > a.maxb)
        return false;
    uint32_t blk = last;
    for (uint32_t i = 0; i < nb; ++i)
    {
        blk = sm.bcache[first + i];
        a.chain[((uint64_t)g * a.n_buckets + p) * a.maxb + len + i] = blk;
        hf.fresh[rb + i] = blk;
    }
    sm.last[p] = blk;
    sm.fill[p] = ((fill + c - 1) & ((1u << a.page_log2) - 1)) + 1;
    sm.clen[p] = len + nb;
    sm.urows[p] += c;
    return true;
}

// A step's places for few buckets (at most 32 * kLanePer), by one warp, the
// others of its half at a barrier: two barriers of 512 threads fewer (64
// buckets: 4,500 cycles of a step's 20,000 were spent here by the general form;
// S 5.9 -> 5.7 ms for 512M rows; with 256 buckets a warp alone takes longer:
// 2M x 10M rows 2,310 us against 2,214).
constexpr uint32_t kLanePer = 4;
__device__ __forceinline__ uint32_t allocate_few(const EngineArgs & a, const Smem & sm, uint32_t g, uint32_t n)
{
    const Half & hf = sm.hf;
    const uint32_t page = 1u << a.page_log2, P1 = a.n_buckets, lane = threadIdx.x & 31;
    uint32_t cnt[kLanePer], at[kLanePer], run = 0; // bucket j * 32 + lane
#pragma unroll
    for (uint32_t j = 0; j < kLanePer; ++j)
    {
        const uint32_t p = j * 32 + lane;
        cnt[j] = 0;
        if (p < P1)
        {
            const uint32_t c = hf.bins[p];
            if (c)
                cnt[j] = c | (((sm.fill[p] + c + page - 1) >> a.page_log2) - 1u) << 16;
        }
    }
#pragma unroll
    for (uint32_t j = 0; j < kLanePer; ++j)
    {
        uint32_t incl = cnt[j];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o)
                incl += y;
        }
        at[j] = run + incl - cnt[j];
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    const uint32_t need = run >> 16;
    uint32_t have = sm.pscal[0];
    if (need > have)
    {
        uint32_t from = 0, got = 0;
        if (lane == 0)
            got = take_blocks(a, need - have, &from);
        got = __shfl_sync(0xffffffffu, got, 0);
        from = __shfl_sync(0xffffffffu, from, 0);
        if (got == 0)
            return kTileNoRoom;
        for (uint32_t i = lane; i < got; i += 32)
            sm.bcache[have + i] = __ldcg(a.free_stack + from + i);
        have += got;
        __syncwarp();
    }
    bool ok = true;
#pragma unroll
    for (uint32_t j = 0; j < kLanePer; ++j)
        if (j * 32 + lane < P1)
            ok = place_bucket(a, sm, g, j * 32 + lane, cnt[j] & 0xFFFFu, cnt[j] >> 16, at[j] & 0xFFFFu, at[j] >> 16, have - need + (at[j] >> 16)) && ok;
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0)
    {
        if (!ok)
            fail(a, kErrChain);
        hf.off[P1] = n;
        hf.nb0[P1] = need;
        sm.pscal[0] = have - need;
    }
    return ok ? kTileDone : kTileFailed;
}

// The step's places, by its half: the bucket counts scanned, the blocks its
// chains need (an empty chain counts as a full last block) taken from the
// group's cache of free blocks, and the chains brought to their state after
// the step.  A half runs this in its turn, so steps allocate in input order.
// hf.bins is zero on a kTileDone return.
__device__ __forceinline__ uint32_t allocate_step(const EngineArgs & a, const Smem & sm, uint32_t half, uint32_t g, uint32_t n)
{
    const Half & hf = sm.hf;
    const uint32_t page = 1u << a.page_log2, P1 = a.n_buckets;
    const uint32_t tid = threadIdx.x & (kHNT - 1), lane = tid & 31, warp = tid >> 5;
    const uint32_t per = (P1 + kHNT - 1) / kHNT, p0 = tid * per; // at most kPer
    constexpr uint32_t kPer = 2048 / kHNT;
    // rows (low half: at most 4096) and new blocks (at most 4096 + 2048)
    uint32_t cnt[kPer], sum = 0;
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j)
    {
        cnt[j] = 0;
        if (j < per && p0 + j < P1)
        {
            const uint32_t c = hf.bins[p0 + j];
            if (c)
                cnt[j] = c | (((sm.fill[p0 + j] + c + page - 1) >> a.page_log2) - 1u) << 16;
            sum += cnt[j];
        }
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o)
            incl += y;
    }
    if (lane == 31)
        hf.wsum[warp] = incl;
    half_sync(half);
    static_assert(kHNT / 32 == 16, "the scan of the warps' sums");
    uint32_t w = hf.wsum[lane & 15];
#pragma unroll
    for (int o = 1; o < 16; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, w, o, 16);
        if ((lane & 15) >= (uint32_t)o)
            w += y;
    }
    const uint32_t need = __shfl_sync(0xffffffffu, w, 15) >> 16;
    const uint32_t before = __shfl_sync(0xffffffffu, w, warp ? warp - 1 : 0);
    uint32_t run = incl - sum + (warp ? before : 0u);
    // the cache is refilled from the pool's stack kRefill blocks beyond the
    // need at a time, so the groups rarely meet on the stack
    uint32_t have = sm.pscal[0];
    if (need > have)
    {
        if (tid == 0)
        {
            uint32_t from;
            const uint32_t t = take_blocks(a, need - have, &from);
            hf.scal[0] = t ? kTileDone : kTileNoRoom;
            hf.scal[1] = from;
            hf.scal[2] = t;
        }
        half_sync(half);
        if (hf.scal[0] != kTileDone)
            return kTileNoRoom;
        const uint32_t from = hf.scal[1], got = hf.scal[2];
        for (uint32_t i = tid; i < got; i += kHNT)
            sm.bcache[have + i] = __ldcg(a.free_stack + from + i);
        have += got;
        half_sync(half);
    }
    const uint32_t base = have - need; // this step's blocks: bcache[base, +need)
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j)
        if (j < per && p0 + j < P1)
        {
            if (!place_bucket(a, sm, g, p0 + j, cnt[j] & 0xFFFFu, cnt[j] >> 16, run & 0xFFFFu, run >> 16, base + (run >> 16)))
            {
                fail(a, kErrChain);
                hf.scal[0] = kTileFailed;
            }
            run += cnt[j];
        }
    if (tid == 0)
    {
        hf.off[P1] = n;
        hf.nb0[P1] = need;
    }
    half_sync(half);
    if (tid == 0)
        sm.pscal[0] = base;
    return hf.scal[0];
}

// One half's step `k` of the launch.  Consecutive rows of a bucket go to
// consecutive rows of its blocks.  A step is a chain of latencies (shared
// atomics, the scan, the permutation, the stores); the other half's step
// fills them: 5.4 us a step of 4096 rows of 12 bytes, against 8.6 us for
// steps of all 1024 threads, whose first warp scanned the buckets alone.
// What bounds it now is the instructions of a row (issue slots 40% busy, DRAM
// 21%, 8 to 9 warps of 32 at a barrier).  The kernel is held to 64 registers,
// which the step, the refines and the arguments share: 182 bytes of spill
// stores and 432 of loads a thread; what they cost has not been measured.  hf.bins is zero on entry and on a kTileDone return.
__device__ uint32_t scatter_step(const EngineArgs & a, const Smem & sm, uint32_t g, uint32_t half, uint32_t k, uint32_t n, bool ok)
{
    const Half & hf = sm.hf;
    const uint32_t page = 1u << a.page_log2, tid = threadIdx.x & (kHNT - 1);
    const uint64_t * keys = reinterpret_cast<const uint64_t *>(hf.stage);
    volatile uint32_t * turn = sm.scal + kTurn;
    volatile uint32_t * stop = sm.scal + kStop;
    uint32_t dr[kHRows]; // bucket | rank << 11
#pragma unroll
    for (int j = 0; j < kHRows; ++j)
    {
        const uint32_t i = j * kHNT + tid;
        dr[j] = kNone;
        if (ok && i < n)
        {
            const uint32_t p = (uint32_t)(int_hash64(keys[i]) >> (64u - a.b1));
            dr[j] = p | atomicAdd(&hf.bins[p], 1u) << 11;
        }
    }
    if (tid == 0)
    {
        // the steps before this one allocate first (bounded: a step that
        // gives up passes the turn on)
        uint32_t spin = 0;
        while (*turn != k && ++spin < kWaitLimit)
        {
        }
        __threadfence_block();
        hf.scal[0] = *turn == k ? *stop : kTileFailed;
    }
    if (!half_sync_and(half, ok) && tid == 0)
        hf.scal[0] = kTileFailed; // a bulk copy was not there in time
    uint32_t state;
    if (a.n_buckets <= 32 * kLanePer)
    {
        if (tid < 32)
        {
            __syncwarp();
            state = hf.scal[0];
            if (state == kTileDone)
                state = allocate_few(a, sm, g, n);
            __syncwarp();
            if (tid == 0)
                hf.scal[0] = state;
        }
        half_sync(half);
        state = hf.scal[0];
    }
    else
    {
        half_sync(half);
        state = hf.scal[0];
        if (state == kTileDone)
            state = allocate_step(a, sm, half, g, n);
    }
    if (tid == 0)
    {
        if (state == kTileFailed)
        {
            if (!aborted(a))
                fail(a, 1);
            *stop = kTileFailed;
        }
        else if (state == kTileNoRoom && *stop == kTileDone)
        {
            *stop = kTileNoRoom;
            sm.scal[kStopStep] = k; // the first step not taken
        }
        __threadfence_block();
        *turn = k + 1;
    }
    if (state != kTileDone)
        return state;
#pragma unroll
    for (int j = 0; j < kHRows; ++j)
        if (dr[j] != kNone)
            hf.perm[hf.off[dr[j] & 2047u] + (dr[j] >> 11)] = (j * kHNT + tid) | (dr[j] & 2047u) << 12;
    half_sync(half);
#pragma unroll 1
    for (uint32_t s0 = 0; s0 < n; s0 += 4 * kHNT)
    {
        uint32_t row[4], blk[4], slot[4], live = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
            const uint32_t s = s0 + j * kHNT + tid;
            row[j] = blk[j] = slot[j] = 0;
            if (s < n)
            {
                const uint32_t e = hf.perm[s], p = e >> 12;
                const uint2 fl = hf.fl[p];
                const uint32_t q = fl.x + s; // slot counted from the chain's last block
                row[j] = e & 4095u;
                blk[j] = q < page ? fl.y : hf.fresh[hf.nb0[p] + (q >> a.page_log2) - 1u];
                slot[j] = q & (page - 1);
                live |= 1u << j;
            }
        }
        block_column<uint64_t>(a, hf.stage, 0, row, blk, slot, live);
        for (uint32_t c = 0; c < a.pin.n; ++c)
            switch (a.pin.width[c])
            {
                case 1: block_column<uint8_t>(a, hf.stage + a.stage_off[c], a.col_off[c], row, blk, slot, live); break;
                case 2: block_column<uint16_t>(a, hf.stage + a.stage_off[c], a.col_off[c], row, blk, slot, live); break;
                case 4: block_column<uint32_t>(a, hf.stage + a.stage_off[c], a.col_off[c], row, blk, slot, live); break;
                case 8: block_column<uint64_t>(a, hf.stage + a.stage_off[c], a.col_off[c], row, blk, slot, live); break;
                default: block_column<uint4>(a, hf.stage + a.stage_off[c], a.col_off[c], row, blk, slot, live); break;
            }
    }
    return kTileDone;
}

// ---------------------------------------------------------------------------
// S: refine bucket p of group g -- its rows counted by leaf, its blocks
// published as refined.  Returns the rows refined.
// ---------------------------------------------------------------------------
__device__ void refine_bucket(const EngineArgs & a, const Smem & sm, uint32_t g, uint32_t p, unsigned long long c0)
{
    const uint32_t page = 1u << a.page_log2;
    const uint32_t LB = 1u << a.lb_log2, shift = 64u - a.total_bits;
    const uint32_t len = sm.clen[p], rows = sm.urows[p], tail = sm.fill[p];
    const uint32_t * ch = a.chain + ((uint64_t)g * a.n_buckets + p) * a.maxb;
    for (uint32_t l = threadIdx.x; l < LB; l += kENT)
        sm.acc[l] = 0;
    __syncthreads();
    // the chain's rows in one run, four loads in flight a thread
    for (uint32_t i0 = 0; i0 < rows; i0 += 4 * kENT)
    {
        uint64_t k[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            const uint32_t i = i0 + u * kENT + threadIdx.x;
            k[u] = 0;
            if (i < rows)
                k[u] = __ldcg(reinterpret_cast<const unsigned long long *>(block_ptr(a, ch[i >> a.page_log2])) + (i & (page - 1)));
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i0 + u * kENT + threadIdx.x < rows)
                atomicAdd(&sm.acc[(uint32_t)(int_hash64(k[u]) >> shift) & (LB - 1u)], 1u);
    }
    for (uint32_t j = threadIdx.x; j < len; j += kENT)
    {
        const uint32_t blk = ch[j], n = j + 1 == len ? tail : page;
        a.blk_rows[blk] = n;
        a.blk_rem[blk] = n;
        a.blk_bucket[blk] = p;
        a.blk_c0[blk] = c0;
        a.blk_state[blk] = p;
    }
    __syncthreads();
    for (uint32_t l = threadIdx.x; l < LB; l += kENT)
        if (sm.acc[l])
            atomicAdd(a.leaf_rows + ((uint64_t)p << a.lb_log2) + l, sm.acc[l]);
    if (threadIdx.x == 0)
    {
        if (g == 0)
            a.ctl->blocks0 += len;
        sm.clen[p] = 0;
        sm.fill[p] = page;
        sm.urows[p] = 0;
    }
    __syncthreads();
}

// A warp's refine of a bucket of few rows: as refine_bucket, counted without
// shared memory (rows of one leaf in a step of 32 rows together).
__device__ __forceinline__ void refine_small(const EngineArgs & a, const Smem & sm, uint32_t g, uint32_t p, unsigned long long c0)
{
    const uint32_t page = 1u << a.page_log2, shift = 64u - a.total_bits, lane = threadIdx.x & 31;
    const uint32_t len = sm.clen[p], rows = sm.urows[p], tail = sm.fill[p];
    const uint32_t * ch = a.chain + ((uint64_t)g * a.n_buckets + p) * a.maxb;
    for (uint32_t i0 = 0; i0 < rows; i0 += 128)
    {
        uint64_t k[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            const uint32_t i = i0 + u * 32 + lane;
            k[u] = 0;
            if (i < rows)
                k[u] = __ldcg(reinterpret_cast<const unsigned long long *>(block_ptr(a, ch[i >> a.page_log2])) + (i & (page - 1)));
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            const bool on = i0 + u * 32 + lane < rows;
            const uint32_t leaf = on ? (uint32_t)(int_hash64(k[u]) >> shift) : kNone;
            const uint32_t same = __match_any_sync(0xffffffffu, leaf);
            if (on && (uint32_t)__ffs(same) - 1u == lane)
                atomicAdd(a.leaf_rows + leaf, (uint32_t)__popc(same));
        }
    }
    for (uint32_t j = lane; j < len; j += 32)
    {
        const uint32_t blk = ch[j], n = j + 1 == len ? tail : page;
        a.blk_rows[blk] = n;
        a.blk_rem[blk] = n;
        a.blk_bucket[blk] = p;
        a.blk_c0[blk] = c0;
        a.blk_state[blk] = p;
    }
    __syncwarp();
    if (lane == 0)
    {
        sm.clen[p] = 0;
        sm.fill[p] = page;
        sm.urows[p] = 0;
    }
}

// Refines the group's largest bucket, of equal ones the first
// (src/PHJBep.cpp:376-395), until its unrefined bytes are below `low` (every
// bucket that holds rows when low is 0).  The buckets so refined are the first
// ones in that order, so they are found at once -- by a binary search of the
// order's last key -- and refined side by side: those of few rows a warp
// each, the others by the whole CTA.  One after the other they took 2 to 5
// us each, most of it barriers and the search for the largest (2M x 10M Zipf
// rows, 256 buckets, 116 MiB, 82,475 refines: a join of 4,370 us against
// 2,260; 8M x 64M rows, 64 buckets, 20,983 refines: 3,150 against 2,920).
constexpr uint32_t kSmallRows = 1024;
__device__ void refine_down_to(const EngineArgs & a, const Smem & sm, uint32_t g, uint64_t & unref_bytes, uint64_t low)
{
    if (unref_bytes == 0 || (low && unref_bytes < low))
        return;
    // order: rows, then the lower bucket
    uint32_t * slot = sm.scal + kRefineSlot; // three sums in turn, the two lists' lengths
    auto key = [&](uint32_t p, uint32_t r) -> uint64_t { return (uint64_t)r << 11 | (2047u - p); };
    constexpr uint32_t kMine = 2048 / kENT;
    uint32_t mine[kMine];
#pragma unroll
    for (uint32_t j = 0; j < kMine; ++j)
        mine[j] = j * kENT + threadIdx.x < a.n_buckets ? sm.urows[j * kENT + threadIdx.x] : 0u;
    uint64_t last = 2048; // refined: keys from this one on
    __syncthreads();      // (the slots are no longer read)
    if (threadIdx.x < 5)
        slot[threadIdx.x] = 0;
    __syncthreads();
    if (low)
    {
        uint64_t none = (unref_bytes / a.rb + 1) << 11; // a key past all
        for (uint32_t it = 0; none - last > 1; ++it)
        {
            const uint64_t mid = last + (none - last) / 2;
            uint32_t sum = 0;
#pragma unroll
            for (uint32_t j = 0; j < kMine; ++j)
                sum += key(j * kENT + threadIdx.x, mine[j]) >= mid ? mine[j] : 0u;
            sum = __reduce_add_sync(0xffffffffu, sum);
            if ((threadIdx.x & 31) == 0 && sum)
                atomicAdd(slot + it % 3, sum);
            if (threadIdx.x == 0)
                slot[(it + 1) % 3] = 0;
            __syncthreads();
            // (a slot is cleared again two steps on, past the next barrier)
            if ((uint64_t)*reinterpret_cast<volatile uint32_t *>(slot + it % 3) * a.rb + low > unref_bytes)
                last = mid;
            else
                none = mid;
        }
    }
    // the lists: small ones from the front, the others from the back
    uint32_t rows = 0;
#pragma unroll
    for (uint32_t j = 0; j < kMine; ++j)
    {
        const uint32_t p = j * kENT + threadIdx.x;
        if (mine[j] && key(p, mine[j]) >= last)
        {
            rows += mine[j];
            if (mine[j] <= kSmallRows)
                sm.list[atomicAdd(slot + 3, 1u)] = p;
            else
                sm.list[a.n_buckets - 1u - atomicAdd(slot + 4, 1u)] = p;
        }
    }
    rows = __reduce_add_sync(0xffffffffu, rows);
    __syncthreads(); // the lists; the sums are no longer read
    if (threadIdx.x == 0)
        slot[0] = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && rows)
        atomicAdd(slot, rows);
    const uint32_t n_small = slot[3], n_large = slot[4];
    const unsigned long long c0 = vload(&a.ctl->cursor); // the cursor stands still outside E
    for (uint32_t i = threadIdx.x >> 5; i < n_small; i += kENT / 32)
        refine_small(a, sm, g, sm.list[i], c0);
    __syncthreads();
    for (uint32_t i = 0; i < n_large; ++i)
        refine_bucket(a, sm, g, sm.list[a.n_buckets - 1u - i], c0);
    const uint32_t total = slot[0];
    if (threadIdx.x == 0)
    {
        atomicAdd(&a.ctl->global_leaf_rows, (unsigned long long)total);
        atomicAdd(&a.ctl->rows_refined, (unsigned long long)total);
        atomicAdd(&a.ctl->refinements, (unsigned long long)(n_small + n_large));
    }
    const uint64_t bytes = (uint64_t)total * a.rb;
    unref_bytes = unref_bytes > bytes ? unref_bytes - bytes : 0;
}

// ---------------------------------------------------------------------------
// E: the eviction range (one CTA).  From the cursor on, leaves are
// taken until the rows they hold take the global leaf bytes below the low
// water (every leaf in the final drain).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kENT) k_bep_range(const __grid_constant__ EngineArgs a)
{
    __shared__ uint32_t ws[kENT / 32];
    __shared__ uint32_t s_hit;
    const int mode = vload(&a.ctl->ev_mode);
    __syncthreads(); // (cleared below)
    if (threadIdx.x == 0)
    {
        a.ctl->ev_mode = 0;
        a.ctl->ev_len = 0;
        a.ctl->work_n = 0;
        a.ctl->work_next = 0;
        a.ctl->build_n = 0;
        a.ctl->build_next = 0;
        a.ctl->t_evict0 = mode ? now_ns() : 0ull;
    }
    if (mode == 0)
        return; // no E: the following kernels find nothing to do
    const bool final_drain = mode == 2;
    const uint64_t n = a.n_leaves;
    const uint64_t lo_abs = vload(&a.ctl->cursor), lo = lo_abs % n;
    const uint64_t g_rows = vload(&a.ctl->global_leaf_rows);
    uint64_t len = n;
    if (!final_drain)
    {
        // rows that may stay: (global - taken) * rb < leaf_low
        const uint64_t keep_max = a.leaf_low ? (a.leaf_low - 1) / a.rb : 0;
        const uint64_t need = g_rows > keep_max ? g_rows - keep_max : 0;
        uint64_t taken = 0;
        len = 0;
        constexpr uint32_t kPer = 8; // leaves a thread sums per step
        for (uint64_t base = 0; base < n && taken < need; base += (uint64_t)kENT * kPer)
        {
            const uint64_t i0 = base + (uint64_t)threadIdx.x * kPer;
            uint32_t v[kPer], mine = 0;
#pragma unroll
            for (uint32_t u = 0; u < kPer; ++u)
            {
                v[u] = i0 + u < n ? __ldcg(a.leaf_rows + (lo + i0 + u) % n) : 0u;
                mine += v[u];
            }
            uint32_t tot;
            const uint32_t ex = block_excl_scan<kENT>(mine, ws, &tot);
            if (threadIdx.x == 0)
                s_hit = kNone;
            __syncthreads();
            // the leaf whose inclusive prefix first reaches `need`
            if (taken + ex < need && taken + ex + mine >= need)
            {
                uint64_t run = taken + ex;
                uint32_t u = 0;
                for (; u < kPer; ++u)
                {
                    run += v[u];
                    if (run >= need)
                        break;
                }
                s_hit = threadIdx.x * kPer + u;
            }
            __syncthreads();
            const uint32_t hit = s_hit;
            __syncthreads();
            if (hit != kNone)
            {
                len = base + hit + 1;
                taken = need;
            }
            else
            {
                taken += tot;
                len = umin64(base + (uint64_t)kENT * kPer, n);
            }
        }
    }
    if (threadIdx.x == 0)
    {
        a.ctl->ev_lo = lo_abs;
        a.ctl->ev_len = len;
        a.ctl->cursor = lo_abs + len;
        a.ctl->evict_phases += 1;
        if (a.ctl->input_done)
            a.ctl->finished = 1; // the post-probe drain
    }
    for (uint32_t p = threadIdx.x; p <= a.n_buckets; p += kENT)
    {
        a.bucket_cnt[p] = 0;
        a.bucket_fill[p] = 0;
    }
}

// Leaf-in-bucket intervals of bucket p inside the eviction range [lo,
// lo + len) (mod n_leaves): up to two, [x0, x1) and [y0, y1).
__device__ __forceinline__ void bucket_intervals(const EngineArgs & a, uint32_t p, uint64_t lo, uint64_t len, uint32_t & x0, uint32_t & x1,
                                                 uint32_t & y0, uint32_t & y1)
{
    const uint64_t n = a.n_leaves, LB = 1ull << a.lb_log2;
    const uint64_t start = (uint64_t)p << a.lb_log2;
    const uint64_t s = (start + n - lo) % n; // the bucket's first leaf, counted from the range's start
    x0 = x1 = y0 = y1 = 0;
    if (s + LB <= n)
    {
        if (len > s)
            x1 = (uint32_t)umin64(LB, len - s);
    }
    else
    {
        // the range starts inside this bucket: leaves [0, w) come last in
        // the range's order, leaves [w, LB) first
        const uint64_t w = n - s;
        if (len > s)
            x1 = (uint32_t)umin64(w, len - s);
        y0 = (uint32_t)w;
        y1 = (uint32_t)umin64(LB, w + len);
    }
}

__device__ __forceinline__ bool bucket_in_range(const EngineArgs & a, uint32_t p, uint64_t lo, uint64_t len)
{
    uint32_t x0, x1, y0, y1;
    bucket_intervals(a, p, lo, len, x0, x1, y0, y1);
    return x1 > x0 || y1 > y0;
}

// The part of this E's range [lo_abs, lo_abs + len) a block refined at
// cursor c0 still has unprobed rows in: a leaf's rows in the block are
// probed the first time the cursor reaches the leaf at or after c0, i.e.
// at positions [c0, c0 + n_leaves); rows of leaves passed since are probed.
__device__ __forceinline__ uint64_t block_len(const EngineArgs & a, unsigned long long c0, uint64_t lo_abs, uint64_t len)
{
    const uint64_t end = c0 + a.n_leaves;
    return end <= lo_abs ? 0 : umin64(len, end - lo_abs);
}

// A lookup in two halves, so that several rows' first loads are in flight
// at once: probe_issue loads the aligned pair of cells the key's probe
// starts at (through L2);
// probe_finish compares, follows the table past the pair when needed, and
// returns the match count (the next-chain's length when some leaf table has
// a repeated key) and the head build row.
__device__ __forceinline__ const Cell * leaf_table(const EngineArgs & a, uint64_t h, uint64_t & cap)
{
    const uint32_t L = (uint32_t)(h >> (64u - a.total_bits));
    if (a.ulog >= 0)
    {
        cap = 1ull << a.ulog;
        return a.cells + ((uint64_t)L << a.ulog);
    }
    const ulonglong2 m = __ldcg(reinterpret_cast<const ulonglong2 *>(a.meta + L));
    cap = ((m.y >> 40) & 0xffu) ? 1ull << ((uint32_t)(m.y >> 32) & 0xffu) : 0ull;
    return a.cells + m.x;
}

__device__ __forceinline__ CellPair probe_issue(const EngineArgs & a, uint64_t h)
{
    uint64_t cap;
    const Cell * tab = leaf_table(a, h, cap);
    if (cap == 0)
    {
        CellPair none;
        none.a = make_ulonglong2(0ull, INVALID_REF);
        none.b = none.a;
        return none;
    }
    return load_pair<true>(tab + probe_start(h, cap));
}

__device__ __forceinline__ uint32_t probe_finish(const EngineArgs & a, uint64_t key, uint64_t h, const CellPair & pr, bool chains, uint32_t & head)
{
    uint64_t r = INVALID_REF;
    if (ref_valid(pr.a.y))
    {
        if (pr.a.x == key)
            r = pr.a.y;
        else if (ref_valid(pr.b.y))
        {
            if (pr.b.x == key)
                r = pr.b.y;
            else
            {
                // past the pair: follow the table
                uint64_t cap;
                const Cell * tab = leaf_table(a, h, cap);
                const uint64_t mask = cap - 1;
                uint64_t pos = (probe_start(h, cap) + 2) & mask;
                for (uint64_t step = 2; step < cap; ++step)
                {
                    const ulonglong2 c = __ldcg(reinterpret_cast<const ulonglong2 *>(tab + pos));
                    if (!ref_valid(c.y))
                        break;
                    if (c.x == key)
                    {
                        r = c.y;
                        break;
                    }
                    pos = (pos + 1) & mask;
                }
            }
        }
    }
    if (!ref_valid(r))
        return 0;
    head = ref_row(r);
    if (!chains)
        return 1;
    uint32_t c = 1;
    for (unsigned long long x = __ldcg(reinterpret_cast<const unsigned long long *>(a.next) + head); ref_valid(x);
         x = __ldcg(reinterpret_cast<const unsigned long long *>(a.next) + ref_row(x)))
        ++c;
    return c;
}

// Every claim of this E's range: the leaf's rows leave the global count, a
// leaf that held rows is an eviction, and one whose table is not built is
// queued; the refined blocks to probe are counted per bucket.
__global__ void __launch_bounds__(512) k_bep_claim(const __grid_constant__ EngineArgs a)
{
    const uint64_t lo_abs = vload(&a.ctl->ev_lo), len = vload(&a.ctl->ev_len);
    if (len == 0)
        return;
    const uint64_t n = a.n_leaves, lo = lo_abs % n;
    const uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    unsigned long long rows = 0, ev = 0, skips = 0;
    for (uint64_t i = i0; i < len; i += stride)
    {
        const uint32_t L = (uint32_t)((lo + i) % n);
        if (atomicCAS(a.leaf_lock + L, 0u, 1u) != 0u)
        {
            ++skips; // held elsewhere
            continue;
        }
        const uint32_t r = __ldcg(a.leaf_rows + L);
        if (r)
        {
            a.leaf_rows[L] = 0;
            rows += r;
            ++ev;
            const uint32_t st = ld_acquire_u32(a.state + L);
            if (st < kBuilt)
                a.build_queue[atomicAdd(&a.ctl->build_n, 1u)] = L;
            else if (st == kBuiltDup)
                atomicExch(&a.ctl->any_dup, 1); // built by an earlier run over these tables
        }
        atomicExch(a.leaf_lock + L, 0u);
    }
    for (uint64_t b = i0; b < a.n_blocks; b += stride)
    {
        const uint32_t p = a.blk_state[b];
        if (p != kNone && bucket_in_range(a, p, lo, block_len(a, a.blk_c0[b], lo_abs, len)))
            atomicAdd(a.bucket_cnt + p, 1u);
    }
    for (int o = 16; o > 0; o >>= 1)
    {
        rows += __shfl_xor_sync(0xffffffffu, rows, o);
        ev += __shfl_xor_sync(0xffffffffu, ev, o);
        skips += __shfl_xor_sync(0xffffffffu, skips, o);
    }
    if ((threadIdx.x & 31) == 0)
    {
        if (rows)
        {
            atomicAdd(&a.ctl->global_leaf_rows, (unsigned long long)(-(long long)rows));
            atomicAdd(&a.ctl->rows_claimed, rows);
        }
        if (ev)
            atomicAdd(&a.ctl->evictions, ev);
        if (skips)
            atomicAdd(&a.ctl->skip_retries, skips);
    }
}

// Block counts per bucket into work offsets, the buckets in the range's
// order (one CTA).
__global__ void __launch_bounds__(kENT) k_bep_offsets(const __grid_constant__ EngineArgs a)
{
    __shared__ uint32_t bins[1u << 11];
    __shared__ uint32_t ws[kENT / 32];
    if (vload(&a.ctl->ev_len) == 0)
        return;
    const uint32_t P1 = a.n_buckets, first = (uint32_t)((vload(&a.ctl->ev_lo) % a.n_leaves) >> a.lb_log2);
    for (uint32_t q = threadIdx.x; q < P1; q += kENT)
        bins[q] = a.bucket_cnt[(first + q) % P1];
    __syncthreads();
    const uint32_t total = scan_bins(bins, P1, ws);
    for (uint32_t q = threadIdx.x; q < P1; q += kENT)
        a.bucket_cnt[(first + q) % P1] = bins[q];
    if (threadIdx.x == 0)
        a.ctl->work_n = total;
}

// The refined blocks of the range's buckets into the work list.
__global__ void __launch_bounds__(512) k_bep_list(const __grid_constant__ EngineArgs a)
{
    const uint64_t lo_abs = vload(&a.ctl->ev_lo), len = vload(&a.ctl->ev_len);
    if (blockIdx.x == 0 && threadIdx.x == 0)
    {
        const unsigned long long t = now_ns(), t0 = a.ctl->t_evict0;
        if (t0)
            a.ctl->ns_evict += t - t0;
        a.ctl->t_probe0 = t0 ? t : 0ull;
    }
    if (len == 0)
        return;
    const uint64_t lo = lo_abs % a.n_leaves, stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < a.n_blocks; b += stride)
    {
        const uint32_t p = a.blk_state[b];
        if (p != kNone && bucket_in_range(a, p, lo, block_len(a, a.blk_c0[b], lo_abs, len)))
            a.work[a.bucket_cnt[p] + atomicAdd(a.bucket_fill + p, 1u)] = (uint32_t)b;
    }
}

// Work items of the probe kernels: a part of at most 256 rows of a listed
// block, in list order (bucket by bucket), so the warps in flight cover
// little more than one bucket and its leaf tables and build rows stay in L2.
constexpr uint32_t kPartRows = 256;
struct PartItem
{
    uint32_t blk, first, rows; // rows [first, first + rows) of the block
    uint32_t x0, x1, y0, y1;   // the range's leaves of its bucket
    bool whole;                // ... are all of them
};

__device__ __forceinline__ bool part_item(const EngineArgs & a, uint64_t w, uint64_t n_blocks_listed, uint64_t lo_abs, uint64_t len, PartItem & it)
{
    const uint32_t page = 1u << a.page_log2, part_rows = page < kPartRows ? page : kPartRows, parts = page / part_rows;
    if (w >= n_blocks_listed * parts)
        return false;
    it.blk = a.work[w / parts];
    it.first = (uint32_t)(w % parts) * part_rows;
    const uint32_t nrows = a.blk_rows[it.blk];
    it.rows = it.first < nrows ? min(part_rows, nrows - it.first) : 0u;
    const uint32_t p = a.blk_bucket[it.blk];
    bucket_intervals(a, p, lo_abs % a.n_leaves, block_len(a, a.blk_c0[it.blk], lo_abs, len), it.x0, it.x1, it.y0, it.y1);
    it.whole = it.x0 == 0 && it.x1 == (1u << a.lb_log2);
    return true;
}

__device__ __forceinline__ bool leaf_in(const PartItem & it, uint32_t l)
{
    return it.whole || l - it.x0 < it.x1 - it.x0 || l - it.y0 < it.y1 - it.y0;
}

// `done` of the block's rows are probed; a block whose rows all are goes
// back to the pool.
__device__ __forceinline__ void rows_done(const EngineArgs & a, uint32_t blk, uint32_t done)
{
    if (done && atomicSub(a.blk_rem + blk, done) == done)
    {
        a.blk_state[blk] = kNone;
        const long long slot = (long long)atomicAdd(reinterpret_cast<unsigned long long *>(&a.ctl->free_top), 1ull);
        a.free_stack[slot] = blk;
    }
}

// E's probes when no key repeats and the build payloads are gathered in one
// piece (kGather 16: packed rows; 4 or 8: the one column; 0: none): per part
// the lookups, one reservation of its output rows, then its matches 128 at a
// time, as k_probe_inline (probe.cu) writes them, the build rows gathered to
// shared memory meanwhile.  Bound as k_probe_fused by the request path from
// L1 to the crossbar: a cell pair and a build row a probe row.  Measured:
// 6.7 ms for the 512M rows against 64M build rows and 0.88 ms for 64M rows
// against 8M, where the chain-following warps of the persistent grid took
// 12.3 and 1.9 ms.
constexpr int kBPNT = 256;
constexpr uint32_t kBKeys = 0, kBRow = 2048, kBStage = 3072, kBQueue = 5120, kBList = 5632, kBWarpBytes = 5888;
template <int kGather, bool kUniform>
__global__ void __launch_bounds__(kBPNT, 3) k_bep_probe(const __grid_constant__ EngineArgs a, const void * __restrict__ gathered,
                                                        const __grid_constant__ PackSpec pk)
{
    __shared__ __align__(16) uint8_t bsm[kBPNT / 32 * kBWarpBytes];
    if (vload(a.err))
        return; // a leaf's build gave up: its table cannot be read
    if (vload(&a.ctl->any_dup))
        return; // chains have to be followed: k_bep_probe_chains
    const uint32_t lane = threadIdx.x & 31;
    uint8_t * wsm = bsm + (threadIdx.x >> 5) * kBWarpBytes;
    uint64_t * key_s = reinterpret_cast<uint64_t *>(wsm + kBKeys);
    uint32_t * brow_s = reinterpret_cast<uint32_t *>(wsm + kBRow);
    uint4 * stage = reinterpret_cast<uint4 *>(wsm + kBStage);
    uint16_t * qrow = reinterpret_cast<uint16_t *>(wsm + kBQueue);
    uint8_t * list = wsm + kBList;
    const uint64_t lo_abs = vload(&a.ctl->ev_lo), len = vload(&a.ctl->ev_len);
    const uint64_t listed = len ? vload(&a.ctl->work_n) : 0u;
    const uint32_t shift = 64u - a.total_bits, lmask = (1u << a.lb_log2) - 1u;
    const uint64_t ucap = kUniform ? 1ull << a.ulog : 0ull;
    unsigned long long probed = 0;
    for (;;)
    {
        unsigned long long w = 0;
        if (lane == 0)
            w = atomicAdd(&a.ctl->work_next, 1ull);
        w = __shfl_sync(0xffffffffu, w, 0);
        PartItem it;
        if (!part_item(a, w, listed, lo_abs, len, it))
            break;
        const uint8_t * B = block_ptr(a, it.blk);
        const uint64_t * keys = reinterpret_cast<const uint64_t *>(B) + it.first;
#pragma unroll
        for (int k = 0; k < (int)kPartRows / 32; ++k)
            if ((uint32_t)k * 32 + lane < it.rows)
                cp_async_small<8>(key_s + k * 32 + lane, keys + k * 32 + lane);
        cp_async_wait_all();
        uint32_t qn = 0, done = 0;
#pragma unroll 1
        for (uint32_t g = 0; g < it.rows; g += 128)
        {
            uint64_t key[4];
            CellPair cell[4];
            uint32_t live = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u)
            {
                const uint32_t i = g + u * 32 + lane;
                key[u] = 0;
                cell[u].a = make_ulonglong2(0ull, INVALID_REF);
                cell[u].b = cell[u].a;
                if (i < it.rows)
                {
                    key[u] = ld_shared_u64(key_s + i);
                    const uint64_t h = int_hash64(key[u]);
                    const uint32_t L = (uint32_t)(h >> shift);
                    if (leaf_in(it, L & lmask))
                    {
                        live |= 1u << u;
                        if (kUniform)
                            cell[u] = load_pair<false>(a.cells + ((uint64_t)L << a.ulog) + probe_start(h, ucap));
                        else
                        {
                            const ulonglong2 m = __ldg(reinterpret_cast<const ulonglong2 *>(a.meta + L));
                            if ((m.y >> 40) & 0xffu)
                                cell[u] = load_pair<false>(a.cells + m.x + probe_start(h, 1ull << ((uint32_t)(m.y >> 32) & 0xffu)));
                        }
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
            {
                const uint32_t i = g + u * 32 + lane;
                uint64_t head = INVALID_REF;
                bool more = false;
                if ((live >> u & 1u) && ref_valid(cell[u].a.y))
                {
                    if (cell[u].a.x == key[u])
                        head = cell[u].a.y;
                    else if (ref_valid(cell[u].b.y))
                    {
                        if (cell[u].b.x == key[u])
                            head = cell[u].b.y;
                        else
                            more = true;
                    }
                }
                const uint32_t m = __ballot_sync(0xffffffffu, more);
                if (more)
                    qrow[qn + __popc(m & ((1u << lane) - 1u))] = (uint16_t)i;
                qn += __popc(m);
                done += __popc(__ballot_sync(0xffffffffu, live >> u & 1u));
                brow_s[i] = ref_valid(head) ? ref_row(head) : kNone;
            }
        }
        __syncwarp();
        for (uint32_t j = lane; j < qn; j += 32)
        {
            const uint32_t i = qrow[j];
            const uint64_t qk = key_s[i], h = int_hash64(qk);
            const Cell * tab;
            uint64_t cap = ucap;
            if (kUniform)
                tab = a.cells + ((h >> shift) << a.ulog);
            else
                tab = leaf_table(a, h, cap);
            uint64_t pos = (probe_start(h, cap) + 2) & (cap - 1);
            for (uint64_t step = 2; step < cap; step += 2)
            {
                const CellPair c = load_pair<false>(tab + pos);
                if (!ref_valid(c.a.y))
                    break;
                if (c.a.x == qk || (ref_valid(c.b.y) && c.b.x == qk))
                {
                    brow_s[i] = ref_row(c.a.x == qk ? c.a.y : c.b.y);
                    break;
                }
                if (!ref_valid(c.b.y))
                    break;
                pos = (pos + 2) & (cap - 1);
            }
        }
        __syncwarp();
        uint32_t total = 0;
#pragma unroll
        for (int k = 0; k < (int)kPartRows / 32; ++k)
        {
            const uint32_t i = (uint32_t)k * 32 + lane;
            const bool hit = i < it.rows && brow_s[i] != kNone;
            const uint32_t m = __ballot_sync(0xffffffffu, hit);
            if (hit)
                list[total + __popc(m & ((1u << lane) - 1u))] = (uint8_t)i;
            total += __popc(m);
        }
        __syncwarp();
        if (total)
        {
            unsigned long long b0 = 0;
            if (lane == 0)
                b0 = atomicAdd(&a.ctl->out_rows, (unsigned long long)total);
            uint64_t base = 0;
#pragma unroll 1
            for (uint32_t j0 = 0; j0 < total; j0 += 128)
            {
                uint32_t idx[4], one = 0;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                {
                    const uint32_t j = j0 + u * 32 + lane;
                    idx[u] = 0;
                    if (j < total)
                    {
                        idx[u] = list[j];
                        one |= 1u << u;
                        if constexpr (kGather == 16)
                            cp_async16(stage + u * 32 + lane, static_cast<const uint4 *>(gathered) + brow_s[idx[u]]);
                        else if constexpr (kGather != 0)
                            cp_async_small<kGather>(stage + u * 32 + lane, static_cast<const uint8_t *>(gathered) + (uint64_t)brow_s[idx[u]] * kGather);
                    }
                }
                uint64_t v[4];
                if (a.pin.n)
                    load_list(v, B + a.col_off[0], a.pin.width[0], it.first, idx, one);
                if (j0 == 0)
                    base = __shfl_sync(0xffffffffu, b0, 0);
                const uint64_t out = base + j0 + lane;
#pragma unroll
                for (int u = 0; u < 4; ++u)
                {
                    if (out + 32 * u >= a.out_cap)
                        one &= ~(1u << u);
                    if (one >> u & 1u)
                        __stcs(a.out_keys + out + 32 * u, key_s[idx[u]]);
                }
#pragma unroll 1
                for (uint32_t c = 0; c < a.pin.n; ++c)
                {
                    uint64_t nx[4];
                    if (c + 1 < a.pin.n)
                        load_list(nx, B + a.col_off[c + 1], a.pin.width[c + 1], it.first, idx, one);
                    store_list(v, a.out_r[c], a.pin.width[c], out, one);
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        v[u] = nx[u];
                }
                if constexpr (kGather != 0)
                {
                    cp_async_wait_all();
#pragma unroll 1
                    for (uint32_t c = 0; c < a.bpart.n; ++c)
                    {
                        uint64_t x[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            x[u] = reinterpret_cast<const uint64_t *>(stage + u * 32 + lane)[pk.off[c] >> 3] >> ((pk.off[c] & 7u) * 8u);
                        store_list(x, a.out_l[c], a.bpart.width[c], out, one);
                    }
                }
                __syncwarp(); // the stage is refilled by the next batch
            }
        }
        if (lane == 0)
            rows_done(a, it.blk, done);
        probed += done;
        __syncwarp(); // the warp's shared memory is filled again by the next part
    }
    if (lane == 0 && probed)
        atomicAdd(&a.ctl->rows_probed, probed);
}

// E's probes in every other case: chains are followed, columns of any width
// are copied row by row.  (64 registers, 180 and 176 bytes spilled; k_bep_probe
// spills 60 and 80 against tables of unequal size, 8 and 8 of one.)  `only_dup`: k_bep_probe has done the work unless a
// key repeats.
__global__ void __launch_bounds__(kBPNT, 4) k_bep_probe_chains(const __grid_constant__ EngineArgs a, int only_dup)
{
    const bool chains = vload(&a.ctl->any_dup) != 0; // some leaf table has a repeated key
    if ((only_dup && !chains) || vload(a.err))
        return; // (err: a leaf's build gave up)
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t lo_abs = vload(&a.ctl->ev_lo), len = vload(&a.ctl->ev_len);
    const uint64_t listed = len ? vload(&a.ctl->work_n) : 0u;
    const uint32_t shift = 64u - a.total_bits, lmask = (1u << a.lb_log2) - 1u;
    unsigned long long probed = 0;
    for (;;)
    {
        unsigned long long w = 0;
        if (lane == 0)
            w = atomicAdd(&a.ctl->work_next, 1ull);
        w = __shfl_sync(0xffffffffu, w, 0);
        PartItem it;
        if (!part_item(a, w, listed, lo_abs, len, it))
            break;
        const uint8_t * B = block_ptr(a, it.blk);
        const uint64_t * keys = reinterpret_cast<const uint64_t *>(B) + it.first;
        uint32_t done = 0;
#pragma unroll 1
        for (uint32_t r0 = 0; r0 < it.rows; r0 += 128)
        {
            uint64_t key[4];
            uint32_t head[4], cnt[4], live = 0;
            CellPair pr[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
            {
                const uint32_t i = r0 + u * 32 + lane;
                key[u] = i < it.rows ? keys[i] : 0ull;
                const uint64_t h = int_hash64(key[u]);
                if (i < it.rows && leaf_in(it, (uint32_t)(h >> shift) & lmask))
                {
                    live |= 1u << u;
                    pr[u] = probe_issue(a, h);
                }
            }
            uint32_t rel[4], total = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u)
            {
                head[u] = 0;
                cnt[u] = (live >> u & 1u) ? probe_finish(a, key[u], int_hash64(key[u]), pr[u], chains, head[u]) : 0u;
                done += __popc(__ballot_sync(0xffffffffu, live >> u & 1u));
                uint32_t x = cnt[u];
#pragma unroll
                for (int d = 1; d < 32; d <<= 1)
                {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
                    if (lane >= (uint32_t)d)
                        x += y;
                }
                rel[u] = total + x - cnt[u];
                total += __shfl_sync(0xffffffffu, x, 31);
            }
            if (total == 0)
                continue;
            unsigned long long out0 = 0;
            if (lane == 0)
                out0 = atomicAdd(&a.ctl->out_rows, (unsigned long long)total);
            out0 = __shfl_sync(0xffffffffu, out0, 0);
#pragma unroll
            for (int u = 0; u < 4; ++u)
            {
                uint64_t o = out0 + rel[u];
                uint32_t b = head[u];
                for (uint32_t m = 0; m < cnt[u]; ++m, ++o)
                {
                    if (o < a.out_cap)
                    {
                        __stcs(a.out_keys + o, key[u]);
                        for (uint32_t c = 0; c < a.bpart.n; ++c)
                            copy_elem_out(a.out_l[c], o, a.bpart.col[c], b, a.bpart.width[c]);
                        for (uint32_t c = 0; c < a.pin.n; ++c)
                            copy_elem_out(a.out_r[c], o, B + a.col_off[c], it.first + r0 + u * 32 + lane, a.pin.width[c]);
                    }
                    if (m + 1 < cnt[u])
                        b = ref_row(__ldg(reinterpret_cast<const unsigned long long *>(a.next) + b));
                }
            }
        }
        if (lane == 0)
            rows_done(a, it.blk, done);
        probed += done;
    }
    if (lane == 0 && probed)
        atomicAdd(&a.ctl->rows_probed, probed);
}

// After the last E: its probes' time.
__global__ void k_bep_stamp(EngineCtl * c)
{
    if (c->t_probe0)
        c->ns_probe += now_ns() - c->t_probe0;
    c->t_probe0 = 0;
}

// The last group to arrive after a wave's S: records the peak, decides
// whether an E follows (the leaf high water, or a drain of every leaf when
// a group found too few free blocks) and whether input is left.  A low pool
// right after a forced drain cannot be helped: the run ends.  At the end of
// the input the E is the drain of every leaf.
struct WaveEnd
{
    const EngineArgs * a;
    bool end_of_input;
    __device__ void operator()() const
    {
        EngineCtl * c = a->ctl;
        const unsigned long long r = vload(&c->global_leaf_rows);
        if (r > c->peak_leaf_rows)
            c->peak_leaf_rows = r;
        const bool low = vload(&c->pool_low) != 0;
        if (low && c->forced_last)
        {
            atomicExch(&c->abort, kErrPool);
            atomicExch(a->err, kErrPool);
        }
        c->forced_last = low;
        if (low)
            c->forced_drains += 1;
        c->pool_low = 0;
        c->evict_now = low ? 2 : (r > 0 && r * a->rb >= a->leaf_high ? 1 : 0);
        c->ns_s_crit += c->wave_s_max;
        c->wave_s_max = 0;
        c->waves += 1;
        c->no_more_input = vload(&c->groups_done) >= gridDim.x;
        c->started = 1;
        c->ev_mode = end_of_input ? 2 : c->evict_now;
        if (end_of_input)
            c->input_done = 1;
    }
};

__global__ void __launch_bounds__(kENT, 1) k_bep_scatter(const __grid_constant__ EngineArgs a)
{
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar[2];
    if (vload(&a.ctl->finished) || aborted(a) || vload(a.err))
        return; // nothing is left to do (no group changes these before a barrier of this launch)
    const uint32_t page = 1u << a.page_log2;
    const uint32_t P1 = a.n_buckets, LB = 1u << a.lb_log2;
    const uint32_t g = blockIdx.x, G = gridDim.x;
    const uint32_t half = threadIdx.x / kHNT, tid = threadIdx.x & (kHNT - 1);
    Smem sm;
    {
        uint8_t * p = smem_raw;
        auto take = [&](uint64_t bytes) {
            uint8_t * q = p;
            p += (bytes + 15) & ~15ull;
            return q;
        };
        auto words = [&](uint64_t n) { return reinterpret_cast<uint32_t *>(take(4 * n)); };
        p += half * a.half_bytes;
        sm.hf.stage = take(a.stage_bytes);
        sm.hf.perm = words(a.stage_rows);
        sm.hf.bins = words(P1);
        sm.hf.off = words(P1 + 1);
        sm.hf.nb0 = words(P1 + 1);
        sm.hf.fl = reinterpret_cast<uint2 *>(words(2 * P1));
        sm.hf.fresh = words(a.fresh_words);
        sm.hf.wsum = words(kHNT / 32);
        sm.hf.scal = words(4);
        p = smem_raw + 2 * a.half_bytes;
        sm.list = reinterpret_cast<uint32_t *>(reinterpret_cast<uint8_t *>(sm.hf.off) - (uint64_t)half * a.half_bytes);
        sm.acc = words(LB);
        sm.scal = words(32);
        sm.persist = words(a.persist_words);
        sm.fill = sm.persist;
        sm.clen = sm.fill + P1;
        sm.urows = sm.clen + P1;
        sm.last = sm.urows + P1;
        sm.pscal = sm.last + P1; // (an even number of words before it)
        sm.bcache = sm.pscal + kPersistScal;
    }
    const uint64_t lo = (a.probe_rows * g / G) & ~15ull, hi = g + 1 == G ? a.probe_rows : (a.probe_rows * (g + 1) / G) & ~15ull;
    uint64_t pos = lo, unref_bytes = 0;
    bool counted = false; // this group is counted in groups_done
    uint32_t * kept = a.group_state + (uint64_t)g * a.persist_words;
    const bool resumed = vload(&a.ctl->started) != 0;
    for (uint32_t i = threadIdx.x; i < a.persist_words; i += kENT)
        sm.persist[i] = resumed ? __ldcg(kept + i) : (i < P1 ? page : 0u); // (fill = page: no block yet)
    for (uint32_t p = tid; p < P1; p += kHNT)
        sm.hf.bins[p] = 0;
    if (threadIdx.x == 0)
    {
        sm.scal[kTurn] = 0;
        sm.scal[kStop] = kTileDone;
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_barrier_init();
    }
    __syncthreads();
    if (resumed)
    {
        pos = *reinterpret_cast<const uint64_t *>(sm.pscal + 2);
        unref_bytes = *reinterpret_cast<const uint64_t *>(sm.pscal + 4);
        counted = sm.pscal[1] != 0;
    }
    // (every group reads these before the launch's first barrier lets any
    // group go on)
    uint32_t gen = vload(&a.ctl->bar_gen), wave = (uint32_t)vload(&a.ctl->waves);
    bool more = vload(&a.ctl->no_more_input) == 0;
    unsigned long long t_probe = 0;
    if (g == 0 && threadIdx.x == 0 && a.ctl->t_probe0)
    {
        t_probe = now_ns() - a.ctl->t_probe0; // the E before this launch
        a.ctl->t_probe0 = 0;
        a.ctl->ns_probe += t_probe;
    }

    // Steps of the launch: step k is rows [pos0 + k * stage_rows, ..), the
    // half k & 1's.  A half's next step is copied in once its stage is free.
    const uint64_t pos0 = pos;
    auto step_row = [&](uint32_t k) -> uint64_t { return umin64(hi, pos0 + (uint64_t)k * a.stage_rows); };
    auto step_rows = [&](uint32_t k) -> uint32_t { return (uint32_t)(step_row(k + 1) - step_row(k)); };
    auto tma_ok = [&](uint32_t n) -> bool {
        if (!a.use_tma || n == 0 || ((n * 8u) & 15u))
            return false;
        for (uint32_t c = 0; c < a.pin.n; ++c)
            if ((n * a.pin.width[c]) & 15u)
                return false;
        return true;
    };
    uint32_t parity = 0;     // phase of bar[half] to wait for
    uint32_t mine = half;    // this half's next step
    bool in_flight = false;  // its copies are under way
    uint8_t * stage = sm.hf.stage;
    auto issue = [&] {
        const uint32_t n = step_rows(mine);
        in_flight = tma_ok(n);
        if (!in_flight || tid != 0)
            return;
        const uint64_t r = step_row(mine);
        uint32_t bytes = n * 8u;
        for (uint32_t c = 0; c < a.pin.n; ++c)
            bytes += n * a.pin.width[c];
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(&bar[half], bytes);
        bulk_copy_g2s(stage, a.pin.keys + r, n * 8u, &bar[half]);
        for (uint32_t c = 0; c < a.pin.n; ++c)
            bulk_copy_g2s(stage + a.stage_off[c], static_cast<const uint8_t *>(a.pin.col[c]) + r * a.pin.width[c], n * a.pin.width[c], &bar[half]);
    };
    if (more)
        issue();
    // before the launch ends, the copies in flight have to land
    auto land = [&] {
        if (in_flight)
            (void)mbar_wait(&bar[half], parity, a.err, 1);
        __syncthreads();
    };
    auto keep = [&] {
        if (threadIdx.x == 0)
        {
            sm.pscal[1] = counted ? 1u : 0u;
            *reinterpret_cast<uint64_t *>(sm.pscal + 2) = pos;
            *reinterpret_cast<uint64_t *>(sm.pscal + 4) = unref_bytes;
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < a.persist_words; i += kENT)
            kept[i] = sm.persist[i];
    };
    const uint32_t wave_steps = (uint32_t)(a.tile_rows / a.stage_rows);
    for (uint32_t k_end = wave_steps; more; ++wave, k_end += wave_steps)
    {
        // -------- S: this wave's tile of the slice, then the refine trigger --------
        const uint64_t t0 = now_ns();
        const uint64_t end = step_row(k_end);
        while (mine < k_end && step_rows(mine) != 0)
        {
            const uint32_t n = step_rows(mine);
            bool ok = true;
            if (in_flight)
            {
                ok = mbar_wait(&bar[half], parity, a.err, 1);
                if (ok)
                {
                    parity ^= 1u;
                    in_flight = false;
                }
            }
            else
            {
                const uint64_t r = step_row(mine);
                for (uint32_t i = tid; i < n; i += kHNT)
                    reinterpret_cast<uint64_t *>(stage)[i] = a.pin.keys[r + i];
                for (uint32_t c = 0; c < a.pin.n; ++c)
                    for (uint32_t i = tid; i < n; i += kHNT)
                        copy_elem(stage + a.stage_off[c], i, a.pin.col[c], r + i, a.pin.width[c]);
                half_sync(half);
            }
            if (scatter_step(a, sm, g, half, mine, n, ok) != kTileDone)
                break;
            half_sync(half); // the stage is free
            mine += 2;
            issue();
        }
        __syncthreads(); // both halves' steps, and the chains' state
        const uint32_t stop = sm.scal[kStop];
        if (stop == kTileFailed)
        {
            land();
            return;
        }
        // (a step without room ends the wave: the steps from it on were not
        // taken, and wait for the drain this forces after the wave)
        const uint64_t done = stop == kTileDone ? end : step_row(sm.scal[kStopStep]);
        if (threadIdx.x == 0)
        {
            if (stop != kTileDone)
                atomicExch(&a.ctl->pool_low, 1);
            atomicAdd(&a.ctl->rows_scattered, (unsigned long long)(done - pos));
            if (g == 0)
                a.ctl->tiles0 += ceil_div(done - pos, a.stage_rows);
        }
        unref_bytes += (done - pos) * a.rb;
        pos = done;
        if (pos >= hi && !counted)
        {
            counted = true;
            if (threadIdx.x == 0)
                atomicAdd(&a.ctl->groups_done, 1u);
        }
        const uint64_t t_ref = now_ns();
        if (pos < end)
            refine_down_to(a, sm, g, unref_bytes, 0); // stalled: everything it holds goes to the drain
        else if (unref_bytes >= a.unref_high)
            refine_down_to(a, sm, g, unref_bytes, a.unref_low);
        if (threadIdx.x == 0)
        {
            const unsigned long long t = now_ns(), dt = t - t0;
            if (g == 0)
            {
                a.ctl->ns_refine0 += t - t_ref;
                a.ctl->ns_shuffle += dt;
            }
            atomicMax(&a.ctl->wave_s_max, dt);
        }
        if (wave == a.test_stall_wave && g == 0 && threadIdx.x == 0)
        {
            // test hook: this group holds back from the barrier until the
            // others' bounded wait runs out and ends the grid (bounded too)
            const uint64_t ts = now_ns();
            while (!aborted(a) && now_ns() - ts < 4 * a.wait_limit_ns)
                __nanosleep(1000);
        }
        // the last group to arrive records the peak and decides the E
        if (!grid_sync(a, gen, WaveEnd{&a, false}))
        {
            land();
            return;
        }
        const int ev = vload(&a.ctl->evict_now);
        const bool left = vload(&a.ctl->no_more_input) == 0;
        if (ev)
        {
            land();
            keep();
            return;
        }
        if (!left)
            break;
    }
    if (more)
        land();
    // -------- end of the slices: refine every bucket that holds rows; the
    // post-probe drain follows --------
    {
        const uint64_t t0 = now_ns();
        refine_down_to(a, sm, g, unref_bytes, 0);
        if (g == 0 && threadIdx.x == 0)
            a.ctl->ns_shuffle += now_ns() - t0;
    }
    if (!grid_sync(a, gen, WaveEnd{&a, true}))
        return;
    keep();
}

__global__ void k_engine_init(uint32_t * __restrict__ free_stack, uint32_t * __restrict__ blk_state, uint32_t n_blocks, EngineCtl * ctl)
{
    if (blockIdx.x == 0 && threadIdx.x == 0)
        ctl->free_top = (long long)n_blocks; // the stack starts full
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_blocks; i += gridDim.x * blockDim.x)
    {
        free_stack[i] = n_blocks - 1 - i;
        blk_state[i] = kNone;
    }
}
} // namespace

bool bep_engine_supported(uint32_t b1, uint32_t total_bits)
{
    return b1 >= 1 && b1 <= 11 && total_bits >= b1 && total_bits - b1 <= 13;
}

BepEngineResult bep_engine_run(phj_ctx * ctx, Scratch & s, const BepEngineInput & in, phj_output * out)
{
    BepEngineResult res{};
    const uint32_t G = (uint32_t)ctx->num_sms; // one group per SM
    EngineArgs a{};
    a.pin = in.probe;
    a.probe_rows = in.probe_rows;
    a.bpart = in.build;
    a.state = in.lt->state;
    a.meta = in.lt->meta;
    a.cells = in.lt->cells;
    a.next = in.lt->next;
    a.leaf_off = in.leaf_off;
    a.ulog = in.lt->uniform_log2cap;
    a.b1 = in.b1;
    a.total_bits = in.total_bits;
    a.lb_log2 = in.total_bits - in.b1;
    a.n_leaves = 1u << in.total_bits;
    a.n_buckets = 1u << in.b1;
    uint32_t rb = 8;
    for (uint32_t c = 0; c < in.probe.n; ++c)
        rb += in.probe.width[c];
    a.rb = rb;
    // the budget per group and the water marks (src/PHJBep.cpp:180-190)
    const uint64_t budget = in.budget_bytes;
    const uint64_t per_group = budget / G;
    a.unref_high = per_group / 2;
    a.unref_low = a.unref_high / 2;
    a.leaf_high = budget * 5 / 8;
    a.leaf_low = a.leaf_high * 5 / 8;
    const uint64_t P1 = a.n_buckets, LB = 1ull << a.lb_log2;
    const uint64_t high_rows = a.unref_high / rb;
    // block rows: a power of two, 64..8192, about what one bucket of a group
    // gathers before its group refines (so a refined block is mostly full)
    uint32_t page_log2 = 6;
    while (page_log2 < 13 && (2ull << page_log2) <= std::max<uint64_t>(high_rows / P1, 1))
        ++page_log2;
    a.page_log2 = page_log2;
    const uint64_t page = 1ull << page_log2;
    uint64_t off = page * 8;
    for (uint32_t c = 0; c < in.probe.n; ++c)
    {
        a.col_off[c] = (uint32_t)off;
        off += page * in.probe.width[c];
    }
    a.block_bytes = (off + 255) & ~255ull;
    // input rows a group scatters between two looks at the global leaf
    // count: half its unrefined high water, at least 256 and at most 16
    // blocks (4096 to 64K rows), so one wave overshoots the marks by little;
    // in steps of at most 4096 rows, at least two a wave (one for each half
    // of the CTA), both in shared memory beside the rest
    a.tile_rows = std::min<uint64_t>(std::min<uint64_t>(std::max<uint64_t>(page * 16, 4096), 65536), std::max<uint64_t>(256, (high_rows / 2) & ~255ull));
    auto smem_of = [&](uint32_t rows) -> uint64_t {
        auto room = [](uint64_t bytes) { return (bytes + 15) & ~15ull; };
        a.stage_rows = rows;
        uint64_t at = 8ull * rows;
        for (uint32_t c = 0; c < in.probe.n; ++c)
        {
            a.stage_off[c] = (uint32_t)at;
            at += ((uint64_t)rows * in.probe.width[c] + 15) & ~15ull;
        }
        a.stage_bytes = (uint32_t)((at + 127) & ~127ull);
        a.fresh_words = (uint32_t)(rows / page + P1 + 1);
        a.bcache_words = a.fresh_words + 2 * kRefill + 2;
        a.persist_words = (uint32_t)((4 * P1 + kPersistScal + a.bcache_words + 1) & ~1ull);
        a.half_bytes = (uint32_t)(
            a.stage_bytes + room(4ull * rows) + room(4 * P1) + room(8 * P1) + 2 * room(4 * (P1 + 1)) + room(4ull * a.fresh_words) + room(kHNT / 8) + room(16));
        return 2ull * a.half_bytes + room(4 * LB) + room(32 * 4) + room(4ull * a.persist_words);
    };
    size_t smem = 0;
    uint32_t step = 64;
    for (uint32_t rows = 128; rows <= kETile && 2 * rows <= a.tile_rows; rows *= 2)
        if (smem_of(rows) + 1024 <= (size_t)ctx->smem_optin)
            step = rows;
    smem = smem_of(step);
    if (smem + 1024 > (size_t)ctx->smem_optin)
        throw Error(PHJ_ERR_UNSUPPORTED, "PHJ (BEP): the device budget engine's shared memory does not fit this configuration");
    a.tile_rows = a.tile_rows / step * step;
    a.use_tma = (reinterpret_cast<uintptr_t>(in.probe.keys) & 15u) == 0;
    for (uint32_t c = 0; c < in.probe.n; ++c)
        a.use_tma = a.use_tma && (reinterpret_cast<uintptr_t>(in.probe.col[c]) & 15u) == 0;
    const uint64_t slice = ceil_div(std::max<uint64_t>(in.probe_rows, 1), G) + 16; // (slices start on multiples of 16 rows)
    // pool, in blocks: a group's unrefined chains hold at most its high
    // water plus a tile in full blocks and one part block per bucket; the
    // refined blocks hold the leaf rows (up to the leaf high water plus one
    // wave of refines) and one part block per refine still unprobed.  Past
    // the whole probe side (a quarter more for blocks partly probed) no
    // more is needed.  Should the pool still run low, the engine drains
    // every leaf and goes on.
    const uint64_t unref_blocks = G * (ceil_div(high_rows + a.tile_rows, page) + P1 + 1);
    const uint64_t leaf_rows_max = a.leaf_high / rb + G * (high_rows + a.tile_rows);
    const uint64_t by_budget = unref_blocks + ceil_div(leaf_rows_max, page) + 2 * G * P1;
    const uint64_t by_input = ceil_div(in.probe_rows + in.probe_rows / 4, page) + 2 * G * (P1 + 2) + G * ceil_div(a.tile_rows, page);
    const uint64_t n_blocks = std::max<uint64_t>(std::min(by_budget, by_input), 2 * unref_blocks) + (uint64_t)G * (kRefill + 8);
    if (n_blocks >= (1ull << 31))
        throw Error(PHJ_ERR_UNSUPPORTED, "PHJ (BEP): the probe side needs more blocks than the device budget engine indexes");
    a.n_blocks = (uint32_t)n_blocks;
    a.maxb = (uint32_t)(ceil_div(std::min<uint64_t>(high_rows + a.tile_rows + page, slice + page), page) + 2);
    a.pool = s.get<uint8_t>((uint64_t)a.n_blocks * a.block_bytes);
    a.free_stack = s.get<uint32_t>(a.n_blocks);
    a.blk_state = s.get<uint32_t>(a.n_blocks);
    a.blk_rows = s.get<uint32_t>(a.n_blocks);
    a.blk_rem = s.get<uint32_t>(a.n_blocks);
    a.blk_bucket = s.get<uint32_t>(a.n_blocks);
    a.blk_c0 = s.get<unsigned long long>(a.n_blocks);
    a.chain = s.get<uint32_t>((uint64_t)G * P1 * a.maxb);
    a.leaf_rows = s.get<uint32_t>(a.n_leaves);
    a.leaf_lock = s.get<uint32_t>(a.n_leaves);
    a.bucket_cnt = s.get<uint32_t>(P1 + 1);
    a.bucket_fill = s.get<uint32_t>(P1 + 1);
    a.work = s.get<uint32_t>(a.n_blocks);
    a.build_queue = s.get<uint32_t>(a.n_leaves);
    a.out_keys = out->keys;
    for (uint32_t c = 0; c < out->left.n_payloads; ++c)
        a.out_l[c] = out->lcol[c];
    for (uint32_t c = 0; c < out->right.n_payloads; ++c)
        a.out_r[c] = out->rcol[c];
    a.out_cap = out->cap;
    a.wait_limit_ns = (uint64_t)ctx->wait_limit_ms * 1000000ull;
    a.test_stall_wave = ctx->test_engine_stall_wave >= 0 ? (uint32_t)ctx->test_engine_stall_wave : kNone;
    a.group_state = s.get<uint32_t>((uint64_t)G * a.persist_words);
    a.ctl = s.get<EngineCtl>(1);
    a.err = ctx->d_err;
    PHJ_CUDA(cudaMemsetAsync(a.ctl, 0, sizeof(EngineCtl), ctx->stream));
    PHJ_CUDA(cudaMemsetAsync(a.leaf_rows, 0, (size_t)a.n_leaves * 4, ctx->stream));
    PHJ_CUDA(cudaMemsetAsync(a.leaf_lock, 0, (size_t)a.n_leaves * 4, ctx->stream));
    k_engine_init<<<(unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(a.n_blocks, 256), (uint64_t)ctx->num_sms * 8)), 256, 0,
                    ctx->stream>>>(a.free_stack, a.blk_state, a.n_blocks, a.ctl);
    PHJ_LAUNCHED(ctx, "bep_engine_init");
    PHJ_CUDA(cudaFuncSetAttribute(k_bep_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    PHJ_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bep_scatter, kENT, smem));
    if (per_sm < 1)
        throw Error(PHJ_ERR_UNSUPPORTED, "PHJ (BEP): the device budget engine does not fit on an SM");
    if (std::getenv("PHJ_DEBUG"))
        std::fprintf(stderr, "[phj] bep_engine: %u groups, page %llu rows (%llu B), %u blocks (%.2f GB), maxb %u, wave %llu rows in steps of %u, smem %zu\n",
                     G, (unsigned long long)page, (unsigned long long)a.block_bytes, a.n_blocks, a.n_blocks * (double)a.block_bytes / 1e9, a.maxb,
                     (unsigned long long)a.tile_rows, a.stage_rows, smem);
    // the leaf builds (bep.cu), from the claims' queue
    BepLeaves bl{};
    bl.state = a.state;
    bl.leaf_off = a.leaf_off;
    bl.build_keys = a.bpart.keys;
    bl.meta = a.meta;
    bl.cells = a.cells;
    bl.next = a.next;
    bl.leaf_bits = a.total_bits;
    bl.n_leaves = a.n_leaves;
    bl.smem_cells = bep_smem_cells(*in.lt);
    bl.wait_limit_ns = a.wait_limit_ns;
    bl.ctr = s.get<unsigned long long>(4);
    PHJ_CUDA(cudaMemsetAsync(bl.ctr, 0, 4 * sizeof(unsigned long long), ctx->stream));
    bl.queue = a.build_queue;
    bl.queue_len = &a.ctl->build_n; // build_n, build_next
    bl.any_dup = &a.ctl->any_dup;
    // the probes: one gather a build row where the payloads allow it
    ProbeArgs pa{};
    pa.build = in.build;
    pa.build.keys = nullptr;
    pack_build_payloads(ctx, s, pa, in.build_rows);
    PackSpec pk{};
    int gather = -1;
    const void * gathered = nullptr;
    if (pa.packed)
    {
        gather = 16;
        gathered = pa.packed;
        for (uint32_t c = 0; c < in.build.n; ++c)
            pk.off[c] = pa.packed_off[c];
    }
    else if (in.build.n == 0)
        gather = 0;
    else if (in.build.n == 1 && (in.build.width[0] == 4 || in.build.width[0] == 8))
    {
        gather = (int)in.build.width[0];
        gathered = in.build.col[0];
    }
    for (uint32_t c = 0; c < in.probe.n; ++c)
        if (in.probe.width[c] > 8)
            gather = -1;
    void (*probe)(EngineArgs, const void *, PackSpec) = nullptr;
    auto pick = [&](auto uniform) {
        constexpr bool kU = decltype(uniform)::value;
        switch (gather)
        {
            case 16: return k_bep_probe<16, kU>;
            case 8: return k_bep_probe<8, kU>;
            case 4: return k_bep_probe<4, kU>;
            default: return k_bep_probe<0, kU>;
        }
    };
    if (gather >= 0)
        probe = a.ulog >= 0 ? pick(std::true_type{}) : pick(std::false_type{});
    const unsigned sms = (unsigned)ctx->num_sms;
    const unsigned block_grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(std::max<uint64_t>(a.n_blocks, a.n_leaves), 512), sms * 4));
    EngineCtl c{};
    int e = 0;
    int rec = -1;
    {
        KTimer kt(ctx, "bep_engine", in.probe_rows, 0);
        rec = kt.idx;
        unsigned int waves = 0;
        for (uint32_t round = 0;; ++round)
        {
            // S and E in turn; the first E's read-back says whether more
            // than the final drain is to come, then pairs go out in growing
            // numbers (a pair past the end costs its launches)
            const uint32_t pairs = round < 2 ? 1u : std::min<uint32_t>(1u << (round - 1), 8u);
            for (uint32_t k = 0; k < pairs; ++k)
            {
                void * args[] = {&a};
                PHJ_CUDA(cudaLaunchCooperativeKernel((const void *)k_bep_scatter, dim3(G), dim3(kENT), args, smem, ctx->stream));
                PHJ_LAUNCHED(ctx, "bep_scatter");
                k_bep_range<<<1, kENT, 0, ctx->stream>>>(a);
                PHJ_LAUNCHED(ctx, "bep_range");
                k_bep_claim<<<block_grid, 512, 0, ctx->stream>>>(a);
                PHJ_LAUNCHED(ctx, "bep_claim");
                k_bep_offsets<<<1, kENT, 0, ctx->stream>>>(a);
                PHJ_LAUNCHED(ctx, "bep_offsets");
                bep_build_queue(ctx, bl);
                k_bep_list<<<block_grid, 512, 0, ctx->stream>>>(a);
                PHJ_LAUNCHED(ctx, "bep_list");
                if (probe)
                {
                    probe<<<sms * 3, kBPNT, 0, ctx->stream>>>(a, gathered, pk);
                    PHJ_LAUNCHED(ctx, "bep_probe");
                }
                k_bep_probe_chains<<<sms * 4, kBPNT, 0, ctx->stream>>>(a, probe ? 1 : 0);
                PHJ_LAUNCHED(ctx, "bep_probe_chains");
            }
            k_bep_stamp<<<1, 1, 0, ctx->stream>>>(a.ctl);
            PHJ_LAUNCHED(ctx, "bep_stamp");
            read_small(ctx, {{&c, a.ctl, sizeof(c)}, {&e, ctx->d_err, sizeof(e)}});
            if (c.finished || e != 0 || c.abort)
                break;
            if (c.waves == waves)
                throw Error(PHJ_ERR_CUDA, "internal: the device budget engine stands still");
            waves = c.waves;
        }
    }
    unsigned long long built[2] = {0, 0}; // tables built, waits on a BUILDING leaf
    read_small(ctx, {{built, bl.ctr, sizeof(built)}});
    if (e == 0)
        e = c.abort;
    // the launch's algorithmic bytes, as the join's: every probe row read
    // once, every output row written once
    {
        uint64_t orow = 8;
        for (uint32_t c2 = 0; c2 < in.build.n; ++c2)
            orow += in.build.width[c2];
        for (uint32_t c2 = 0; c2 < in.probe.n; ++c2)
            orow += in.probe.width[c2];
        if (rec >= 0)
            ctx->records[rec].bytes = in.probe_rows * rb + std::min<uint64_t>(c.out_rows, a.out_cap) * orow;
    }
    res.err = e;
    res.out_rows = c.out_rows;
    res.evictions = c.evictions;
    res.refinements = c.refinements;
    res.skip_retries = c.skip_retries + built[1];
    res.tables_built = built[0];
    res.evict_phases = c.evict_phases;
    res.peak_bytes = c.peak_leaf_rows * rb;
    res.ms_shuffle = c.ns_shuffle * 1e-6;
    res.ms_evict = c.ns_evict * 1e-6;
    res.ms_probe = c.ns_probe * 1e-6;
    res.pool_bytes = (uint64_t)a.n_blocks * a.block_bytes;
    if (std::getenv("PHJ_DEBUG"))
        std::fprintf(stderr,
                     "[phj] bep_engine rows: scattered %llu refined %llu claimed %llu probed %llu out %llu; E phases %llu (forced %llu), "
                     "S critical path %.3f ms (group 0: %llu tiles, %llu blocks refined in %.3f ms), err %d\n",
                     c.rows_scattered, c.rows_refined, c.rows_claimed, c.rows_probed, c.out_rows, c.evict_phases, c.forced_drains, c.ns_s_crit * 1e-6,
                     c.tiles0, c.blocks0, c.ns_refine0 * 1e-6, e);
    res.groups = G;
    return res;
}
} // namespace phjg
