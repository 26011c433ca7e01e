// small.cu -- joins with a small build side in one launch.
//
// A join of a few thousand build rows is a few microseconds of work; run
// through the partitioned path it was a dozen launches and three host round
// trips (4K x 32K rows: 145 us a call).  Here the build side is cut into
// pieces of at most 8192 rows; every CTA builds the table of one piece in its
// shared memory (all CTAs of a piece the same one, from L2) and probes its
// share of the probe side against it.  No partitioning, no table in memory,
// no scratch: the output rows are reserved with one atomic a warp chunk on a
// counter of the context, and the last CTA hands the row count to the host
// through mapped memory and clears the counter for the next join.
//
// The output is sized for one row per probe row, exact for unique build
// keys; a join with more rows is counted and run again (api.cu).  4K x 32K
// rows: 145 -> 31 us a call; the no-allocation join of 16K x 256K 63 -> 39.
#include "internal.h"
#include "piece.cuh"

namespace phjg
{
namespace
{
constexpr int kSNT = 1024;
constexpr uint32_t kSRows = 8192; // build rows a piece holds

struct SmallArgs
{
    ProbeSides sides;
    uint32_t build_rows, probe_rows;
    uint32_t pieces, piece_rows, slots; // slots of a piece's table
    int dup_wide;                       // chunks of kU * 32 rows also where keys have more than four rows
    int unique_only;                    // a piece with a repeated key is not probed
    SmallCounters * ctr;
    SmallResult * host;                 // mapped host memory
};

// CTA c: piece c % pieces, the (c / pieces)-th share of the probe rows.
// Bound by its chain of dependent steps: key load, table build (rows / 1024
// inserts a thread), probe key load, lookup, reservation, payload loads,
// stores.  One chunk of 32 rows a warp (kU 1) spreads a short probe side
// over all SMs; 128 rows (kU 4) keep more loads in flight on a long one.  (Only
// that form counts the rows of repeated keys: it costs half a microsecond.)
template <int kU>
__global__ void __launch_bounds__(kSNT, 1) k_small_join(const __grid_constant__ SmallArgs a)
{
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ ProbeSides J;
    __shared__ int s_linked; // 0 when no key repeats
    __shared__ int s_over;
    uint64_t * keys = reinterpret_cast<uint64_t *>(smem);
    uint32_t * slots = reinterpret_cast<uint32_t *>(smem + 8ull * kSRows);
    uint16_t * nxt = reinterpret_cast<uint16_t *>(slots + a.slots);
    if (threadIdx.x < sizeof(ProbeSides) / 8)
        reinterpret_cast<uint64_t *>(&J)[threadIdx.x] = reinterpret_cast<const uint64_t *>(&a.sides)[threadIdx.x];
    const uint32_t piece = blockIdx.x % a.pieces, share = blockIdx.x / a.pieces, shares = gridDim.x / a.pieces;
    const uint32_t c0 = piece * a.piece_rows, rows = min(a.piece_rows, a.build_rows - min(c0, a.build_rows));
    // (J is visible after this call's barriers)
    build_piece<kSRows, kSNT, (kU > 1)>(a.sides.build.keys + c0, rows, slots, keys, nxt, a.slots - 1, &s_linked);
    const PieceTable<kSRows> tab{slots, keys, nxt, a.slots - 1};
    // the CTAs take a warp's chunk each in turn: a short probe side is spread
    // over all of them
    const uint32_t first = ((threadIdx.x >> 5) * shares + share) * 32, step = shares * (kSNT / 32) * 32;
    if (s_linked && a.unique_only)
    {
        if (threadIdx.x == 0)
            atomicOr(&a.ctr->repeats, 1u);
    }
    else if (s_linked && kU > 1 && (a.dup_wide || s_linked * 4 <= (int)rows * 3))
        probe_piece<kWarpWrites, kU>(J, first * kU, step * kU, a.probe_rows, c0, tab, &a.ctr->out_rows, &s_over);
    else if (s_linked)
        probe_piece<kWarpWrites, 1>(J, first, step, a.probe_rows, c0, tab, &a.ctr->out_rows, &s_over);
    else
        probe_piece<kUnique, kU>(J, first * kU, step * kU, a.probe_rows, c0, tab, &a.ctr->out_rows, &s_over);
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        if (atomicAdd(&a.ctr->done, 1u) == gridDim.x - 1)
        {
            const unsigned long long rows = atomicExch(&a.ctr->out_rows, 0ull);
            a.host->out_rows = atomicExch(&a.ctr->repeats, 0u) ? kSmallJoinRepeats : rows;
            a.ctr->done = 0;
            __threadfence_system();
        }
    }
}
} // namespace

// Every probe row is looked up once a piece, at about 9.8 us a million
// lookups, after 24 us a call.  Measured against the other path (build rows
// of one 8-byte payload): partitioned joins take about 100 us + 10.5 us a
// million probe rows, so the launch wins while (pieces - 1) x probe rows
// stay under about 7.6M (64K x 512K: 74 us against 142; 64K x 2M: 177
// against 159).  The no-allocation join's global table takes 50 us + 38 us a
// million, less the more build rows there are; with 8 to 20 payload bytes a
// side the launch wins up to four pieces (16K x 256K: 40 against 64 us; 32K x
// 786K 63-73 against 76-80) and beyond them while (pieces - 1) x probe rows
// stay under 1.4M (40K x 320K: 50-55 against 56-60; 40K x 512K 59-67 against
// 61-63; 57K x 256K 54-61 against 60; 57K x 456K 65-74 against 64-67).
bool small_join_eligible(const phj_ctx * ctx, uint64_t build_rows, uint64_t probe_rows, bool noalloc)
{
    const uint64_t pieces = ceil_div(build_rows, kSRows), free_pieces = noalloc ? 3 : 1;
    const uint64_t most = (uint64_t)ctx->num_sms * (!noalloc ? 50000 : pieces <= 4 ? 20400 : 9200);
    return build_rows > 0 && probe_rows > 0 && pieces <= 8 && probe_rows < (1ull << 31) &&
           (pieces <= free_pieces || (pieces - 1) * probe_rows <= most);
}

uint64_t small_join(phj_ctx * ctx, const Cols & build, uint64_t build_rows, const Cols & probe, uint64_t probe_rows, uint64_t * out_keys,
                    void * const * out_l, void * const * out_r, uint64_t out_cap, const char * name, bool unique_only, cudaEvent_t start, cudaEvent_t stop)
{
    SmallArgs a{};
    a.sides.build = build;
    a.sides.probe = probe;
    a.sides.out_keys = out_keys;
    for (uint32_t c = 0; c < build.n; ++c)
        a.sides.out_l[c] = out_l[c];
    for (uint32_t c = 0; c < probe.n; ++c)
        a.sides.out_r[c] = out_r[c];
    a.sides.out_cap = out_cap;
    a.build_rows = (uint32_t)build_rows;
    a.probe_rows = (uint32_t)probe_rows;
    a.pieces = (uint32_t)ceil_div(build_rows, kSRows);
    a.piece_rows = (uint32_t)ceil_div(build_rows, a.pieces);
    a.slots = (uint32_t)std::max<uint64_t>(4, bit_ceil64(a.piece_rows + a.piece_rows / 2));
    a.unique_only = unique_only ? 1 : 0;
    a.ctr = ctx->small_ctr;
    a.host = reinterpret_cast<SmallResult *>(small_host(ctx));
    const bool wide = probe_rows > (uint64_t)ctx->num_sms / a.pieces * kSNT;
    const uint64_t rows_cta = (uint64_t)kSNT * (wide ? 2 : 1);
    const uint32_t shares = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div(probe_rows, rows_cta), (uint64_t)ctx->num_sms / a.pieces));
    // Keys of more than four rows make a chunk's output rows many: a warp then
    // takes 128 probe rows at a time only if it has two such chunks to do, and
    // else 32 (8K rows of 64 a key x 400K: 300 us a join against 420).  Fewer
    // rows a key want the loads in flight (64K rows of two a key and piece x
    // 400K: 151 against 218).
    a.dup_wide = ceil_div(probe_rows, 128) >= 2ull * shares * (kSNT / 32);
    const size_t smem = 8ull * kSRows + 4ull * a.slots + 2ull * a.piece_rows;
    if (ctx->time_kernels)
    {
        KernelRecord r;
        r.name = name;
        r.form = "small_join";
        r.rows = probe_rows;
        r.start = start;
        r.stop = stop;
        ctx->records.push_back(r);
    }
    PHJ_CUDA(cudaEventRecord(start, ctx->stream));
    (wide ? k_small_join<4> : k_small_join<1>)<<<shares * a.pieces, kSNT, smem, ctx->stream>>>(a);
    PHJ_LAUNCHED(ctx, "small_join");
    PHJ_CUDA(cudaEventRecord(stop, ctx->stream));
    PHJ_CUDA(cudaStreamSynchronize(ctx->stream));
    const uint64_t rows = const_cast<volatile SmallResult *>(a.host)->out_rows;
    return rows;
}

void set_small_smem_limits()
{
    const int most = 8 * kSRows + 4 * 2 * kSRows + 2 * kSRows;
    for (auto * k : {k_small_join<1>, k_small_join<4>})
        PHJ_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
}
} // namespace phjg
