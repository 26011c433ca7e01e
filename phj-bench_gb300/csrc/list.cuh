// list.cuh -- a warp's list of matching probe rows, written out 128 rows at a
// time (probe.cu, bep_engine.cu).
#pragma once

#include "common.cuh"

namespace phjg
{
// A load of a value read once: without a line of its own in L1, whose lines
// (what shared memory leaves of 228 KB) bound the loads in flight.
__device__ __forceinline__ uint64_t load_once(const uint8_t * p)
{
    uint16_t v;
    asm("ld.global.nc.L1::no_allocate.u8 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint64_t load_once(const uint16_t * p)
{
    uint16_t v;
    asm("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint64_t load_once(const uint32_t * p)
{
    uint32_t v;
    asm("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint64_t load_once(const uint64_t * p)
{
    uint64_t v;
    asm("ld.global.nc.L1::no_allocate.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}

// Four values a lane of a probe payload column of at most 8 bytes, in 64-bit
// registers: rows row0 + idx[u].
__device__ __forceinline__ void load_list(uint64_t (&v)[4], const void * src, uint32_t width, uint64_t row0, const uint32_t (&idx)[4], uint32_t one)
{
    switch (width)
    {
#define PHJ_LOAD_LIST(W, T)                                                                                                                          \
    case W:                                                                                                                                          \
        _Pragma("unroll") for (int u = 0; u < 4; ++u) if (one >> u & 1u) v[u] = load_once(static_cast<const T *>(src) + row0 + idx[u]);                 \
        break;
        PHJ_LOAD_LIST(1, uint8_t)
        PHJ_LOAD_LIST(2, uint16_t)
        PHJ_LOAD_LIST(4, uint32_t)
        default: PHJ_LOAD_LIST(8, uint64_t)
#undef PHJ_LOAD_LIST
    }
}

// Four values a lane to output rows out + 32 * u of a column.
__device__ __forceinline__ void store_list(const uint64_t (&v)[4], void * dst, uint32_t width, uint64_t out, uint32_t one)
{
    switch (width)
    {
#define PHJ_STORE_LIST(W, T)                                                                                                                         \
    case W:                                                                                                                                          \
        _Pragma("unroll") for (int u = 0; u < 4; ++u) if (one >> u & 1u) __stcs(static_cast<T *>(dst) + out + 32 * u, (T)v[u]);                      \
        break;
        PHJ_STORE_LIST(1, uint8_t)
        PHJ_STORE_LIST(2, uint16_t)
        PHJ_STORE_LIST(4, uint32_t)
        default: PHJ_STORE_LIST(8, uint64_t)
#undef PHJ_STORE_LIST
    }
}
} // namespace phjg
