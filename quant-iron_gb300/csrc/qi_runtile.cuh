// qi_runtile.cuh — tiles of a state in shared memory with three of their bits in registers, as the
// gate runs (qi_gaterun.cu) and the SumOp passes (qi_sumrun.cu) use them.
//
// A tile holds 2^ubits units of 16 bytes (one FP64 or two FP32 amplitudes).  In a phase a thread
// holds the 2^S units that differ in the phase's S register bits; the other unit bits are
// spread over the thread index in the order the host gives.
#pragma once
#include "qi_device.cuh"
#include "qi_internal.hpp"

#include <algorithm>

namespace qi {

constexpr int kRunTileBits = 11;    // units of a tile: at most 2^11 (32 KB of shared memory)
constexpr int kRunSelBits = 3;      // register bits of a gate run's phase (2^3 units per thread)
constexpr int kRunMaxProg = 24576;  // bytes of program a pass may hold (copied to shared memory)

struct RunPhaseHdr {   // 32 bytes
    uint8_t rb[4];     // unit bits held in registers
    uint8_t tb[16];    // unit bit of thread-index bit j
    uint16_t nops;
    uint16_t col[4];   // byte offset in the tile of each register bit (swizzled)
    uint16_t pad;
};
static_assert(sizeof(RunPhaseHdr) == 32, "program layout");

// Register amplitudes: index bit 0 is qubit 0 for FP32 (the two halves of a unit), then the
// register bits in ascending qubit order.
template <typename T> struct RunShape;
template <> struct RunShape<double> { static constexpr int kRegBits = kRunSelBits, kUnitBits = 0; };
template <> struct RunShape<float> { static constexpr int kRegBits = kRunSelBits + 1, kUnitBits = 1; };

constexpr int top_bit(int x) { return x >= 16 ? 16 : x >= 8 ? 8 : x >= 4 ? 4 : x >= 2 ? 2 : 1; }

__device__ __forceinline__ double flip_sign(double x, uint32_t s) {   // s = 0 or 1
    return __hiloint2double(__double2hiint(x) ^ (int)(s << 31), __double2loint(x));
}
__device__ __forceinline__ float flip_sign(float x, uint32_t s) { return __int_as_float(__float_as_int(x) ^ (int)(s << 31)); }

// Unit address in shared memory: the low three bits are XORed with the higher groups of three, so
// that eight lanes whose unit indices differ in three bits of distinct residues modulo 3 read
// eight different 16-byte bank groups (the host orders the thread bits that way).
__host__ __device__ __forceinline__ uint32_t run_swizzle(uint32_t u) { return u ^ (((u >> 3) ^ (u >> 6) ^ (u >> 9)) & 7u); }

__device__ __forceinline__ void copy16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// A thread's place in a phase, packed: byte offset of its first unit in the tile (low half), local
// amplitude index with the register bits clear (high half).
__device__ __forceinline__ uint32_t run_place(const RunPhaseHdr &hd, uint32_t tid, int thread_bits, int unit_bit) {
    uint32_t u = 0;
    for (int j = 0; j < thread_bits; ++j) u |= ((tid >> j) & 1u) << hd.tb[j];
    return (run_swizzle(u) << 4) | (u << (16 + unit_bit));
}
// Byte offsets of its 2^S units.
template <int S>
__device__ __forceinline__ void run_units(uint32_t (&at)[1 << S], uint32_t place, const RunPhaseHdr &hd) {
    at[0] = place & 0xffffu;
#pragma unroll
    for (int j = 0; j < S; ++j) {
        const uint32_t c = hd.col[j];
#pragma unroll
        for (int k = 0; k < (1 << j); ++k) at[(1 << j) | k] = at[k] ^ c;
    }
}

template <typename T, int S>
__device__ __forceinline__ void run_load(typename Cx<T>::V2 (&v)[1 << (S + RunShape<T>::kUnitBits)], const void *tile,
                                         const uint32_t (&at)[1 << S]) {
#pragma unroll
    for (int k = 0; k < (1 << S); ++k) {
        const uint4 q = *reinterpret_cast<const uint4 *>(static_cast<const char *>(tile) + at[k]);
        if constexpr (sizeof(T) == 8) {
            v[k] = Cx<T>::make(__hiloint2double((int)q.y, (int)q.x), __hiloint2double((int)q.w, (int)q.z));
        } else {
            v[2 * k] = Cx<T>::make(__uint_as_float(q.x), __uint_as_float(q.y));
            v[2 * k + 1] = Cx<T>::make(__uint_as_float(q.z), __uint_as_float(q.w));
        }
    }
}
template <typename T, int S>
__device__ __forceinline__ void run_store(const typename Cx<T>::V2 (&v)[1 << (S + RunShape<T>::kUnitBits)], void *tile,
                                          const uint32_t (&at)[1 << S]) {
#pragma unroll
    for (int k = 0; k < (1 << S); ++k) {
        uint4 q;
        if constexpr (sizeof(T) == 8) {
            q = make_uint4((uint32_t)__double2loint(v[k].x), (uint32_t)__double2hiint(v[k].x),
                           (uint32_t)__double2loint(v[k].y), (uint32_t)__double2hiint(v[k].y));
        } else {
            q = make_uint4(__float_as_uint(v[2 * k].x), __float_as_uint(v[2 * k].y), __float_as_uint(v[2 * k + 1].x),
                           __float_as_uint(v[2 * k + 1].y));
        }
        *reinterpret_cast<uint4 *>(static_cast<char *>(tile) + at[k]) = q;
    }
}

// Rows of a tile: thread tid's units are tid + i * blockDim.x; with at least one row per step (or one row
// in all) they lie at its own place (first) plus step i's (both from the table of row offsets), in
// global memory and, the swizzle being linear, in the tile.
struct RunCopy {
    uint64_t first;       // unit offset within the state, relative to the tile's base
    uint32_t at;          // byte offset in the tile
    __device__ __forceinline__ RunCopy(const uint64_t *rows, uint32_t tid, int lowu)
        : first(rows[tid >> lowu] + (tid & ((1u << lowu) - 1u))), at(run_swizzle(tid) << 4) {}
    static __device__ __forceinline__ uint64_t step(const uint64_t *rows, uint32_t u0, int lowu) {
        return rows[u0 >> lowu] + (u0 & ((1u << lowu) - 1u));
    }
};

// Host: thread-bit order of a phase whose register unit bits are `regu` (into hd.rb / hd.tb).
inline void run_phase_bits(RunPhaseHdr &hd, uint32_t regu, int ubits) {
    int nr = 0, nb = 0;
    for (int u = 0; u < ubits; ++u)
        if ((regu >> u) & 1u) {
            hd.col[nr] = (uint16_t)(run_swizzle(1u << u) << 4);
            hd.rb[nr++] = (uint8_t)u;
        }
    uint32_t used = regu;
    for (int r = 0; r < 3; ++r)   // three of distinct residues modulo 3 first: no bank conflicts
        for (int u = r; u < ubits; u += 3)
            if (!((used >> u) & 1u)) {
                hd.tb[nb++] = (uint8_t)u;
                used |= 1u << u;
                break;
            }
    for (int u = 0; u < ubits; ++u)
        if (!((used >> u) & 1u)) hd.tb[nb++] = (uint8_t)u;
}

}  // namespace qi
