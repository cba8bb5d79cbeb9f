// Device building blocks shared by the transform kernels: rounds through
// shared memory, a column tile's global accesses, and the rows of a row tile.
#pragma once

#include "device.cuh"
#include "ntt_engine.cuh"

#include <type_traits>

namespace fpm {

namespace {

template <int NSUB, int XS, class SWZ, int RB>
using RP = Rounds<NSUB, XS, SWZ, RB>;

// Column-pass shared layout for RB register bits.
template <int RB>
using SwzC = std::conditional_t<RB == 3, SwzCol, SwzRow>;

// The threads that own one tile: the whole block, or one 128-thread half of a
// 256-thread block (the grouped row pass of mixed geometries runs two
// 128-thread tiles per block).
struct BlockTeam {
    static __device__ __forceinline__ uint32_t tid() { return threadIdx.x; }
    static __device__ __forceinline__ void sync() { __syncthreads(); }
};
struct HalfTeam {
    static __device__ __forceinline__ uint32_t tid() { return threadIdx.x & 127u; }
    static __device__ __forceinline__ void sync() {
        asm volatile("bar.sync %0, 128;" ::"r"(1u + (threadIdx.x >> 7)) : "memory");
    }
};

// Round R through shared memory on NV tiles.
template <int NSUB, int XS, class SWZ, int RB, int R, bool LAZY, int NV, class TEAM = BlockTeam, class TW>
__device__ __forceinline__ void fwd_step(uint32_t* const (&tiles)[NV], const TW& tw, uint32_t p) {
    const uint32_t base = round_base<NSUB, XS, SWZ, RB, R>(TEAM::tid());
    uint32_t v[NV][1 << RB];
#pragma unroll
    for (int o = 0; o < NV; ++o) load_round<NSUB, XS, SWZ, RB, R>(tiles[o], v[o], base);
    fwd_round<NSUB, XS, SWZ, RB, R, LAZY, NV>(v, base, tw, p);
#pragma unroll
    for (int o = 0; o < NV; ++o) store_round<NSUB, XS, SWZ, RB, R>(tiles[o], v[o], base);
    TEAM::sync();
}

template <int NSUB, int XS, class SWZ, int RB, int R, int REND, bool LAZY, int NV, class TEAM = BlockTeam,
          class TW>
__device__ __forceinline__ void fwd_range(uint32_t* const (&tiles)[NV], const TW& tw, uint32_t p) {
    if constexpr (R < REND) {
        fwd_step<NSUB, XS, SWZ, RB, R, LAZY, NV, TEAM>(tiles, tw, p);
        fwd_range<NSUB, XS, SWZ, RB, R + 1, REND, LAZY, NV, TEAM>(tiles, tw, p);
    }
}

// Inverse rounds R, R - 1, ..., RLO through shared memory.
template <int NSUB, int XS, class SWZ, int RB, int R, int RLO, bool LAZY, bool NEG, class TEAM = BlockTeam,
          class TW>
__device__ __forceinline__ void inv_range(uint32_t* tile, const TW& tw, uint32_t p) {
    if constexpr (R >= RLO) {
        const uint32_t base = round_base<NSUB, XS, SWZ, RB, R>(TEAM::tid());
        uint32_t v[1 << RB];
        load_round<NSUB, XS, SWZ, RB, R>(tile, v, base);
        inv_round<NSUB, XS, SWZ, RB, R, LAZY, NEG>(v, base, tw, p);
        store_round<NSUB, XS, SWZ, RB, R>(tile, v, base);
        TEAM::sync();
        inv_range<NSUB, XS, SWZ, RB, R - 1, RLO, LAZY, NEG, TEAM>(tile, tw, p);
    }
}

// Canonical residue from a lazy one (< 4p).
__device__ __forceinline__ uint32_t canon4(uint32_t x, uint32_t p) {
    x = umin32(x, x - 2 * p);
    return umin32(x, x - p);
}

// The pointwise product of two forward transforms' values (lazy ones below 4p):
// x y 2^-32 mod p, below 2p (lazy) or canonical.
template <bool LAZY>
__device__ __forceinline__ uint32_t pointwise(uint32_t x, uint32_t y, const PrimeConsts& pc) {
    if constexpr (LAZY) {
        // below 2p each, so the Montgomery product stays below 2p
        x = umin32(x, x - 2 * pc.p);
        y = umin32(y, y - 2 * pc.p);
    }
    return mont_mul(x, y, pc.p, pc.pneg);
}

template <int LOGR, int LOGS>
__device__ __forceinline__ uint32_t col_offset(uint32_t i, uint32_t c0) {
    constexpr int XS = 11 - LOGR;
    return ((i >> XS) << LOGS) + c0 + (i & ((1u << XS) - 1u));
}

template <int LOGR, int LOGS, int RB, int R, int NV>
__device__ __forceinline__ void col_global_load(const uint32_t* const (&X)[NV], uint32_t (&v)[NV][1 << RB],
                                                uint32_t base, uint32_t c0) {
    constexpr int XS = 11 - LOGR, sh = RP<LOGR, XS, SwzC<RB>, RB>::lo(R);
    constexpr uint32_t step = (1u << LOGS) << sh;
    const uint32_t at = col_offset<LOGR, LOGS>(base, c0);
#pragma unroll
    for (int o = 0; o < NV; ++o) {
        const uint32_t* x = X[o] + at;
#pragma unroll
        for (int k = 0; k < (1 << RB); ++k) v[o][k] = x[k * step];
    }
}

template <int LOGR, int LOGS, int RB, int R, int NV>
__device__ __forceinline__ void col_global_store(uint32_t* const (&X)[NV], const uint32_t (&v)[NV][1 << RB],
                                                 uint32_t base, uint32_t c0) {
    constexpr int XS = 11 - LOGR, sh = RP<LOGR, XS, SwzC<RB>, RB>::lo(R);
    constexpr uint32_t step = (1u << LOGS) << sh;
    const uint32_t at = col_offset<LOGR, LOGS>(base, c0);
#pragma unroll
    for (int o = 0; o < NV; ++o) {
        uint32_t* x = X[o] + at;
#pragma unroll
        for (int k = 0; k < (1 << RB); ++k) x[k * step] = v[o][k];
    }
}

// A row tile: G whole rows, 2048 elements, or 4096 for S = 2048, so that a row
// always has its partner beside it: with one row a block each block brought in
// both rows' twiddle tables (32 KB for 16 KB of residues), twice the table
// traffic of the other lengths, and four blocks of 128 threads filled an SM's
// shared memory.  Transform before -> after: N = 2^18, K = 71 218 -> 198 us,
// N = 2^17, K = 140 199 -> 183, K = 36 51.4 -> 49.8.
template <int LOGS>
struct RowGeom {
    static constexpr int kBits = LOGS == 11 ? 12 : 11;
    static constexpr uint32_t kTile = 1u << kBits;
    static constexpr uint32_t S = 1u << LOGS;
    static constexpr uint32_t G = kTile >> LOGS;
    static_assert(G >= 2, "rows and their partners");
    static constexpr uint32_t kSlots = G;
    static constexpr uint32_t kStride = S + 4;                 // entries; pads rows across banks
    static constexpr uint32_t kFlip = G / 2;
    static constexpr uint32_t kPairsPerBlock = G / 2;
};
template <int LOGS>
using RowSwz = SwzRowT<RowGeom<LOGS>::kBits>;

template <int LOGS>
__device__ __forceinline__ uint32_t row_of_slot(uint32_t slot, uint32_t u0, uint32_t R) {
    using RG = RowGeom<LOGS>;
    return slot < RG::G / 2 ? u0 + slot : R - 1 - u0 - (slot - RG::G / 2);
}

template <int LOGS>
constexpr int row_threads() {
    return 1 << (RowGeom<LOGS>::kBits - row_pass_rb(LOGS));
}

// The row pass's tables barrier sits after the tiles and the tables.
template <int LOGS>
constexpr size_t row_bar_offset() {
    return 2 * RowGeom<LOGS>::kTile * sizeof(uint32_t) + RowGeom<LOGS>::kSlots * RowGeom<LOGS>::kStride * sizeof(uint2);
}

// Bytes of tiles and tables of a mixed-geometry row block for rows up to
// 2^max_log_s: room for one 256-thread tile or, in halves, two 128-thread ones.
// (With a region the size of the largest tile for each half, S = 2048 took 130
// KB, one block an SM: N = 2^17, 2^16, 2^14 and 2^13 in one batch 295 us, with
// this 262 at the same code otherwise.)
constexpr uint32_t mixed_row_bytes(uint32_t max_log_s) {
    const int threads[6] = {row_threads<6>(), row_threads<7>(), row_threads<8>(),
                            row_threads<9>(), row_threads<10>(), row_threads<11>()};
    const size_t need[6] = {row_bar_offset<6>(), row_bar_offset<7>(), row_bar_offset<8>(),
                            row_bar_offset<9>(), row_bar_offset<10>(), row_bar_offset<11>()};
    size_t r = 0;
    for (uint32_t s = 6; s <= max_log_s && s <= 11; ++s) {
        const size_t n = threads[s - 6] == 256 ? need[s - 6] : 2 * need[s - 6];
        r = n > r ? n : r;
    }
    return static_cast<uint32_t>((r + 2047) / 2048 * 2048);   // halves on 1024 bytes
}

}  // namespace

}  // namespace fpm
