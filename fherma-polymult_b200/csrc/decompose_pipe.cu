// Decompose on the tensor cores as a persistent, warp-specialised pipeline.
//
// Same arithmetic as decompose_tc.cu (reference decompose_many rns.cuh:110-128):
//
//     D[m][4j + s] = sum_k byte_k(x_m) * byte_s(2^(8k) sigma_j mod p_j)   (< 2^24)
//     x_m mod p_j  = (sum_s D[m][4j + s] 2^(8s)) mod p_j
//
// Organisation on the B200: one CTA per SM works on one operand (a pair launch
// splits the CTAs between a and b) and walks its 128-coefficient tiles:
//   * warp 0 loads the operand's whole constant image once (equal chunks of at
//     most 64 primes x 4 bytes x 4L bytes: at most 160 KB, resident in shared
//     memory) and then, one thread, issues the MMAs, one chunk at a time: D
//     goes to one of two 256-column TMEM buffers;
//   * warps 1-4 bring each tile's limbs into a ring of operand slots in the
//     MMA's 128-byte-swizzled K-major layout (the layout the tensor cores read at
//     full rate).  Rows of whole 16-byte groups are copied there asynchronously
//     (cp.async), the slot's mbarrier tracking the copies
//     (cp.async.mbarrier.arrive), so a slot is handed to the MMAs the moment its
//     copies land: a warp moves 8 rows x 4 groups at a time, so the global loads
//     are 64-byte runs and the eight lanes of each shared-store phase hit eight
//     different bank groups.  Other rows (RAW) arrive as whole tiles by bulk
//     copies in a ring of their own and are moved to operand slots from there:
//     copied word by word, by cp.async through L1, a pair took 20.1 us at L = 43,
//     N = 65536 (17.6 now), 24.7 at L = 55 (23.4), 27.9 at L = 10, N = 2^18 (24.9);
//   * warps 5-20, four per TMEM lane quadrant, one coefficient per thread,
//     each take a quarter of a chunk's primes: read D, fold the 49-bit sums mod
//     p_j and store the residues (a warp writes 32 consecutive words per
//     prime).
// What bounds it at L = 64 is the fold warps' way through a chunk: TMEM reads,
// folds, stores (106 MB in 23.8 us at K = 139; 16 us without them).  So every
// fold warp gets the same share of every chunk (K = 139 is 3 chunks of 48 with 12
// primes a warp; as 64 + 64 + 11, 16 a warp, the last chunk took as long as a
// full one), warps whose rows and primes all exist store without a test per
// prime, and a store's address is one 32-bit add: together 25.3 us where unequal
// chunks took 33.4 (K = 71 at N = 2^18 47.6 for 68.0, K = 60 at N = 32768 8.2 for
// 9.0, all before the rings and the fold below).  The fold constants stay in the
// parameter bank: from shared memory, which the MMAs load heavily, they took
// K = 60 from 8.2 to 9.1 us (and K = 139 from 25.3 to 24.4).
// The fold constants come from kernel parameters.  Every wait is bounded
// (DevPoint::wait_ns); a timeout raises an abort flag that every role checks,
// and the error word gets bit 0.
#include "device.cuh"
#include "kernels.h"
#include "pdl.cuh"
#include "tc.cuh"

#include <algorithm>

namespace fpm {

namespace {

constexpr int kThreads = 672;                      // 21 warps
constexpr int kLoadWarp0 = 1;                      // warps 1-4
constexpr int kLoaders = 128;
constexpr int kEpiWarp0 = 5;                       // warps 5-20
constexpr int kEpi = 512;
constexpr uint32_t kRows = 128;
constexpr uint32_t kMaxSlots = 8;                  // operand tiles in their ring
constexpr uint32_t kMaxRaw = 8;                    // raw tiles in theirs
constexpr uint32_t kBars = 1 + 2 * kMaxSlots + 2 * kMaxRaw + 4;
constexpr uint32_t kBufCols = 256;                 // TMEM columns of one of the two buffers

// Operand tiles and the constant image in the 128-byte-swizzle layout
// (sw128_offset): a tile is 128 rows, a constant chunk `cols` columns, each
// with kb K bytes.
__host__ __device__ inline uint32_t a_bytes(uint32_t kb) { return static_cast<uint32_t>(sw128_bytes(kRows, kb)); }
__host__ __device__ inline size_t b_bytes(uint32_t kb, int nch, uint32_t cols) {
    return static_cast<size_t>(nch) * sw128_bytes(cols, kb);
}
constexpr size_t kSmemLimit = 227 * 1024;

// The rings: `slots` operand tiles, and for rows that are not whole 16-byte
// groups (L not a multiple of 4) `raw` tiles as they lie in memory (128 L words).
struct Rings {
    uint32_t slots, raw;
};
__host__ __device__ inline uint32_t raw_bytes(int L) { return kRows * 4 * static_cast<uint32_t>(L); }
__host__ inline size_t smem_bytes(uint32_t kb, int nch, uint32_t cols, int L, Rings r) {
    return b_bytes(kb, nch, cols) + r.slots * size_t(a_bytes(kb)) + r.raw * size_t(raw_bytes(L)) + kBars * 8 + 16;
}
// Whole 16-byte groups are copied straight into operand slots, so every slot is
// a tile in flight: as many as shared memory holds beside the constants, 2 to
// kMaxSlots.  A tile's limbs are about 2 us away once the pipelines run, and two
// 16 KB tiles held a CTA to one a microsecond: a pair with more slots than two
// takes 44.1 us for 47.4 (L = 32, K = 71, N = 2^18), 15.0 for 17.3 (L = 16,
// K = 36, N = 2^17); L = 64 has room for two.  Other rows wait in the raw ring, four
// tiles or more of it before a third operand slot.  Without room for a raw tile
// they are copied word by word.
// No ring is longer than the tiles a CTA takes: shared memory that is not
// asked for is there for the next kernel's blocks.
__host__ inline Rings ring_sizes(uint32_t kb, int nch, uint32_t cols, int L, uint32_t cta_tiles) {
    Rings r{2, 0};
    if (L & 3) {
        r = Rings{4, kMaxRaw};
        while (r.raw > 4 && smem_bytes(kb, nch, cols, L, r) > kSmemLimit) --r.raw;
        while (r.slots > 2 && smem_bytes(kb, nch, cols, L, r) > kSmemLimit) --r.slots;
        while (r.raw > 0 && smem_bytes(kb, nch, cols, L, r) > kSmemLimit) --r.raw;
    } else {
        r.slots = kMaxSlots;
        while (r.slots > 2 && smem_bytes(kb, nch, cols, L, r) > kSmemLimit) --r.slots;
    }
    r.slots = r.slots < cta_tiles ? r.slots : cta_tiles;
    r.raw = r.raw < cta_tiles ? r.raw : cta_tiles;
    return r;
}

struct Smem {
    uint8_t* b;            // resident constant image
    uint8_t* a;            // [slots] operand tiles
    uint8_t* raw;          // [raw] tiles as they lie in memory
    uint64_t* b_full;      // [1]
    uint64_t* a_full;      // [kMaxSlots]
    uint64_t* a_empty;     // [kMaxSlots]
    uint64_t* r_full;      // [kMaxRaw] a raw tile landed
    uint64_t* r_empty;     // [kMaxRaw] and the loaders have read it
    uint64_t* d_full;      // [2]
    uint64_t* d_empty;     // [2]
    uint32_t* tmem_base;
    volatile uint32_t* abort;
};

__device__ inline Smem carve(uint8_t* base, uint32_t kb, int nch, uint32_t cols, int L, Rings rings) {
    Smem s;
    s.b = base;
    s.a = base + b_bytes(kb, nch, cols);
    s.raw = s.a + rings.slots * a_bytes(kb);
    s.b_full = reinterpret_cast<uint64_t*>(s.raw + rings.raw * raw_bytes(L));
    s.a_full = s.b_full + 1;
    s.a_empty = s.a_full + kMaxSlots;
    s.r_full = s.a_empty + kMaxSlots;
    s.r_empty = s.r_full + kMaxRaw;
    s.d_full = s.r_empty + kMaxRaw;
    s.d_empty = s.d_full + 2;
    s.tmem_base = reinterpret_cast<uint32_t*>(s.b_full + kBars);
    s.abort = s.tmem_base + 1;
    return s;
}

// Asynchronous global -> shared copies of 16 or 4 bytes; with have == false
// nothing is read and the destination is zero-filled.
__device__ __forceinline__ void cp_async16_zfill(void* dst, const void* src, bool have) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_addr(dst)), "l"(src),
                 "r"(have ? 16u : 0u)
                 : "memory");
}
__device__ __forceinline__ void cp_async4_zfill(void* dst, const void* src, bool have) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(tc::smem_addr(dst)), "l"(src),
                 "r"(have ? 4u : 0u)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// One arrival on `bar` once every cp.async this thread issued so far has
// completed (the barrier's count includes it: .noinc).
__device__ __forceinline__ void cp_async_arrive_noinc(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_addr(bar)) : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Loads NC consecutive columns (a multiple of 8, at most 64) of this thread's
// TMEM lane and waits for them; naming the registers keeps every read of them
// below the wait.
template <int NC>
__device__ __forceinline__ void tmem_read(uint32_t taddr, uint32_t (&r)[NC]) {
    static_assert(NC % 8 == 0 && NC <= 64, "columns in eights");
    int at = 0;
#pragma unroll
    for (; at + 32 <= NC; at += 32) tc::tmem_ld32(taddr + at, *reinterpret_cast<uint32_t(*)[32]>(r + at));
    if constexpr (NC % 32 >= 16) {
        tc::tmem_ld16(taddr + NC / 32 * 32, *reinterpret_cast<uint32_t(*)[16]>(r + NC / 32 * 32));
    }
    if constexpr (NC % 16 == 8) tc::tmem_ld8(taddr + NC - 8, r + NC - 8);
    tc::tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < NC; i += 8)
        asm volatile("" : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]), "+r"(r[i + 4]), "+r"(r[i + 5]),
                          "+r"(r[i + 6]), "+r"(r[i + 7])::"memory");
}

// A GEMM sum D is below 4L 255^2 <= 256 * 65025 (L <= 64), so both halves of
// sum_s D_s 2^(8s), A = D_0 + 2^8 D_1 and B = D_2 + 2^8 D_3, are below
// 257 * 256 * 65025 < 2^32, and the residue is X = A + 2^16 B mod p, X < 2^48.1.
static_assert(kMaxL <= 64, "D_0 + 2^8 D_1 must fit 32 bits");
// Canonical: f = {p, 2^16 mod p, its Shoup companion, floor(2^32 / p)}.
__device__ __forceinline__ uint32_t fold_halves(uint32_t A, uint32_t B, uint4 f) {
    return add_mod(shoup(A, 1u, f.w, f.x), shoup(B, f.y, f.z, f.x), f.x);
}
// A value below 2p, congruent to the residue, for a transform whose first
// butterflies take lazy input: f = {p, mu = floor(2^49 / p)}.  With
// t = floor(B / 2) + floor(A / 2^17) > X / 2^17 - 1.5 the quotient estimate
// floor(t mu / 2^32) is at most X / p and above X / p - X / 2^49 - 1.5 2^17 / p
// - 1, so more than X / p - 1.6 (p > 2^24).  One high product and one low one,
// where a Shoup quotient for each half took two of each on the pipe that
// multiplies: 44.1 -> 40.7 us for a pair at N = 2^18, K = 71, L = 32, 15.0 ->
// 14.6 at N = 2^17, K = 36, L = 16.
__device__ __forceinline__ uint32_t fold_halves(uint32_t A, uint32_t B, uint2 f) {
    const uint32_t q = mulhi32((B >> 1) + (A >> 17), f.y);
    return A + (B << 16) - q * f.x;
}
template <bool LAZY>
__device__ __forceinline__ auto fold_consts(const DecConsts& fc, int j) {
    if constexpr (LAZY) {
        return fc.lazy[j];
    } else {
        return fc.fold[j];
    }
}

// CTAs [0, split) take operand 0 (la -> ra), [split, gridDim.x) operand 1.
// P: primes per fold warp and chunk.
// RAW: rows that are not whole 16-byte groups, in a raw ring.
// parts > 1 (few tiles): each tile is `parts` CTAs' work, part i taking the 4 P
// primes from 4 P i of the image's (whose chunks hold fc.piece / P such runs).
template <int P, bool LAZY, bool RAW>
__global__ void __launch_bounds__(kThreads, 1)
    k_decompose_pipe(DevPoint d, const __grid_constant__ DecConsts fc, const uint32_t* __restrict__ la,
                     const uint32_t* __restrict__ lb, uint32_t* __restrict__ ra, uint32_t* __restrict__ rb,
                     int operand0, uint32_t n_begin, uint32_t n_end, uint32_t split, uint32_t parts, Rings rings) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    pdl_launch_dependents();
    // The 128-byte swizzle is a function of the shared address: the
    // operand atoms need a 1024-byte aligned base (error bit 4 otherwise).
    if (tc::smem_addr(smem_raw) & 1023u) {
        if (threadIdx.x == 0) atomicOr(d.err, 4u);
        return;
    }
    const uint32_t kb = d.dec_kb;
    const int nch = parts > 1 ? 1 : static_cast<int>(fc.chunks);
    constexpr uint32_t cols = 16 * P;
    // (The shuffle tells the compiler that the warp index is uniform.)
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int L = d.L, K = d.K;
    const Smem sm = carve(smem_raw, kb, nch, cols, L, rings);
    const uint32_t slots = rings.slots;
    const bool second = blockIdx.x >= split;
    const int operand = operand0 + (second ? 1 : 0);
    const uint32_t* limbs = second ? lb : la;
    uint32_t* res = second ? rb : ra;
    const uint8_t* img = fc.img[operand];
    // This CTA's place among its operand's: part of every tile, first tile, step.
    const uint32_t place = blockIdx.x - (second ? split : 0), places = second ? gridDim.x - split : split;
    const uint32_t part = parts > 1 ? place % parts : 0, t0 = parts > 1 ? place / parts : place;
    const uint32_t ts = parts > 1 ? places / parts : places;
    const uint32_t tiles = (n_end - n_begin + kRows - 1) / kRows;
    const uint32_t chunk_bytes = static_cast<uint32_t>(sw128_bytes(cols, kb));
    const uint64_t lim = d.wait_ns;

    if (threadIdx.x == 0) {
        tc::mbar_init(sm.b_full, 1);
        for (uint32_t i = 0; i < slots; ++i) {
            tc::mbar_init(&sm.a_full[i], kLoaders);
            tc::mbar_init(&sm.a_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(&sm.d_full[i], 1);
            tc::mbar_init(&sm.d_empty[i], kEpi / 32);
        }
        for (uint32_t i = 0; RAW && i < rings.raw; ++i) {
            tc::mbar_init(&sm.r_full[i], 1);
            tc::mbar_init(&sm.r_empty[i], kLoaders / 32);
        }
        *sm.abort = 0;
        tc::fence_mbar_init();
        // The constant image is read-only plan data: it loads under the
        // preceding kernel's tail.
        // (Test hook: with kFaultDecompose the image is never requested, so the
        // MMA issuer's wait for it runs out.)
        const uint32_t total = static_cast<uint32_t>(b_bytes(kb, nch, cols));
        if (!(d.fault & kFaultDecompose)) {
            tc::mbar_arrive_expect_tx(sm.b_full, total);
            if (parts == 1) {
                for (uint32_t off = 0; off < total; off += chunk_bytes)
                    tc::bulk_g2s(sm.b + off, img + off, chunk_bytes, sm.b_full);
            } else {
                // The part's columns of the image chunk that holds them, one
                // run per 128 K bytes.
                const uint32_t img_cols = 16 * fc.piece, first = part * P;
                const uint8_t* src = img + (first / fc.piece) * sw128_bytes(img_cols, kb) + (first % fc.piece) * 16 * 128;
                for (uint32_t off = 0; off < total; off += cols * 128, src += img_cols * 128)
                    tc::bulk_g2s(sm.b + off, src, cols * 128, sm.b_full);
            }
        }
    }
    if (warp == 0) tc::tmem_alloc(sm.tmem_base, 512);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *sm.tmem_base;
    pdl_wait();   // the limbs and the residues belong to the kernels around this one

    if (warp == 0) {
        // ---- MMA issuer ----
        if (lane == 0) {
            constexpr uint32_t idesc = tc::idesc_u8(cols);
            bool ok = tc::wait_or_abort(sm.b_full, 0, sm.abort, lim);
            uint64_t* last_bar = nullptr;   // the barrier of the latest commit
            uint32_t last_par = 0;
            uint32_t g = 0, s = 0, ph = 0;   // chunk count; operand slot and its phase
            for (uint32_t t = t0; ok && t < tiles; t += ts) {
                ok = tc::wait_or_abort(&sm.a_full[s], ph, sm.abort, lim);
                if (!ok) break;
                // The limbs came through the generic proxy (cp.async).
                tc::fence_proxy_async_smem();
                const uint32_t a0 = tc::smem_addr(sm.a + s * a_bytes(kb));
                for (int c = 0; c < nch; ++c, ++g) {
                    const int buf = g & 1;
                    if (g >= 2) {
                        ok = tc::wait_or_abort(&sm.d_empty[buf], ((g - 2) >> 1) & 1, sm.abort, lim);
                        if (!ok) break;
                    }
                    tc::tc_fence_after();
                    const uint32_t b0 = tc::smem_addr(sm.b + c * chunk_bytes);
                    for (uint32_t kk = 0; kk < kb / 32; ++kk) {
                        const uint32_t half = kk >> 2, step = (kk & 3) * 32;
                        const uint64_t ad = tc::smem_desc_sw128(a0 + half * kRows * 128 + step);
                        const uint64_t bd = tc::smem_desc_sw128(b0 + half * cols * 128 + step);
                        tc::mma_u8(tmem + buf * kBufCols, ad, bd, idesc, kk > 0);
                    }
                    tc::mma_commit(&sm.d_full[buf]);
                    last_bar = &sm.d_full[buf];
                    last_par = (g >> 1) & 1;
                }
                if (!ok) break;
                tc::mma_commit(&sm.a_empty[s]);
                last_bar = &sm.a_empty[s];
                last_par = ph;
                if (++s == slots) s = 0, ph ^= 1;
            }
            // MMAs still running must finish before the CTA may exit.
            if (last_bar) tc::wait_parity(last_bar, last_par, lim);
            // So must the constant image, if an abort came before it landed.
            if (!(d.fault & kFaultDecompose)) tc::wait_parity(sm.b_full, 0, lim);
        }
        __syncwarp();
    } else if (RAW && warp < kEpiWarp0 &&
               raw_tiles_aligned(reinterpret_cast<uintptr_t>(limbs), n_begin, n_end, L)) {
        // ---- loaders, rows that are not whole 16-byte groups: a tile arrives
        // as it lies in memory, one bulk copy (its rows are contiguous and, 128
        // rows a tile, start and end on 16 bytes); a thread then moves one row
        // to the operand slot, word by word out (lanes L words apart), 16
        // bytes at a time in.
        const uint32_t m = threadIdx.x - kLoadWarp0 * 32;
        const uint32_t G = kb / 16;
        uint32_t s = 0, ph = 0, rs = 0, rph = 0, i = 0;
        // Lane 0 of the first loader warp requests the tiles, rings.raw ahead.
        const bool asks = m == 0;
        uint32_t ask_t = t0, asked = 0;
        auto ask = [&](uint32_t slot) {
            const uint32_t r0 = n_begin + ask_t * kRows;
            const uint32_t bytes = min(kRows, n_end - r0) * 4 * static_cast<uint32_t>(L);
            tc::mbar_arrive_expect_tx(&sm.r_full[slot], bytes);
            tc::bulk_g2s(sm.raw + slot * raw_bytes(L), limbs + static_cast<size_t>(r0) * L, bytes, &sm.r_full[slot]);
            ask_t += ts;
            ++asked;
        };
        if (asks)
            for (uint32_t k = 0; k < rings.raw && ask_t < tiles; ++k) ask(k);
        __syncwarp();
        bool ok = true;
        for (uint32_t t = t0; t < tiles; t += ts, ++i) {
            const uint32_t nk = min(kRows, n_end - (n_begin + t * kRows));
            ok = tc::wait_or_abort(&sm.r_full[rs], rph, sm.abort, lim);
            if (ok && i >= slots) ok = tc::wait_or_abort(&sm.a_empty[s], ph ^ 1, sm.abort, lim);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const uint32_t row = tc::smem_addr(sm.raw + rs * raw_bytes(L)) + m * 4 * static_cast<uint32_t>(L);
            uint8_t* at = sm.a + s * a_bytes(kb);
#pragma unroll 4
            for (uint32_t gq = 0; gq < G; ++gq) {
                uint32_t w[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k)
                    w[k] = m < nk && 4 * gq + k < static_cast<uint32_t>(L) ? tc::ld_shared_once(row + 16 * gq + 4 * k) : 0u;
                *reinterpret_cast<uint4*>(at + sw128_offset(m, 16 * gq, kRows)) = make_uint4(w[0], w[1], w[2], w[3]);
            }
            // The row is written (to the MMAs) and read (back to the copies).
            tc::fence_proxy_async_smem();
            tc::mbar_arrive(&sm.a_full[s]);
            tc::mbar_arrive_warp(&sm.r_empty[rs]);
            if (asks && ask_t < tiles) {
                ok = tc::wait_or_abort(&sm.r_empty[rs], rph, sm.abort, lim);
                if (ok) ask(rs);
            }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            if (++s == slots) s = 0, ph ^= 1;
            if (++rs == rings.raw) rs = 0, rph ^= 1;
        }
        // Every copy asked for lands before the CTA may exit.
        if (asks) {
            const uint32_t from = asked > rings.raw ? asked - rings.raw : 0;
            for (uint32_t k = from; k < asked; ++k)
                tc::wait_parity(&sm.r_full[k % rings.raw], (k / rings.raw) & 1, lim);
        }
        __syncwarp();
    } else if (warp < kEpiWarp0) {
        // ---- loaders: each tile's limbs, K-major with a padded K stride ----
        // The copies go from global to shared memory asynchronously (cp.async,
        // zero-filled where a position has no limb: rows past nk, limbs past
        // L), so one whole tile is in flight while the previous one completes.
        // A warp covers an 8-row x 4-group block per instruction: every lane
        // group of a shared-store phase hits distinct banks.
        const uint32_t lt = threadIdx.x - kLoadWarp0 * 32, lw = lt >> 5;
        const bool vec = (reinterpret_cast<uintptr_t>(limbs) & 15u) == 0 && (L & 3) == 0;
        const uint32_t G = kb / 16;                    // 16-byte K groups per row
        const uint32_t r = lane & 7, gi = lane >> 3;   // row in block, group (or limb) in block
        const uint32_t gbs = (G + 3) / 4;
        uint32_t i = 0, s = 0, ph = 0;
        bool ok = true;
        for (uint32_t t = t0; t < tiles; t += ts, ++i) {
            if (i >= slots) {
                ok = tc::wait_or_abort(&sm.a_empty[s], ph ^ 1, sm.abort, lim);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
            uint8_t* at = sm.a + s * a_bytes(kb);
            const uint32_t n0 = n_begin + t * kRows;
            const uint32_t nk = min(kRows, n_end - n0);
            if (vec) {
                // Block (mb, gb): rows 8 mb .. + 7, 16-byte groups 4 gb .. + 3
                // (group gq of a row is limbs 4 gq .. 4 gq + 3).
                const uint32_t q4 = static_cast<uint32_t>(L) / 4;
                const uint4* src4 = reinterpret_cast<const uint4*>(limbs + static_cast<size_t>(n0) * L);
                for (uint32_t blk = lw; blk < 16 * gbs; blk += kLoaders / 32) {
                    const uint32_t mm = 8 * (blk & 15) + r, gq = 4 * (blk >> 4) + gi;
                    if (gq < G) {
                        const bool have = mm < nk && gq < q4;
                        cp_async16_zfill(at + sw128_offset(mm, 16 * gq, kRows), have ? src4 + mm * q4 + gq : src4,
                                         have);
                    }
                }
            } else {
                // Block (mb, gq): rows 8 mb .. + 7, limbs 4 gq .. 4 gq + 3.
                const uint32_t* src = limbs + static_cast<size_t>(n0) * L;
                for (uint32_t blk = lw; blk < 16 * G; blk += kLoaders / 32) {
                    const uint32_t mm = 8 * (blk & 15) + r, l = 4 * (blk >> 4) + gi;
                    const bool have = mm < nk && l < static_cast<uint32_t>(L);
                    cp_async4_zfill(at + sw128_offset(mm, 4 * l, kRows), have ? src + mm * L + l : src, have);
                }
            }
            // The slot's barrier completes when this thread's copies have
            // landed (the hardware arrives for it), so the loader goes on to
            // the next slot at once; the MMA issuer fences the async proxy.
            cp_async_commit();
            cp_async_arrive_noinc(&sm.a_full[s]);
            if (++s == slots) s = 0, ph ^= 1;
        }
        // Whatever is still in flight lands before the CTA may exit.
        cp_async_wait<0>();
    } else {
        // ---- epilogue: thread = one coefficient, P primes of each chunk ----
        const int ew = warp - kEpiWarp0;
        const uint32_t qd = warp & 3, piece = ew >> 2;
        const uint32_t m = qd * 32 + lane;
        const uint32_t tq = tmem + ((qd * 32) << 16) + piece * (4 * P);
        uint32_t g = 0;
        for (uint32_t t = t0; t < tiles; t += ts) {
            const uint32_t n0 = n_begin + t * kRows;
            const bool live = m < min(kRows, n_end - n0);
            const bool whole = n0 + qd * 32 + 32 <= n_end;   // every row of the warp is live
            bool ok = true;
            for (int c = 0; c < nch; ++c, ++g) {
                const int buf = g & 1;
                ok = tc::wait_or_abort(&sm.d_full[buf], (g >> 1) & 1, sm.abort, lim);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc::tc_fence_after();
                const int j0 = (c + static_cast<int>(part)) * (4 * P) + static_cast<int>(piece) * P;
                uint32_t r[4 * P];
                tmem_read<4 * P>(tq + buf * kBufCols, r);
                // The 2 P half-sums are formed before the buffer is released:
                // half as many values stay live through the folds.
                uint32_t hs[P][2];
#pragma unroll
                for (int k = 0; k < P; ++k) {
                    const uint32_t* rr = r + 4 * k;
                    hs[k][0] = rr[0] + (rr[1] << 8);
                    hs[k][1] = rr[2] + (rr[3] << 8);
                }
                tc::tc_fence_before();
                tc::mbar_arrive_warp(&sm.d_empty[buf]);
                // Byte offsets into the residues fit 32 bits (K N words below
                // 2^30), one add a prime.
                uint32_t at = (static_cast<uint32_t>(j0) * d.N + n0 + m) * 4u;
                const uint32_t stride = d.N * 4u;
                uint8_t* out = reinterpret_cast<uint8_t*>(res);
                if (whole && j0 + P <= K) {
#pragma unroll
                    for (int k = 0; k < P; ++k) {
                        *reinterpret_cast<uint32_t*>(out + at) = fold_halves(hs[k][0], hs[k][1], fold_consts<LAZY>(fc, j0 + k));
                        at += stride;
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < P; ++k) {
                        if (live && j0 + k < K)
                            *reinterpret_cast<uint32_t*>(out + at) =
                                fold_halves(hs[k][0], hs[k][1], fold_consts<LAZY>(fc, j0 + k));
                        at += stride;
                    }
                }
            }
            if (!ok) break;
        }
    }

    tc::tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *sm.abort) atomicOr(d.err, 1u);
    if (warp == 0) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, 512);
    }
}

}  // namespace

DecConsts make_dec_consts(const HostPlan& pl, const uint8_t* img_a, const uint8_t* img_b) {
    DecConsts dc{};
    dc.img[0] = img_a;
    dc.img[1] = img_b;
    dc.chunks = pl.dec_wchunks;
    dc.piece = pl.dec_wpiece;
    // Transforms of N >= 2048 start with lazy butterflies; k_ntt_small (N < 256)
    // and the full-reduction window want canonical input, and N = 256 .. 1024,
    // whose butterflies are lazy too, get it as well.
    dc.lazy_out = pl.lazy && pl.g.logN > kSmallLogN && *std::min_element(pl.primes.begin(), pl.primes.end()) > (1u << 24);
    for (int j = 0; j < pl.K; ++j) {
        if (dc.lazy_out) {
            const uint32_t p = pl.primes[j];
            dc.lazy[j] = make_uint2(p, static_cast<uint32_t>((1ull << 49) / p));
        } else {
            dc.fold[j] = pl.dec_fold[j];
        }
    }
    return dc;
}

namespace {

using DecKernel = void (*)(DevPoint, const DecConsts, const uint32_t*, const uint32_t*, uint32_t*, uint32_t*, int,
                           uint32_t, uint32_t, uint32_t, uint32_t, Rings);

template <bool LAZY, bool RAW>
DecKernel dec_kernel(uint32_t piece) {
    switch (piece) {
        case 2: return k_decompose_pipe<2, LAZY, RAW>;
        case 4: return k_decompose_pipe<4, LAZY, RAW>;
        case 6: return k_decompose_pipe<6, LAZY, RAW>;
        case 8: return k_decompose_pipe<8, LAZY, RAW>;
        case 10: return k_decompose_pipe<10, LAZY, RAW>;
        case 12: return k_decompose_pipe<12, LAZY, RAW>;
        case 14: return k_decompose_pipe<14, LAZY, RAW>;
        case 16: return k_decompose_pipe<16, LAZY, RAW>;
        default: throw std::runtime_error("decompose: unsupported chunk size");
    }
}

}  // namespace

bool decompose_pipe_supported(const HostPlan& pl) {
    return pl.K <= kMaxK && pl.dec_wchunks >= 1 && pl.dec_wpiece >= 2 && pl.dec_wpiece <= 16 &&
           smem_bytes(pl.dec_kb, static_cast<int>(pl.dec_wchunks), 16 * pl.dec_wpiece, pl.L, Rings{2, 0}) <= kSmemLimit;
}

void decompose_pipe_init_attributes() {
    for (uint32_t piece = 2; piece <= 16; piece += 2)
        for (DecKernel k : {dec_kernel<false, false>(piece), dec_kernel<false, true>(piece),
                            dec_kernel<true, false>(piece), dec_kernel<true, true>(piece)})
            check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemLimit)),
                  "decompose_pipe smem");
}

void launch_decompose_pipe(const DevPoint& d, const DecConsts& dc, const uint32_t* a, const uint32_t* b,
                           uint32_t* A, uint32_t* B, int operand0, uint32_t n_begin, uint32_t n_end, int sms,
                           cudaStream_t st) {
    if (n_end <= n_begin) return;
    const uint32_t tiles = (n_end - n_begin + kRows - 1) / kRows;
    const int operands = b ? 2 : 1;
    // CTAs per operand: one per SM in all, no more than the operand's tiles.
    uint32_t per = static_cast<uint32_t>(sms) / operands;
    if (per < 1) per = 1;
    if (per > tiles) per = tiles;
    uint32_t piece = dc.piece, parts = 1;
    if (const DecParts cut = decompose_parts(d.N, d.K, tiles, static_cast<uint32_t>(operands), sms); cut.parts > 1) {
        piece = cut.piece;
        parts = cut.parts;
    }
    const uint32_t grid = per * parts * operands;
    const uint32_t split = operands == 2 ? per * parts : grid;
    const int nch = parts > 1 ? 1 : static_cast<int>(dc.chunks);
    const uint32_t cols = 16 * piece;
    const Rings rings = ring_sizes(d.dec_kb, nch, cols, d.L, (tiles + per - 1) / per);
    const DecKernel kernel =
        rings.raw ? (dc.lazy_out ? dec_kernel<true, true>(piece) : dec_kernel<false, true>(piece))
                  : (dc.lazy_out ? dec_kernel<true, false>(piece) : dec_kernel<false, false>(piece));
    check(launch_pdl(kernel, dim3(grid), dim3(kThreads), smem_bytes(d.dec_kb, nch, cols, d.L, rings), st, d, dc, a, b ? b : a, A,
                     B ? B : A, operand0, n_begin, n_end, split, parts, rings),
          "decompose launch");
}

}  // namespace fpm
