// CRT on the tensor cores as a persistent, warp-specialised pipeline.
//
// Arithmetic (reference CrtView rns.cuh:225-240, crt_columns / crt_combine
// rns_kernels.cuh:265-364): c = sum_j y_j M_j - v P mod q, v = round(sum_j
// y_j / p_j).  Here -v P rides in the GEMM as a (K+1)-th row: multiplier v,
// constant -P mod q, so
//
//     X = sum_{j<K} y_j M_j + v (-P mod q) = c (mod q),   X < 2^38 q.
//
// The low L - 1 limbs of every constant go through the 8-bit GEMM
// D[m][u] = sum_{j,s} byte_s(y_j(m)) byte_{u-s}(Mlow_j) (entries < 2^26); the
// top limb and the rounding sum run on the CUDA cores.  The prime basis covers
// 2^20 N q^2, so sum_j y_j / p_j lies within 2^-21 of an integer v and any
// estimate within 1/2 - 2^-21 rounds to it.  The stagers sum in single
// precision, y_j rounded to a float times 1 / p_j by FFMA: each term is off by
// less than 2^-23 and each of the roundings of a partial sum by less than
// 2^-24 (K + 1); the host bounds the total (CrtConsts::est_err, 2^-9 at K = 160)
// and the kernel is used only while it is under 1/4.
//
// Organisation on the B200: one CTA per SM walks tiles of 128 coefficients
// (one MMA M); tile i of a CTA accumulates into TMEM buffer i % 2 (256 columns
// each), so a tile's epilogue overlaps the next tile's staging and MMAs:
//   * the constant image (U x 128 bytes per chunk of 32 primes, the last chunk
//     cut to the K steps it uses) is loaded once per CTA by bulk copies and
//     stays resident in shared memory, so the MMAs never wait for constants;
//   * warp 1 (one thread) streams y through a ring of 16 KB boxes with 2-D TMA
//     copies: per chunk a box of 32 primes x 128 coefficients of the
//     prime-major K x N array;
//   * warps 2-9, two threads per row (each half of a chunk's 32 primes), read
//     their 16 values from the box (conflict-free), add up the rounding sum and
//     the top limb, and write the values in the MMA's K-major,
//     128-byte-swizzled byte layout to one of two operand slots.  Boxes and
//     operands have rings of their own, so no warp waits for another's reads
//     (writing over the box in place took a barrier of all eight warps per
//     chunk).  In the last chunk the first half waits for the second half's
//     sums of its 32 rows and puts v in the row;
//   * warp 0 (one thread) issues a chunk's MMAs as soon as its slot holds A,
//     and frees the slot when they finish;
//   * warps 10-13 and 14-17 are two epilogue groups, one per TMEM buffer, one
//     thread per row: a quotient estimate e from the top TMEM columns (within
//     one of floor(X / q)), then one pass from the bottom limb up that
//     assembles X from D with carries, subtracts e q, stores the limbs of its
//     row and tracks the borrows that tell whether X - e q lies in [0, q).  A
//     row whose estimate lies within 2^-8 of an integer (2^-7 of uniform rows) or
//     that came out negative takes a second pass over what it stored, which
//     compares and adds or subtracts q.  Results that are small numbers or q
//     minus small numbers send every row there: with operands all q - 1 this
//     kernel takes 37.3 us for 19.8 at N = 65536, W = 1747, 51.3 for 22.8 at
//     W = 2048.
// Per-prime constants and q come in as kernel parameters and are copied to
// shared memory at the start: read from the parameter bank inside the loops
// (a few KB swept by every chunk and every limb) they made the stagers and
// the epilogue several times slower.
// One epilogue loop serves every limb count: L = 4 at N = 65536 8.6 us a launch,
// L = 16 9.8, L = 55 20.8, where a copy of it unrolled over the limbs took 18.4,
// 22.3 and 32.9 (and stored rows that start off a 16-byte boundary word by word).
// What bounds it is the latency of the stagers and of the epilogue's chain, not
// memory (53 MB in 23.6 us at L = 64) or the tensor cores (20% active): four
// tiles a CTA took 24.8 us, 17.0 without the epilogue, 14.1 without the stagers'
// sums too; one tile 10.5, 6.7 and 5.7 (before the rounding sum lost its shifts,
// 1 us at L = 64).
//
// Every wait is bounded (DevPoint::wait_ns); a timeout raises an abort flag
// that every role checks, the copy and MMA issuers wait out what they have in
// flight, and the error word gets bit 1.
#include "device.cuh"
#include "kernels.h"
#include "pdl.cuh"
#include "tc.cuh"
#include "tmap.h"

#include <cmath>

namespace fpm {

namespace {

constexpr int kThreads = 576;             // 18 warps
constexpr int kMmaWarp = 0;               // also allocates TMEM
constexpr int kYWarp = 1;
constexpr int kStagerWarp0 = 2;           // warps 2-9: row m, half h of each chunk
constexpr int kStagers = 256;
constexpr int kEpiWarp0 = 10;             // warps 10-13 (group 0), 14-17 (group 1)
constexpr uint32_t kCrtTile = 128;        // coefficients per tile
constexpr uint32_t kChunk = 32;           // K rows (primes) per chunk
constexpr int kMaxSlots = 6;
constexpr uint32_t kMaxASlots = 2;
// A slot holds a y box, [32 primes][128 coefficients] u32, or the A operand
// made from one, 128 rows x 128 bytes, 128-byte swizzled: the first ny slots
// are boxes, the last na operands.
constexpr uint32_t kSlot = kChunk * kCrtTile * 4;
constexpr size_t kSmemLimit = 227 * 1024;
// Shared copies of the constants: {1 / p_j bits, top_j} per row j < 32 nch
// (zero beyond the K + 1 rows; kMaxK + 2 entries, a multiple of 16 bytes), then q.
constexpr size_t kConstBytes = (kMaxK + 2) * sizeof(uint2) + ((kMaxL + 2) * 4 + 15) / 16 * 16;

constexpr int kBars = 34;

// Shared-memory plan, the same on host and device: the resident constants
// from 0, then the slot ring (1024-byte aligned), the per-tile top-limb words,
// the constants and the barriers.
struct Layout {
    uint32_t b_bytes;      // resident constant image
    uint32_t slots;        // of both rings
    __host__ __device__ uint32_t na() const { return slots >= 4 ? kMaxASlots : 1u; }
    __host__ __device__ uint32_t ny() const { return slots - na(); }
    __host__ __device__ size_t slot_off() const { return (size_t(b_bytes) + 1023) / 1024 * 1024; }
    __host__ __device__ size_t meta_off() const { return slot_off() + slots * size_t(kSlot); }
    __host__ __device__ size_t xch_off() const { return meta_off() + 2 * kCrtTile * sizeof(uint4); }
    __host__ __device__ size_t const_off() const { return xch_off() + 2 * kCrtTile * sizeof(uint4); }
    __host__ __device__ size_t bar_off() const { return const_off() + kConstBytes; }
    __host__ __device__ size_t bytes() const { return bar_off() + kBars * 8 + 16; }
};

// Bytes of the constant image the MMAs read: full chunks of U x 128 bytes,
// the last one cut to the K steps (8 rows each) its K + 1 - 32 (nch - 1) rows
// need (a prefix of the chunk: 2 core columns of U x 16 bytes per step).
__host__ __device__ inline uint32_t resident_b_bytes(int K, uint32_t U) {
    const int nch = (K + 1 + static_cast<int>(kChunk) - 1) / static_cast<int>(kChunk);
    const int last_rows = K + 1 - static_cast<int>(kChunk) * (nch - 1);
    const uint32_t last_steps = static_cast<uint32_t>(last_rows + 7) / 8;
    return static_cast<uint32_t>(nch - 1) * U * 128 + last_steps * 2 * U * 16;
}

// cta_tiles: tiles a CTA takes; no ring is longer than its chunks (shared
// memory that is not asked for lets the next kernel's blocks start beside this
// one's).
Layout make_layout(int K, uint32_t U, uint32_t cta_tiles) {
    Layout l{resident_b_bytes(K, U), kMaxSlots};
    while (l.slots > 2 && l.bytes() > kSmemLimit) --l.slots;
    const uint32_t chunks = cta_tiles * ((static_cast<uint32_t>(K) + 1 + kChunk - 1) / kChunk);
    if (l.slots > 2 * chunks) l.slots = 2 * chunks;
    return l;
}

struct Smem {
    uint8_t* b;          // resident constant image
    uint8_t* slot;       // [ny][kSlot] y boxes
    uint8_t* aop;        // [na][kSlot] A operands
    uint4* meta;         // [2][128] {top-limb words 0, 1, 2, -}
    uint4* xch;          // [2][128] second halves' sums {rounding sum, top-limb words 0, 1, 2}
    uint2* kc;           // [kMaxK + 2] {1 / p_j bits, top_j}
    uint32_t* qs;        // [L + 2] q, zero above L
    uint64_t* b_full;    // [1] the constant image landed
    uint64_t* y_full;    // [kMaxSlots] the slot's TMA box landed
    uint64_t* y_empty;   // [kMaxSlots] and the stagers have read it
    uint64_t* a_full;    // [kMaxASlots] 128 rows of A staged
    uint64_t* a_empty;   // [kMaxASlots] and its MMAs finished
    uint64_t* x_full;    // [4][2] the second halves' sums of 32 rows are in xch
    uint64_t* d_full;    // [2] a tile's MMAs finished (per TMEM buffer)
    uint64_t* d_empty;   // [2] its epilogue group has read TMEM
    uint64_t* m_full;    // [2] a tile's top-limb words staged
    uint64_t* m_empty;   // [2] and read
    uint32_t* tmem_base;
    volatile uint32_t* abort;
};

__device__ inline Smem carve(uint8_t* base, const Layout& lay) {
    Smem s;
    s.b = base;
    s.slot = base + lay.slot_off();
    s.aop = s.slot + lay.ny() * kSlot;
    s.meta = reinterpret_cast<uint4*>(base + lay.meta_off());
    s.xch = reinterpret_cast<uint4*>(base + lay.xch_off());
    s.kc = reinterpret_cast<uint2*>(base + lay.const_off());
    s.qs = reinterpret_cast<uint32_t*>(base + lay.const_off() + (kMaxK + 2) * sizeof(uint2));
    uint64_t* bars = reinterpret_cast<uint64_t*>(base + lay.bar_off());
    s.b_full = bars;
    s.y_full = bars + 1;
    s.y_empty = s.y_full + kMaxSlots;
    s.a_full = s.y_empty + kMaxSlots;
    s.a_empty = s.a_full + kMaxASlots;
    s.x_full = s.a_empty + kMaxASlots;
    s.d_full = s.x_full + 8;
    s.d_empty = s.d_full + 2;
    s.m_full = s.d_full + 4;
    s.m_empty = s.d_full + 6;
    s.tmem_base = reinterpret_cast<uint32_t*>(bars + kBars);
    s.abort = s.tmem_base + 1;
    return s;
}

static_assert(1 + 2 * kMaxSlots + 2 * kMaxASlots + 8 + 8 <= kBars, "barriers fit before tmem_base");

// Waits for this thread's TMEM loads; naming the registers keeps every read of
// them below the wait.
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15])
                 :
                 : "memory");
}

// The carry chain of one row from the bottom limb up.  X = Z0 + 2^8 Z1 +
// 2^16 Z2 + 2^24 Z3, Z_s the number whose limb l is D[4 l + s] (< 2^26), so
// limb l of 2^(8 s) Z_s is one funnel shift of Z_s[l - 1] and Z_s[l] and the
// limb's share of X is z0 + s1 + s2 + s3 < 2^34 with no products.  e q's words
// come from a running sum, two multiply-adds a limb: what is carried is below
// 2^33, e_lo q_l below (2^32 - 1)^2 and e_hi q_(l-1) below 2^38, so the sum
// never wraps.  The carry chain itself is one signed 64-bit add a limb.
struct LimbChain {
    uint32_t e_lo, e_hi;
    uint64_t eq = 0;     // e q from this limb's word up, the limbs below it added
    uint32_t qp = 0;
    uint32_t z1p = 0, z2p = 0, z3p = 0;
    int64_t cy = 0;
    __device__ __forceinline__ LimbChain(uint32_t lo, uint32_t hi) : e_lo(lo), e_hi(hi) {}
    // extra: what the limb gets besides its columns (a top-limb word).
    __device__ __forceinline__ uint32_t limb(uint32_t z0, uint32_t z1, uint32_t z2, uint32_t z3, uint32_t extra,
                                             uint32_t qk) {
        const uint64_t sd = static_cast<uint64_t>(z0) + __funnelshift_l(z1p, z1, 8) +
                            static_cast<uint64_t>(__funnelshift_l(z2p, z2, 16)) + __funnelshift_l(z3p, z3, 24) + extra;
        z1p = z1;
        z2p = z2;
        z3p = z3;
        eq = static_cast<uint64_t>(e_lo) * qk + (eq >> 32);
        eq += static_cast<uint64_t>(e_hi) * qp;
        qp = qk;
        const int64_t v = static_cast<int64_t>(sd) - static_cast<int64_t>(static_cast<uint32_t>(eq)) + cy;
        cy = v >> 32;
        return static_cast<uint32_t>(v);
    }
    // Four limbs below limb L - 1.
    __device__ __forceinline__ void piece(const uint32_t (&z)[16], const uint32_t* q, uint32_t (&o)[4]) {
        const uint4 q4 = *reinterpret_cast<const uint4*>(q);
        o[0] = limb(z[0], z[1], z[2], z[3], 0u, q4.x);
        o[1] = limb(z[4], z[5], z[6], z[7], 0u, q4.y);
        o[2] = limb(z[8], z[9], z[10], z[11], 0u, q4.z);
        o[3] = limb(z[12], z[13], z[14], z[15], 0u, q4.w);
    }
};

// 2^n exactly, |n| < 1000.
__device__ __forceinline__ double pow2(int n) { return __hiloint2double((1023 + n) << 20, 0); }

// Stores a row's limbs four at a time as aligned 16-byte words: a row starts
// r = 0 .. 3 words past a 16-byte boundary (rows of L words, any L and any
// base), so aligned group g holds limbs 4 g - r .. 4 g - r + 3, the last r of
// piece g - 1 and the first 4 - r of piece g.
template <bool EVEN>
struct RowStore {
    uint32_t* base;      // the row, rounded down to 16 bytes
    uint32_t r;
    bool live;
    uint32_t prev[4] = {};
    __device__ __forceinline__ RowStore(uint32_t* row, bool on)
        : base(row - ((reinterpret_cast<uintptr_t>(row) >> 2) & 3u)),
          r(static_cast<uint32_t>(reinterpret_cast<uintptr_t>(row) >> 2) & 3u),
          live(on) {}
    __device__ __forceinline__ void piece(const uint32_t (&o)[4], int g) {
        if constexpr (EVEN) {
            if (live) *reinterpret_cast<uint4*>(base + 4 * g) = make_uint4(o[0], o[1], o[2], o[3]);
            return;
        }
        const bool r1 = (r & 1u) != 0, r2 = (r & 2u) != 0;
        // t[i + 2]: the word i places from the piece's start, moved by r & 1.
        uint32_t t[6];
        t[0] = r1 ? prev[1] : prev[2];
        t[1] = r1 ? prev[2] : prev[3];
        t[2] = r1 ? prev[3] : o[0];
        t[3] = r1 ? o[0] : o[1];
        t[4] = r1 ? o[1] : o[2];
        t[5] = r1 ? o[2] : o[3];
        uint32_t* at = base + 4 * g;
        const uint4 v = make_uint4(r2 ? t[0] : t[2], r2 ? t[1] : t[3], r2 ? t[2] : t[4], r2 ? t[3] : t[5]);
        if (live) {
            if (g > 0 || r == 0) {
                *reinterpret_cast<uint4*>(at) = v;
            } else {
                // The first r words belong to the row before.
                if (r < 2) at[1] = v.y;
                if (r < 3) at[2] = v.z;
                at[3] = v.w;
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) prev[i] = o[i];
    }
    // After piece g - 1: its last r words, which no aligned group has taken.
    __device__ __forceinline__ void flush(int g) {
        if (!EVEN && live && g > 0) {
            uint32_t* at = base + 4 * g;
            if (r == 1) {
                at[0] = prev[3];
            } else if (r == 2) {
                at[0] = prev[2];
                at[1] = prev[3];
            } else if (r == 3) {
                at[0] = prev[1];
                at[1] = prev[2];
                at[2] = prev[3];
            }
        }
    }
};

// EVEN: every row of C starts on a 16-byte boundary (L a multiple of 4, C
// aligned), so a piece of four limbs is one store.
template <bool EVEN>
__global__ void __launch_bounds__(kThreads, 1)
    k_crt_pipe(DevPoint d, const __grid_constant__ CrtConsts cc, const __grid_constant__ CUtensorMap tmY,
               uint32_t* __restrict__ C, uint32_t n_begin, uint32_t n_end, Layout lay) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    pdl_launch_dependents();
    // The 128-byte swizzle is a function of the shared address: the
    // operand atoms need a 1024-byte aligned base (error bit 4 otherwise).
    if (tc::smem_addr(smem_raw) & 1023u) {
        if (threadIdx.x == 0) atomicOr(d.err, 4u);
        return;
    }
    const Smem sm = carve(smem_raw, lay);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int L = d.L;
    const int K = d.K;
    const uint32_t U = d.crt_u;
    const int nch = (K + 1 + static_cast<int>(kChunk) - 1) / static_cast<int>(kChunk);   // K + 1 rows
    const uint32_t tiles = (n_end - n_begin + kCrtTile - 1) / kCrtTile;
    const uint32_t ny = lay.ny(), na = lay.na();
    const uint64_t lim = d.wait_ns;

    if (threadIdx.x == 0) {
        tc::mbar_init(sm.b_full, 1);
        for (int i = 0; i < 2; ++i) {
            tc::mbar_init(&sm.d_full[i], 1);
            tc::mbar_init(&sm.d_empty[i], kCrtTile / 32);
            tc::mbar_init(&sm.m_full[i], kCrtTile / 32);
            tc::mbar_init(&sm.m_empty[i], kCrtTile / 32);
        }
        for (uint32_t i = 0; i < ny; ++i) {
            tc::mbar_init(&sm.y_full[i], 1);
            tc::mbar_init(&sm.y_empty[i], kStagers / 32);
        }
        for (uint32_t i = 0; i < na; ++i) {
            tc::mbar_init(&sm.a_full[i], kStagers / 32);
            tc::mbar_init(&sm.a_empty[i], 1);
        }
        for (int i = 0; i < 8; ++i) tc::mbar_init(&sm.x_full[i], 1);
        *sm.abort = 0;
        tc::fence_mbar_init();
        // The constant image is read-only plan data: it loads under the
        // preceding kernel's tail.  (Test hook: with kFaultCrt it is never
        // requested, so the MMA issuer's wait for it runs out.)
        if (!(d.fault & kFaultCrt)) {
            tc::mbar_arrive_expect_tx(sm.b_full, lay.b_bytes);
            const uint32_t chunk_bytes = U * 128;
            for (uint32_t off = 0; off < lay.b_bytes; off += chunk_bytes) {
                const uint32_t n = lay.b_bytes - off < chunk_bytes ? lay.b_bytes - off : chunk_bytes;
                tc::bulk_g2s(sm.b + off, d.crt_img_v + off, n, sm.b_full);
            }
        }
    }
    for (int j = threadIdx.x; j <= kMaxK; j += kThreads)
        sm.kc[j] = make_uint2(j < K ? __float_as_uint(cc.cf[j]) : 0u, j <= K ? cc.top[j] : 0u);
    for (int k = threadIdx.x; k < kMaxL + 2; k += kThreads) sm.qs[k] = cc.q[k];
    if (warp == kYWarp && lane == 0) tc::prefetch_tmap(&tmY);
    if (warp == 0) tc::tmem_alloc(sm.tmem_base, 512);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *sm.tmem_base;

    if (warp == kYWarp) {
        // ---- y boxes through the TMA ring ----
        if (lane == 0) {
            pdl_wait();   // y is the preceding kernel's output
            uint32_t par[kMaxSlots] = {};
            bool armed[kMaxSlots] = {};
            uint32_t g = 0;
            bool ok = true;
            for (uint32_t t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
                const int x = static_cast<int>(n_begin + t * kCrtTile);
                for (int c = 0; c < nch; ++c, ++g) {
                    const uint32_t s = g % ny, u = g / ny;
                    if (u >= 1 && !(ok = tc::wait_or_abort(&sm.y_empty[s], (u - 1) & 1, sm.abort, lim))) break;
                    tc::mbar_arrive_expect_tx(&sm.y_full[s], kSlot);
                    tc::tma_load_2d(sm.slot + s * kSlot, &tmY, x, c * static_cast<int>(kChunk), &sm.y_full[s]);
                    par[s] = u & 1;
                    armed[s] = true;
                }
            }
            for (uint32_t s = 0; s < ny; ++s) {
                if (armed[s]) tc::wait_parity(&sm.y_full[s], par[s], lim);
            }
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        // ---- MMA issuer ----
        if (lane == 0) {
            const uint32_t idesc = tc::idesc_u8(U);
            uint32_t g = 0, i = 0;
            uint64_t* last_bar = nullptr;
            uint32_t last_par = 0;
            bool ok = tc::wait_or_abort(sm.b_full, 0, sm.abort, lim);
            for (uint32_t t = blockIdx.x; ok && t < tiles; t += gridDim.x, ++i) {
                const uint32_t buf = i & 1, use = i >> 1;
                if (use >= 1 && !(ok = tc::wait_or_abort(&sm.d_empty[buf], (use - 1) & 1, sm.abort, lim))) break;
                for (int c = 0; c < nch; ++c, ++g) {
                    const uint32_t s = g % na;
                    const uint32_t ph = (g / na) & 1;
                    ok = tc::wait_or_abort(&sm.a_full[s], ph, sm.abort, lim);
                    if (!ok) break;
                    tc::tc_fence_after();
                    const uint32_t a0 = tc::smem_addr(sm.aop + s * kSlot), b0 = tc::smem_addr(sm.b + c * U * 128);
                    // K steps of 8 rows; the last chunk stops after row K.
                    const int rows_c = min(static_cast<int>(kChunk), K + 1 - c * static_cast<int>(kChunk));
                    const uint32_t ksteps = static_cast<uint32_t>(rows_c + 7) / 8;
                    // A and the full constant chunks are 128-byte swizzled;
                    // the short last chunk keeps the plain core-matrix layout
                    // (only its first K steps are resident).
                    const bool swz_b = c + 1 < nch;
                    for (uint32_t kk = 0; kk < ksteps; ++kk) {
                        const uint64_t ad = tc::smem_desc_sw128(a0 + kk * 32);
                        const uint64_t bd = swz_b ? tc::smem_desc_sw128(b0 + kk * 32)
                                                  : tc::smem_desc(b0 + kk * 2 * (U * 16), U * 16, 128);
                        tc::mma_u8(tmem + buf * 256, ad, bd, idesc, c > 0 || kk > 0);
                    }
                    tc::mma_commit(&sm.a_empty[s]);
                    last_bar = &sm.a_empty[s];
                    last_par = ph;
                }
                if (!ok) break;
                tc::mma_commit(&sm.d_full[buf]);
            }
            // MMAs still running, and the constant image (after an abort
            // too), must finish before the CTA may exit.
            if (last_bar) tc::wait_parity(last_bar, last_par, lim);
            if (!(d.fault & kFaultCrt)) tc::wait_parity(sm.b_full, 0, lim);
        }
        __syncwarp();
    } else if (warp < kEpiWarp0) {
        // ---- stagers: thread = row m, primes 16 h .. 16 h + 15 of each chunk ----
        pdl_wait();
        const uint32_t st = threadIdx.x - kStagerWarp0 * 32;
        const uint32_t m = st & (kCrtTile - 1), h = st / kCrtTile;
        constexpr int kHalf = static_cast<int>(kChunk) / 2;
        const uint32_t rw = m >> 5;   // the warp pair (halves 0 and 1) of these 32 rows
        uint32_t g = 0, i = 0;
        uint32_t ys = 0, yph = 0, as_ = 0, aph = 0;   // ring positions of chunk g and their phases
        for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x, ++i) {
            const uint32_t n0 = n_begin + t * kCrtTile;
            const bool live = m < min(kCrtTile, n_end - n0);
            const uint32_t xb = i & 1;
            // The rounding sum as kPart float partial sums; the top-limb sum
            // sum_j y_j top_j (< 2^71) as 96 bits (t01, t2), fed by 64-bit
            // pairs of products (each < 2^63 with 31-bit primes, so a pair
            // cannot wrap).
            constexpr int kPart = 4;
            float vf[kPart] = {};
            uint64_t t01 = 0;
            uint32_t t2 = 0;
            bool ok = true;
#pragma unroll 1
            for (int c = 0; c < nch; ++c) {
                uint32_t yv[kHalf];
                ok = tc::wait_or_abort(&sm.y_full[ys], yph, sm.abort, lim);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const uint32_t yrow = tc::smem_addr(sm.slot + ys * kSlot) + 4 * (h * kHalf * kCrtTile + m);
#pragma unroll
                for (int jj = 0; jj < kHalf; ++jj) yv[jj] = tc::ld_shared_once(yrow + 4 * jj * kCrtTile);
                // Rows j >= K of the box read as zero and 1 / p_j as 0, so every
                // row of the chunk takes part without a test.
                const uint4* kc = reinterpret_cast<const uint4*>(sm.kc + c * static_cast<int>(kChunk) + h * kHalf);
#pragma unroll
                for (int q2 = 0; q2 < kHalf / 2; ++q2) {
                    const uint4 kj = kc[q2];   // two primes
                    const uint32_t y0 = yv[2 * q2], y1 = yv[2 * q2 + 1];
                    vf[(2 * q2) % kPart] = fmaf(__uint2float_rn(y0), __uint_as_float(kj.x), vf[(2 * q2) % kPart]);
                    vf[(2 * q2 + 1) % kPart] = fmaf(__uint2float_rn(y1), __uint_as_float(kj.z), vf[(2 * q2 + 1) % kPart]);
                    const uint64_t grp = static_cast<uint64_t>(y0) * kj.y + static_cast<uint64_t>(y1) * kj.w;
                    t01 += grp;
                    t2 += t01 < grp ? 1u : 0u;
                }
                // Every value has been used, so its load is done: the box goes
                // back (the fence orders these reads before the TMA's writes).
                tc::fence_proxy_async_smem();
                tc::mbar_arrive_warp(&sm.y_empty[ys]);
                if (++ys == ny) ys = 0, yph ^= 1;
                // The operand slot is free once the MMAs of chunk g - na are done.
                if (g >= na) {
                    ok = tc::wait_or_abort(&sm.a_empty[as_], aph ^ 1, sm.abort, lim);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                }
                // Row m's 128 bytes in the 128-byte-swizzle layout
                // (sw128_offset); this half owns 16-byte pieces 4 h .. 4 h + 3.
                uint8_t* as = sm.aop + as_ * kSlot + m * 128;
                const bool last = c == nch - 1;
                if (last && h == 0) {
                    // Row K: the multiplier v of -P mod q, from both halves'
                    // sums, once the second half has written its pieces and
                    // sums (xch[xb] is rewritten two tiles on, at least two
                    // chunks: not before this chunk's MMAs).
                    ok = tc::wait_or_abort(&sm.x_full[2 * rw + xb], (i >> 1) & 1, sm.abort, lim);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    const float vh = (vf[0] + vf[1]) + (vf[2] + vf[3]);
                    const uint4 x = sm.xch[xb * kCrtTile + m];
                    int v = __float2int_rn(vh + __uint_as_float(x.x));
                    v = v < 0 ? 0 : (v > K ? K : v);
                    const uint32_t vu = live ? static_cast<uint32_t>(v) : 0u;
                    const uint64_t other = (static_cast<uint64_t>(x.z) << 32) | x.y;
                    t01 += other;
                    t2 += x.w + (t01 < other ? 1u : 0u);
                    const uint64_t pv = static_cast<uint64_t>(vu) * sm.kc[K].y;
                    t01 += pv;
                    t2 += t01 < pv ? 1u : 0u;
                    const uint32_t kk = static_cast<uint32_t>(K) % kChunk;
#pragma unroll
                    for (int jj = 0; jj < kHalf; ++jj)
                        if (static_cast<uint32_t>(jj) == kk) yv[jj] = vu;
                    if (kk >= static_cast<uint32_t>(kHalf))
                        *reinterpret_cast<uint32_t*>(as + (((kk >> 2) ^ (m & 7)) << 4) + 4 * (kk & 3)) = vu;
                }
#pragma unroll
                for (int q4 = 0; q4 < 4; ++q4)
                    *reinterpret_cast<uint4*>(as + (((4 * h + q4) ^ (m & 7)) << 4)) =
                        make_uint4(yv[4 * q4], yv[4 * q4 + 1], yv[4 * q4 + 2], yv[4 * q4 + 3]);
                if (last && h == 1) {
                    const float vh = (vf[0] + vf[1]) + (vf[2] + vf[3]);
                    sm.xch[xb * kCrtTile + m] = make_uint4(__float_as_uint(vh), static_cast<uint32_t>(t01),
                                                           static_cast<uint32_t>(t01 >> 32), t2);
                    tc::mbar_arrive_warp(&sm.x_full[2 * rw + xb]);
                }
                tc::fence_proxy_async_smem();
                tc::mbar_arrive_warp(&sm.a_full[as_]);
                if (++as_ == na) as_ = 0, aph ^= 1;
                ++g;
            }
            if (!ok) break;
            if (h == 0) {
                const int p = i & 1;
                if (i >= 2) {
                    ok = tc::wait_or_abort(&sm.m_empty[p], ((i - 2) >> 1) & 1, sm.abort, lim);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                }
                // Top-limb sum as three words.
                sm.meta[p * kCrtTile + m] =
                    make_uint4(static_cast<uint32_t>(t01), static_cast<uint32_t>(t01 >> 32), t2, 0u);
                tc::mbar_arrive_warp(&sm.m_full[p]);
            }
        }
    } else {
        // ---- epilogue group grp (TMEM buffer grp): thread = one row ----
        pdl_wait();
        const uint32_t grp = static_cast<uint32_t>(warp - kEpiWarp0) >> 2, qd = warp & 3;
        const uint32_t row = qd * 32 + lane;
        const uint32_t tq = tmem + ((qd * 32) << 16) + grp * 256;
        const int drop = top_drop(L);
        const int tail = (L - 1) / 4;                    // the piece (four limbs, 16 columns) of limb L - 1
        const int top_piece = drop / 4;
        const double piece_w = pow2(32 * (4 * top_piece - drop)), top_w = pow2(32 * (L - 1 - drop));
        const bool spill = static_cast<uint32_t>(tail + 1) * 16 < U;   // the piece above `tail` has columns
        uint32_t k = 0;   // this group's tiles so far
        for (uint32_t t = blockIdx.x + grp * gridDim.x; t < tiles; t += 2 * gridDim.x, ++k) {
            const uint32_t n0 = n_begin + t * kCrtTile;
            const uint32_t rows_t = min(kCrtTile, n_end - n0);
            const bool live = row < rows_t;
            uint32_t* crow = C + static_cast<size_t>(n0 + (live ? row : 0)) * L;
            RowStore<EVEN> out(crow, live);
            bool ok = tc::wait_or_abort(&sm.m_full[grp], k & 1, sm.abort, lim);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const uint4 meta = sm.meta[grp * kCrtTile + row];
            tc::mbar_arrive_warp(&sm.m_empty[grp]);
            ok = tc::wait_or_abort(&sm.d_full[grp], k & 1, sm.abort, lim);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc::tc_fence_after();
            uint32_t ra[16], rb[16];
            // Quotient estimate from the limbs at and above `drop` (columns
            // past limb L - 1 are zero) and the top-limb words:
            // |estimate - X / q| < 2^-11, so e is within one.  A limb's four
            // columns add up exactly in 64 bits before the conversion.
            double xd = 0;
            for (int pc = tail; pc >= top_piece; --pc) {
                tc::tmem_ld16(tq + pc * 16, ra);
                tmem_wait(ra);
#pragma unroll
                for (int ii = 3; ii >= 0; --ii) {
                    const uint64_t z = ra[4 * ii] + (static_cast<uint64_t>(ra[4 * ii + 1]) << 8) +
                                       (static_cast<uint64_t>(ra[4 * ii + 2]) << 16) +
                                       (static_cast<uint64_t>(ra[4 * ii + 3]) << 24);
                    xd = xd * 4294967296.0 + static_cast<double>(z);
                }
            }
            tc::tmem_ld16(tq, ra);
            // (meta.x is limb L - 1's, meta.y and meta.z the two above it.)
            xd = xd * piece_w + ((static_cast<double>(meta.z) * 4294967296.0 + static_cast<double>(meta.y)) * 4294967296.0 +
                                 static_cast<double>(meta.x)) * top_w;
            const double fq = xd * d.q_top_inv;
            const double f = floor(fq);
            const uint64_t e = f > 0 ? static_cast<uint64_t>(f) : 0;
            // With the fraction of the estimate at least 2^-8 from an integer,
            // e = floor(X / q) exactly and X - e q lies in [0, q); otherwise it
            // lies in [-q, 2q) and the row is checked after the pass.
            const double frac = fq - f;
            const bool near = !(frac >= 0x1p-8 && frac <= 1.0 - 0x1p-8);
            // One pass from the bottom, one loop for every L: unrolled over
            // the 66 limbs of the widest modulus (as it was, but for four
            // common L) the code alone cost a small product 6 us of
            // instruction fetch.  TMEM pieces are double-buffered: piece
            // pc + 1 loads while piece pc is used.
            LimbChain ch(static_cast<uint32_t>(e), static_cast<uint32_t>(e >> 32));
            uint32_t o[4];
            tmem_wait(ra);
            int pc = 0;
#pragma unroll 1
            for (; pc + 2 <= tail; pc += 2) {
                tc::tmem_ld16(tq + (pc + 1) * 16, rb);
                ch.piece(ra, sm.qs + 4 * pc, o);
                out.piece(o, pc);
                tmem_wait(rb);
                tc::tmem_ld16(tq + (pc + 2) * 16, ra);
                ch.piece(rb, sm.qs + 4 * pc + 4, o);
                out.piece(o, pc + 1);
                tmem_wait(ra);
            }
            if (pc < tail) {
                tc::tmem_ld16(tq + (pc + 1) * 16, rb);
                ch.piece(ra, sm.qs + 4 * pc, o);
                out.piece(o, pc);
                tmem_wait(rb);
#pragma unroll
                for (int ii = 0; ii < 16; ++ii) ra[ii] = rb[ii];
            }
            // Limbs 4 tail .. L + 1: the last one to four of the result, with
            // the top-limb words, and what lies above it.
#pragma unroll
            for (int ii = 0; ii < 16; ++ii) rb[ii] = 0;
            if (spill) {
                tc::tmem_ld16(tq + (tail + 1) * 16, rb);
                tmem_wait(rb);
            }
            uint32_t over = 0;
            out.flush(tail);
#pragma unroll
            for (int ii = 0; ii < 6; ++ii) {
                const int kl = 4 * tail + ii;
                if (EVEN || kl < L + 2) {
                    const uint32_t(&z)[16] = ii < 4 ? ra : rb;
                    const uint32_t x = EVEN ? (ii == 3 ? meta.x : ii == 4 ? meta.y : ii == 5 ? meta.z : 0u)
                                            : (kl == L - 1 ? meta.x : kl == L ? meta.y : kl == L + 1 ? meta.z : 0u);
                    const uint32_t y = ch.limb(z[4 * (ii & 3)], z[4 * (ii & 3) + 1], z[4 * (ii & 3) + 2],
                                               z[4 * (ii & 3) + 3], x, sm.qs[kl]);
                    if (EVEN ? ii < 4 : kl < L) {
                        o[ii & 3] = y;
                        if (EVEN) {
                            if (ii == 3) out.piece(o, tail);
                        } else if (live) {
                            crow[kl] = y;
                        }
                    } else {
                        over |= y;   // limbs L and L + 1 of a non-negative result
                    }
                }
            }
            const int64_t cy = ch.cy;
            // TMEM is read: the MMAs of this buffer's next tile may start.
            tc::tc_fence_before();
            tc::mbar_arrive_warp(&sm.d_empty[grp]);
            // r = X - e q in [-q, 2q): negative (cy < 0) adds q; a row near an
            // integer quotient subtracts q when r >= q (r past limb L - 1, or
            // its low L limbs at least q).  Rare: a second pass over the row.
            if (live && (cy < 0 || near)) {
                bool sub = false;
                if (cy >= 0) {
                    sub = over != 0;
                    if (!sub) {
                        uint32_t cb = 0;
                        for (int kk = 0; kk < L; ++kk)
                            cb = static_cast<uint32_t>((static_cast<uint64_t>(crow[kk]) - sm.qs[kk] - cb) >> 63);
                        sub = cb == 0;
                    }
                }
                if (cy < 0 || sub) {
                    uint32_t cb = 0;
                    for (int kk = 0; kk < L; ++kk) {
                        const uint32_t x = crow[kk], qk = sm.qs[kk];
                        if (cy < 0) {
                            const uint64_t sum = static_cast<uint64_t>(x) + qk + cb;
                            crow[kk] = static_cast<uint32_t>(sum);
                            cb = static_cast<uint32_t>(sum >> 32);
                        } else {
                            const uint64_t dd = static_cast<uint64_t>(x) - qk - cb;
                            crow[kk] = static_cast<uint32_t>(dd);
                            cb = static_cast<uint32_t>(dd >> 63);
                        }
                    }
                }
            }
        }
    }

    tc::tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *sm.abort) atomicOr(d.err, 2u);
    if (warp == 0) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, 512);
    }
}

}  // namespace

CrtConsts make_crt_consts(const HostPlan& pl, const uint32_t* top) {
    CrtConsts cc{};
    // The rounding sum's constants and a bound on its error (see the head of
    // this file): per term y_j's and 1 / p_j's roundings (y_j / p_j < 1), and one
    // rounding of a sum below K + 1 per term and per final addition.
    for (int j = 0; j <= pl.K; ++j) {
        if (j < pl.K) cc.cf[j] = static_cast<float>(1.0 / pl.primes[j]);
        cc.top[j] = top[j];
    }
    const double ulp = std::ldexp(1.0, -24);
    cc.est_err = static_cast<float>(3 * pl.K * ulp + (pl.K + 8.0) * (pl.K + 1.0) * ulp);
    for (int k = 0; k < pl.L; ++k) cc.q[k] = pl.q[k];
    return cc;
}

bool crt_pipe_supported(const DevPoint& d, const CrtConsts& cc, const uint32_t* Y, uint32_t n_begin,
                        uint32_t n_end) {
    // TMA boxes of y: 16-byte aligned base, row pitch (N words) and column
    // coordinates (n_begin) a multiple of 4 words; the constants resident.
    return d.L >= 2 && d.crt_u <= 256 && d.K + 1 <= kMaxK && d.crt_img_v && (d.N & 3) == 0 && d.N >= kCrtTile &&
           (n_begin & 3) == 0 && n_end <= d.N && (reinterpret_cast<uintptr_t>(Y) & 15) == 0 &&
           make_layout(d.K, d.crt_u, 1).bytes() <= kSmemLimit && cc.est_err < 0.25f;
}

void crt_pipe_init_attributes() {
    for (auto kernel : {k_crt_pipe<true>, k_crt_pipe<false>})
        check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemLimit)),
              "crt_pipe smem");
}

void launch_crt_pipe(const DevPoint& d, const CrtConsts& cc, const uint32_t* Y, uint32_t* c, uint32_t n_begin,
                     uint32_t n_end, int sms, cudaStream_t st) {
    if (n_end <= n_begin) return;
    const uint32_t tiles = (n_end - n_begin + kCrtTile - 1) / kCrtTile;
    const uint32_t grid = tiles < static_cast<uint32_t>(sms) ? tiles : static_cast<uint32_t>(sms);
    const Layout lay = make_layout(d.K, d.crt_u, (tiles + grid - 1) / grid);
    // y: K rows of N words, boxes of 32 primes x 128 coefficients.
    const CUtensorMap tm = make_tmap_u32(Y, static_cast<uint64_t>(d.K), d.N, d.N, kChunk, kCrtTile, TmaSwizzle::kNone);
    const size_t smem = lay.bytes();
    const bool even = (d.L & 3) == 0 && (reinterpret_cast<uintptr_t>(c) & 15) == 0;
    check(launch_pdl(even ? k_crt_pipe<true> : k_crt_pipe<false>, dim3(grid), dim3(kThreads), smem, st, d, cc, tm, c,
                     n_begin, n_end, lay),
          "crt launch");
}

}  // namespace fpm
