// The product's whole transform chain in one launch, for N = 2^8 .. 2^15 where
// that is the faster (ntt_fused_ok).  A product of these sizes is a chain of
// short launches, and what it costs is their number: three passes of a
// microsecond or two of work each, every one behind the start, the first loads
// and the last stores of a launch of its own.
//
//   * N = 2^12 .. 2^15 (rows of S = 64 .. 512, R = 64): a cluster of N / 2048
//     CTAs per prime.  Each holds one 2048-element tile of A and of B: it runs
//     the forward column pass on columns 32 r .. 32 r + 31 (r its rank), sends
//     the results to the row tiles of its peers through distributed shared
//     memory, runs the row pass on its row pairs, sends the product's rows back
//     to the column tiles and runs the inverse column pass.  The residues
//     cross memory once in and once out (12 K N bytes instead of 28).
//   * N = 2^8 .. 2^11 (R = 1): one CTA per prime holds both operands, one
//     group of threads each for the forward rounds; the group of A multiplies
//     and goes back.  (us in a graph, against one butterfly a thread with a
//     barrier and a twiddle load from L2 at every stage: N = 256 K = 6 6.1 -> 1.7,
//     N = 1024 K = 59 10.7 -> 3.1; N = 2048 K = 138, a row pass with one group,
//     8.0 -> 4.3.)
//
// What bounds both is latency: the rounds' serial chain at one block's warps,
// then the exchanges.
//
// Twiddle tables come in by bulk copies under the preceding kernel's tail.  The
// arithmetic is that of the separate passes (ntt.cu), so the residues y_j are
// the same words.
#include "group.cuh"
#include "kernels.h"
#include "ntt_passes.cuh"
#include "pdl.cuh"
#include "tc.cuh"

#include <algorithm>
#include <stdexcept>

namespace fpm {

namespace {

// ---- cluster plumbing ------------------------------------------------------------

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// The first arrival only says that this CTA runs: it has written nothing a peer
// reads.
__device__ __forceinline__ void cluster_arrive_started() {
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
}

// The shared::cluster address, in CTA `rank` of this cluster, of what lies at
// `addr` in this CTA's shared memory.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

__device__ __forceinline__ void cluster_store(uint32_t addr, uint32_t x) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(x) : "memory");
}

// Requests the row tables of this CTA's slots (counted on `bar`, whose expected
// bytes the caller has set); called by warp 0.
template <int LOGS>
__device__ __forceinline__ void row_tables_copy(uint2* tf, const DevPoint& d, int j, uint32_t u0, uint64_t* bar) {
    using RG = RowGeom<LOGS>;
    const uint32_t R = 1u << d.logR;
    for (uint32_t slot = threadIdx.x & 31; slot < RG::kSlots; slot += 32)
        tc::bulk_g2s(tf + slot * RG::kStride, d.row_tw + (static_cast<size_t>(j) * R + row_of_slot<LOGS>(slot, u0, R)) * RG::S,
                     RG::S * sizeof(uint2), bar);
}

// ---- N = 2^12 .. 2^15: a cluster per prime ------------------------------------------

template <int LOGS>
struct ClusterGeom {
    static constexpr int LOGR = 6, XS = 5;
    static constexpr uint32_t R = 1u << LOGR, C = 1u << XS;
    static constexpr int RB = row_pass_rb(LOGS), E = 1 << RB, T = ntt_threads<RB>();
    static constexpr uint32_t kCtas = 1u << (LOGR + LOGS - 11);
    using RG = RowGeom<LOGS>;
    static_assert(RG::G >= 2 && kCtas == R / RG::G && kCtas == (1u << LOGS) / C, "one tile of each pass per CTA");
    // Words: column tiles, row tiles, row tables, column tables, barrier.
    static constexpr uint32_t kRowTiles = 4096, kRowTables = 8192;
    static constexpr uint32_t kColTables = kRowTables + 2 * RG::kSlots * RG::kStride;
    static constexpr uint32_t kBar = kColTables + 2 * 2 * R;
    static constexpr size_t kSmem = kBar * sizeof(uint32_t) + 16;
    static constexpr uint32_t kTableBytes = (RG::kSlots * RG::S + 2 * R) * sizeof(uint2);
    // Resident blocks the registers are sized for (about 50 KB of shared memory
    // each: four fit).
    static constexpr int kBlocks = 4;
};

template <int LOGS, bool LAZY>
__global__ void __launch_bounds__(ClusterGeom<LOGS>::T, ClusterGeom<LOGS>::kBlocks)
    k_ntt_cluster(DevPoint d, uint32_t* A, uint32_t* B) {
    extern __shared__ __align__(1024) uint32_t smem[];
    using CG = ClusterGeom<LOGS>;
    using RG = RowGeom<LOGS>;
    constexpr int LOGR = CG::LOGR, XS = CG::XS, RB = CG::RB, E = CG::E;
    using SC = SwzC<RB>;
    using RPC = RP<LOGR, XS, SC, RB>;
    using RPR = RP<LOGS, 0, SwzRow, RB>;
    static_assert(RPC::all_conflict_free() && RPR::all_conflict_free(), "rounds must be free of bank conflicts");
    constexpr int clast = RPC::kCount - 1, rlast = RPR::kCount - 1;
    const uint32_t rank = blockIdx.x;
    const int j = blockIdx.y;
    uint32_t* const ct[2] = {smem, smem + 2048};                                    // column tiles
    uint32_t* const rt[2] = {smem + CG::kRowTiles, smem + CG::kRowTiles + 2048};    // row tiles
    uint2* tf = reinterpret_cast<uint2*>(smem + CG::kRowTables);
    uint2* cf = reinterpret_cast<uint2*>(smem + CG::kColTables);
    uint2* ci = cf + CG::R;
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + CG::kBar);
    const uint32_t u0 = rank * RG::kPairsPerBlock, c0 = rank * CG::C;
    if (threadIdx.x == 0) {
        tc::mbar_init(bar, 1);
        tc::fence_mbar_init();
        tc::mbar_arrive_expect_tx(bar, CG::kTableBytes);
        tc::bulk_g2s(cf, d.col_f + static_cast<size_t>(j) * CG::R, CG::R * sizeof(uint2), bar);
        tc::bulk_g2s(ci, d.col_i + static_cast<size_t>(j) * CG::R, CG::R * sizeof(uint2), bar);
    }
    __syncthreads();
    if (threadIdx.x < 32) row_tables_copy<LOGS>(tf, d, j, u0, bar);
    __syncwarp();
    cluster_arrive_started();   // waited for before the first store to a peer
    const PrimeConsts pc = d.pc[j];
    const uint32_t p = pc.p;
    constexpr size_t N = size_t(1) << (LOGR + LOGS);
    uint32_t* const X[2] = {A + j * N, B + j * N};
    const SharedTable fcol{cf}, icol{ci};
    const RowTable<LOGS, RG::kStride, false, RG::kFlip> fw{tf};
    const RowTable<LOGS, RG::kStride, true, RG::kFlip> iw{tf};
    // (The CRT's blocks may start once these are at work: let in before the
    // wait they took their places, N = 4096 K = 19 13.4 us a product for 11.1.)
    pdl_wait();
    pdl_launch_dependents();

    // Forward column pass; the last round's results go to the row tiles.
    {
        const uint32_t base = round_base<LOGR, XS, SC, RB, 0>(threadIdx.x);
        uint32_t v[2][E];
        const uint32_t* const Xc[2] = {X[0], X[1]};
        col_global_load<LOGR, LOGS, RB, 0, 2>(Xc, v, base, c0);
        if (!tc::wait_parity(bar, 0, d.wait_ns) && (threadIdx.x & 31) == 0) atomicOr(d.err, 4u);
        fwd_round<LOGR, XS, SC, RB, 0, LAZY, 2>(v, base, fcol, p);
#pragma unroll
        for (int o = 0; o < 2; ++o) store_round<LOGR, XS, SC, RB, 0>(ct[o], v[o], base);
        __syncthreads();
    }
    fwd_range<LOGR, XS, SC, RB, 1, clast, LAZY, 2>(ct, fcol, p);
    {
        const uint32_t base = round_base<LOGR, XS, SC, RB, clast>(threadIdx.x);
        uint32_t v[2][E];
#pragma unroll
        for (int o = 0; o < 2; ++o) load_round<LOGR, XS, SC, RB, clast>(ct[o], v[o], base);
        fwd_round<LOGR, XS, SC, RB, clast, LAZY, 2>(v, base, fcol, p);
        cluster_wait();
        static_assert(RPC::lo(clast) == 0, "the last round's elements are adjacent rows");
        const uint32_t c = c0 + (base & (CG::C - 1));
#pragma unroll
        for (int k = 0; k < E; ++k) {
            // Row u is slot u % (G / 2) of CTA u / (G / 2), its partner
            // R - 1 - u slot G / 2 + u % (G / 2) of the same.
            const uint32_t u = (base >> XS) | k;
            const uint32_t h = u < CG::R / 2 ? u : CG::R - 1 - u;
            const uint32_t slot = (h % RG::kPairsPerBlock) + (u < CG::R / 2 ? 0 : RG::kPairsPerBlock);
            const uint32_t at = tc::smem_addr(rt[0] + SwzRow::f(slot * RG::S + c));
            const uint32_t to = cluster_addr(at, h / RG::kPairsPerBlock);
            cluster_store(to, v[0][k]);
            cluster_store(to + 2048 * sizeof(uint32_t), v[1][k]);
        }
    }
    cluster_arrive();
    cluster_wait();

    // Row pass: forward rounds, product, inverse rounds.
    fwd_range<LOGS, 0, SwzRow, RB, 0, rlast, LAZY, 2>(rt, fw, p);
    {
        const uint32_t base = round_base<LOGS, 0, SwzRow, RB, rlast>(threadIdx.x);
        uint32_t v[2][E];
        load_round<LOGS, 0, SwzRow, RB, rlast>(rt[0], v[0], base);
        load_round<LOGS, 0, SwzRow, RB, rlast>(rt[1], v[1], base);
        fwd_round<LOGS, 0, SwzRow, RB, rlast, LAZY, 2>(v, base, fw, p);
#pragma unroll
        for (int k = 0; k < E; ++k) v[0][k] = pointwise<LAZY>(v[0][k], v[1][k], pc);
        inv_round<LOGS, 0, SwzRow, RB, rlast, LAZY, true>(v[0], base, iw, p);
        store_round<LOGS, 0, SwzRow, RB, rlast>(rt[0], v[0], base);
        __syncthreads();
    }
    inv_range<LOGS, 0, SwzRow, RB, rlast - 1, 1, LAZY, true>(rt[0], iw, p);
    {
        const uint32_t base = round_base<LOGS, 0, SwzRow, RB, 0>(threadIdx.x);
        constexpr int sh = RPR::lo(0);
        uint32_t v[E];
        load_round<LOGS, 0, SwzRow, RB, 0>(rt[0], v, base);
        inv_round<LOGS, 0, SwzRow, RB, 0, LAZY, true>(v, base, iw, p);
        // Back to the column tiles: every CTA has left its column rounds (the
        // barrier above), and none touches its tile before the next one.
        const uint32_t u = row_of_slot<LOGS>(base >> LOGS, u0, CG::R);
#pragma unroll
        for (int k = 0; k < E; ++k) {
            const uint32_t c = (base & (RG::S - 1)) | (k << sh);
            const uint32_t at = tc::smem_addr(ct[0] + SC::f((u << XS) | (c & (CG::C - 1))));
            cluster_store(cluster_addr(at, c >> XS), v[k]);
        }
    }
    cluster_arrive();
    cluster_wait();

    // Inverse column pass; y_j canonical for the CRT.
    {
        const uint32_t base = round_base<LOGR, XS, SC, RB, clast>(threadIdx.x);
        uint32_t v[E];
        load_round<LOGR, XS, SC, RB, clast>(ct[0], v, base);
        inv_round<LOGR, XS, SC, RB, clast, LAZY, false>(v, base, icol, p);
        store_round<LOGR, XS, SC, RB, clast>(ct[0], v, base);
        __syncthreads();
    }
    inv_range<LOGR, XS, SC, RB, clast - 1, 1, LAZY, false>(ct[0], icol, p);
    {
        const uint32_t base = round_base<LOGR, XS, SC, RB, 0>(threadIdx.x);
        uint32_t v[1][E];
        load_round<LOGR, XS, SC, RB, 0>(ct[0], v[0], base);
        inv_round<LOGR, XS, SC, RB, 0, LAZY, false>(v[0], base, icol, p);
        if constexpr (LAZY) {
#pragma unroll
            for (int k = 0; k < E; ++k) v[0][k] = reduce_once(v[0][k], p);
        }
        uint32_t* const Xa[1] = {X[0]};
        col_global_store<LOGR, LOGS, RB, 0, 1>(Xa, v, base, c0);
    }
}

// ---- N = 2^8 .. 2^11: one CTA per prime ------------------------------------------------

template <int LOGN>
struct WholeGeom {
    static constexpr int RB = whole_pass_rb(LOGN), E = 1 << RB;
    static constexpr uint32_t N = 1u << LOGN;
    static constexpr int T = 1 << (LOGN - RB);   // threads per operand
    static constexpr size_t kSmem = 2 * N * sizeof(uint32_t) + N * sizeof(uint2) + 16;
};

// One operand's T threads.
template <int T>
struct OperandTeam {
    static_assert(T % 32 == 0, "whole warps");
    static __device__ __forceinline__ uint32_t tid() { return threadIdx.x % T; }
    static __device__ __forceinline__ void sync() {
        asm volatile("bar.sync %0, %1;" ::"r"(1u + threadIdx.x / T), "n"(T) : "memory");
    }
};

template <int LOGN, bool LAZY>
__global__ void __launch_bounds__(2 * WholeGeom<LOGN>::T) k_ntt_whole(DevPoint d, uint32_t* A, uint32_t* B, int mode) {
    extern __shared__ __align__(1024) uint32_t smem[];
    using WG = WholeGeom<LOGN>;
    constexpr int RB = WG::RB, E = WG::E;
    constexpr uint32_t N = WG::N;
    using SWZ = SwzRowT<LOGN>;
    using RPW = RP<LOGN, 0, SWZ, RB>;
    using TEAM = OperandTeam<WG::T>;
    constexpr int last = RPW::kCount - 1;
    const int j = blockIdx.x;
    // Operand 0 is A's threads, 1 B's.
    const uint32_t op = threadIdx.x / WG::T, tid = TEAM::tid();
    uint32_t* const tile[1] = {smem + op * N};
    uint2* tf = reinterpret_cast<uint2*>(smem + 2 * N);
    uint64_t* bar = reinterpret_cast<uint64_t*>(tf + N);
    if (threadIdx.x == 0) {
        tc::mbar_init(bar, 1);
        tc::fence_mbar_init();
        tc::mbar_arrive_expect_tx(bar, N * sizeof(uint2));
        tc::bulk_g2s(tf, d.row_tw + static_cast<size_t>(j) * N, N * sizeof(uint2), bar);
    }
    const PrimeConsts pc = d.pc[j];
    const uint32_t p = pc.p;
    uint32_t* X = (op ? B : A) + static_cast<size_t>(j) * N;
    const RowTable<LOGN, 0, false, 0> fw{tf};
    const RowTable<LOGN, 0, true, 0> iw{tf};
    __syncthreads();
    // (After the wait, as in the cluster kernel: let in before it the CRT's
    // blocks took N = 1024 K = 59 from 11.7 to 12.2 us a product.)
    pdl_wait();
    pdl_launch_dependents();
    uint32_t v[1][E];
    {
        const uint32_t base = round_base<LOGN, 0, SWZ, RB, 0>(tid);
        constexpr int sh = RPW::lo(0);
#pragma unroll
        for (int k = 0; k < E; ++k) v[0][k] = X[base | (k << sh)];
        if (!tc::wait_parity(bar, 0, d.wait_ns) && (threadIdx.x & 31) == 0) atomicOr(d.err, 4u);
        fwd_round<LOGN, 0, SWZ, RB, 0, LAZY, 1>(v, base, fw, p);
        store_round<LOGN, 0, SWZ, RB, 0>(tile[0], v[0], base);
        TEAM::sync();
    }
    fwd_range<LOGN, 0, SWZ, RB, 1, last, LAZY, 1, TEAM>(tile, fw, p);
    const uint32_t base = round_base<LOGN, 0, SWZ, RB, last>(tid);
    load_round<LOGN, 0, SWZ, RB, last>(tile[0], v[0], base);
    fwd_round<LOGN, 0, SWZ, RB, last, LAZY, 1>(v, base, fw, p);
    if (mode == kRowForward) {
        if constexpr (LAZY) {
#pragma unroll
            for (int k = 0; k < E; ++k) v[0][k] = canon4(v[0][k], p);
        }
        // Through shared memory, so that a warp's stores are whole lines.
        store_round<LOGN, 0, SWZ, RB, last>(tile[0], v[0], base);
        TEAM::sync();
#pragma unroll
        for (int k = 0; k < E; ++k) X[tid + k * WG::T] = tile[0][SWZ::f(tid + k * WG::T)];
        return;
    }
    // B's values to A's threads, which go on alone.
    if (op) store_round<LOGN, 0, SWZ, RB, last>(tile[0], v[0], base);
    __syncthreads();
    if (op) return;
    uint32_t w[E];
    load_round<LOGN, 0, SWZ, RB, last>(smem + N, w, base);
#pragma unroll
    for (int k = 0; k < E; ++k) v[0][k] = pointwise<LAZY>(v[0][k], w[k], pc);
    inv_round<LOGN, 0, SWZ, RB, last, LAZY, true>(v[0], base, iw, p);
    store_round<LOGN, 0, SWZ, RB, last>(tile[0], v[0], base);
    TEAM::sync();
    inv_range<LOGN, 0, SWZ, RB, last - 1, 1, LAZY, true, TEAM>(tile[0], iw, p);
    {
        const uint32_t b0 = round_base<LOGN, 0, SWZ, RB, 0>(tid);
        constexpr int sh = RPW::lo(0);
        load_round<LOGN, 0, SWZ, RB, 0>(tile[0], v[0], b0);
        inv_round<LOGN, 0, SWZ, RB, 0, LAZY, true>(v[0], b0, iw, p);
        if constexpr (LAZY) {
#pragma unroll
            for (int k = 0; k < E; ++k) v[0][k] = reduce_once(v[0][k], p);
        }
#pragma unroll
        for (int k = 0; k < E; ++k) X[b0 | (k << sh)] = v[0][k];
    }
}

// The products of N = 2048 of a batch in one launch: a (possibly persistent)
// grid walks the table's blocks, one a prime.  A batch has blocks enough for
// throughput to count, so one group of N / 16 threads holds both operands (a
// twiddle load serves both, and no thread idles through the inverse rounds).
// Batch of 32, us: one launch a product, each behind the one before, 171 at
// W = 128 and 278 at W = 2048; one launch, two groups a block 65.7 and 209;
// this 65.0 and 187.
template <bool LAZY>
__global__ void __launch_bounds__(WholeGeom<11>::T, 5) k_ntt_whole_group(const __grid_constant__ GroupTable t) {
    extern __shared__ __align__(1024) uint32_t smem[];
    constexpr int LOGN = 11;
    using WG = WholeGeom<LOGN>;
    constexpr int RB = WG::RB, E = WG::E;
    constexpr uint32_t N = WG::N;
    using SWZ = SwzRowT<LOGN>;
    using RPW = RP<LOGN, 0, SWZ, RB>;
    constexpr int last = RPW::kCount - 1, sh = RPW::lo(0);
    uint32_t* const tiles[2] = {smem, smem + N};
    uint2* tf = reinterpret_cast<uint2*>(smem + 2 * N);
    uint64_t* bar = reinterpret_cast<uint64_t*>(tf + N);
    const RowTable<LOGN, 0, false, 0> fw{tf};
    const RowTable<LOGN, 0, true, 0> iw{tf};
    if (threadIdx.x == 0) {
        tc::mbar_init(bar, 1);
        tc::fence_mbar_init();
    }
    __syncthreads();
    uint32_t phase = 0;
    for (uint32_t b = blockIdx.x; b < t.total; b += gridDim.x, phase ^= 1) {
        if (b != blockIdx.x) __syncthreads();   // the previous prime's tiles and table
        const uint32_t i = group_locate(t, b);
        const GroupItem& it = t.item[i];
        const size_t j = it.j0 + (b - t.first[i]);
        if (threadIdx.x == 0) {
            tc::mbar_arrive_expect_tx(bar, N * sizeof(uint2));
            tc::bulk_g2s(tf, it.d.row_tw + j * N, N * sizeof(uint2), bar);
        }
        const PrimeConsts pc = it.d.pc[j];
        const uint32_t p = pc.p;
        uint32_t* const X[2] = {it.A + j * N, it.B + j * N};
        {
            const uint32_t base = round_base<LOGN, 0, SWZ, RB, 0>(threadIdx.x);
            uint32_t v[2][E];
#pragma unroll
            for (int o = 0; o < 2; ++o) {
#pragma unroll
                for (int k = 0; k < E; ++k) v[o][k] = X[o][base | (k << sh)];
            }
            if (!tc::wait_parity(bar, phase, it.d.wait_ns) && (threadIdx.x & 31) == 0) atomicOr(it.d.err, 4u);
            fwd_round<LOGN, 0, SWZ, RB, 0, LAZY, 2>(v, base, fw, p);
#pragma unroll
            for (int o = 0; o < 2; ++o) store_round<LOGN, 0, SWZ, RB, 0>(tiles[o], v[o], base);
            __syncthreads();
        }
        fwd_range<LOGN, 0, SWZ, RB, 1, last, LAZY, 2>(tiles, fw, p);
        {
            const uint32_t base = round_base<LOGN, 0, SWZ, RB, last>(threadIdx.x);
            uint32_t v[2][E];
#pragma unroll
            for (int o = 0; o < 2; ++o) load_round<LOGN, 0, SWZ, RB, last>(tiles[o], v[o], base);
            fwd_round<LOGN, 0, SWZ, RB, last, LAZY, 2>(v, base, fw, p);
#pragma unroll
            for (int k = 0; k < E; ++k) v[0][k] = pointwise<LAZY>(v[0][k], v[1][k], pc);
            inv_round<LOGN, 0, SWZ, RB, last, LAZY, true>(v[0], base, iw, p);
            store_round<LOGN, 0, SWZ, RB, last>(tiles[0], v[0], base);
            __syncthreads();
        }
        inv_range<LOGN, 0, SWZ, RB, last - 1, 1, LAZY, true>(tiles[0], iw, p);
        {
            const uint32_t base = round_base<LOGN, 0, SWZ, RB, 0>(threadIdx.x);
            uint32_t v[E];
            load_round<LOGN, 0, SWZ, RB, 0>(tiles[0], v, base);
            inv_round<LOGN, 0, SWZ, RB, 0, LAZY, true>(v, base, iw, p);
            if constexpr (LAZY) {
#pragma unroll
                for (int k = 0; k < E; ++k) v[k] = reduce_once(v[k], p);
            }
#pragma unroll
            for (int k = 0; k < E; ++k) X[0][base | (k << sh)] = v[k];
        }
    }
}

// Round-major tables of the one-CTA transforms from the plan's entry-order ones.
__global__ void __launch_bounds__(256) k_whole_tables(DevPoint d, int rb, uint2* out) {
    const size_t at = static_cast<size_t>(blockIdx.x) * d.N;
    for (uint32_t e = threadIdx.x; e < d.N; e += blockDim.x)
        out[at + (e ? row_table_pos(static_cast<int>(d.logN), rb, e) : 0u)] = e ? d.full_f[at + e] : make_uint2(0, 0);
}

template <bool LAZY>
void launch_cluster(const DevPoint& d, uint32_t* A, uint32_t* B, int sms, cudaStream_t st) {
    auto run = [&](auto ls) {
        using CG = ClusterGeom<decltype(ls)::value>;
        // Started under the decompose's tail, clusters crowd onto the SMs it
        // leaves free and stay there: only if those take them one by one
        // (the decompose runs a CTA per 128 coefficients and operand, up to one
        // an SM).  Product us, early | not: N = 4096 K = 19 11.1 | 12.4, K = 60
        // 19.6 | 16.8, N = 8192 K = 10 17.6 | 14.7, K = 139 32.0 | 29.5, N = 16384
        // K = 10 19.4 | 15.8, K = 36 22.4 | 21.1.
        const uint32_t busy = std::min<uint32_t>(sms, d.N / 64);
        const bool early = CG::kCtas * static_cast<uint32_t>(d.K) <= static_cast<uint32_t>(sms) - busy;
        check(launch_cluster_grid(k_ntt_cluster<decltype(ls)::value, LAZY>, dim3(CG::kCtas, d.K), dim3(CG::T), CG::kCtas,
                                  early, CG::kSmem, st, d, A, B),
              "transform launch");
    };
    switch (d.logS) {
        case 6: run(std::integral_constant<int, 6>{}); break;
        case 7: run(std::integral_constant<int, 7>{}); break;
        case 8: run(std::integral_constant<int, 8>{}); break;
        case 9: run(std::integral_constant<int, 9>{}); break;
        default: throw std::runtime_error("cluster transform: unsupported row length");
    }
}

template <bool LAZY>
void launch_whole(const DevPoint& d, uint32_t* A, uint32_t* B, int mode, int sms, cudaStream_t st) {
    // Early unless the product's decompose fills the SMs (decompose_parts).
    const bool early = decompose_parts(d.N, d.K, (d.N + 127) / 128, 2, sms).parts == 1;
    auto run = [&](auto ln) {
        using WG = WholeGeom<decltype(ln)::value>;
        check(launch_cluster_grid(k_ntt_whole<decltype(ln)::value, LAZY>, dim3(d.K), dim3(2 * WG::T), 1,
                                  early, WG::kSmem, st, d, A, B, mode),
              "transform launch");
    };
    switch (d.logN) {
        case 8: run(std::integral_constant<int, 8>{}); break;
        case 9: run(std::integral_constant<int, 9>{}); break;
        case 10: run(std::integral_constant<int, 10>{}); break;
        case 11: run(std::integral_constant<int, 11>{}); break;
        default: throw std::runtime_error("one-block transform: unsupported length");
    }
}

template <int LOGS, bool LAZY>
void cluster_attrs() {
    auto k = k_ntt_cluster<LOGS, LAZY>;
    check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(ClusterGeom<LOGS>::kSmem)),
          "cluster smem");
    // Sixteen CTAs (S = 512) are past the portable cluster size.
    if (ClusterGeom<LOGS>::kCtas > 8)
        check(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1), "cluster size");
}

// (Also loads the kernel, so that its first launch may be under capture.)
template <int LOGN, bool LAZY>
void whole_attrs() {
    check(cudaFuncSetAttribute(k_ntt_whole<LOGN, LAZY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(WholeGeom<LOGN>::kSmem)),
          "one-block smem");
}

template <bool LAZY>
void whole_group_attrs() {
    check(cudaFuncSetAttribute(k_ntt_whole_group<LAZY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(WholeGeom<11>::kSmem)),
          "one-block smem");
}

template <bool LAZY>
void whole_group(const GroupTable* t, uint32_t grid, cudaStream_t st, int* occupancy) {
    using WG = WholeGeom<11>;
    if (occupancy) {
        check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(occupancy, k_ntt_whole_group<LAZY>, WG::T, WG::kSmem),
              "occupancy");
    } else {
        k_ntt_whole_group<LAZY><<<grid, WG::T, WG::kSmem, st>>>(*t);
    }
}

}  // namespace

void ntt_whole_group(const GroupTable* t, bool lazy, uint32_t grid, cudaStream_t st, int* occupancy) {
    lazy ? whole_group<true>(t, grid, st, occupancy) : whole_group<false>(t, grid, st, occupancy);
}

void ntt_whole_group_init_attributes() {
    whole_group_attrs<true>();
    whole_group_attrs<false>();
}

void ntt_fused_init_attributes() {
    whole_attrs<8, true>();
    whole_attrs<9, true>();
    whole_attrs<10, true>();
    whole_attrs<11, true>();
    whole_attrs<8, false>();
    whole_attrs<9, false>();
    whole_attrs<10, false>();
    whole_attrs<11, false>();
    cluster_attrs<6, true>();
    cluster_attrs<7, true>();
    cluster_attrs<8, true>();
    cluster_attrs<9, true>();
    cluster_attrs<6, false>();
    cluster_attrs<7, false>();
    cluster_attrs<8, false>();
    cluster_attrs<9, false>();
}

void build_whole_tables(const DevPoint& d, uint2* out, cudaStream_t st) {
    k_whole_tables<<<d.K, 256, 0, st>>>(d, whole_pass_rb(static_cast<int>(d.logN)), out);
    check(cudaGetLastError(), "transform tables launch");
}

// Clusters up to four CTAs per SM in all (592 on 148 SMs: N = 4096 and 8192 at
// any K, 16384 up to K = 74, 32768 up to K = 37), the measured crossover.  A
// cluster lies within a group of SMs that share a network, so fewer are
// resident at once than four CTAs an SM would give: 296, 142, 71 and 31 of
// them for N = 4096 .. 32768 (cudaOccupancyMaxActiveClusters).  The last few wait
// for a whole cluster's places, and still the one launch is no slower up to the
// line (product us in a graph, one launch | three, B200):
//   N = 4096   K = 60  15.5 | 21.7   K = 138 23.2 | 30.4
//   N = 8192   K = 60  18.9 | 23.2   K = 130 30.2 | 35.5
//   N = 16384  K = 36  22.1 | 24.6   K = 71  27.7 | 31.7   K = 72  31.1 | 31.4   K = 74  30.6 | 31.2
//   N = 32768  K = 19  22.9 | 25.3   K = 31  26.3 | 30.3   K = 32  29.0 | 30.8   K = 37  31.2 | 31.9
// and past it the separate passes, which hold more warps an SM, win (transform
// alone: N = 16384 K = 139 26.5 | 23.4, N = 32768 K = 60 26.8 | 23.7).
bool ntt_fused_ok(const DevPoint& d, int mode, int sms) {
    if (d.logN >= kWholeMinLogN && d.logN <= 11) return mode == kRowProduct || mode == kRowForward;
    if (mode != kRowProduct || d.logR != 6 || d.logS < 6 || d.logS > 9) return false;
    const int ctas = d.K << (d.logN - 11);
    return ctas <= ClusterGeom<6>::kBlocks * sms;
}

void launch_ntt_fused(const DevPoint& d, uint32_t* A, uint32_t* B, int mode, int sms, cudaStream_t st) {
    if (d.logN <= 11) {
        d.lazy ? launch_whole<true>(d, A, B, mode, sms, st) : launch_whole<false>(d, A, B, mode, sms, st);
    } else {
        d.lazy ? launch_cluster<true>(d, A, B, sms, st) : launch_cluster<false>(d, A, B, sms, st);
    }
}

}  // namespace fpm
