// One-pass flash attention backward on CTA pairs (head dim 128, non-causal, key-length mask): the two CTAs of a cluster own
// 128 keys each and walk the same 128-query chunks with tcgen05.mma.cta_group::2.  Chosen by tt_attn_bwd_fused (attn_bwd_tcgen05.cu), by
// the waves that the two kernels would take; operands, masks and results are those of attn_bwd_fused_kernel there.
//
// Why pairs.  One CTA alone moves 480 KB through its shared memory per chunk (an N = 128 product reads 8 KB in its 64 clocks, so
// the products alone saturate it) and reduces 64 KB of fp32 dQ into L2, which drains at 25 bytes a clock: ~4500 clocks a
// chunk where the tensor cores need 2560.  A pair halves what does not grow with the keys:
//   * the streamed operand of a product is split over the two CTAs (each holds 64 of the 128 queries of S^T = K Q^T and dP^T = V dO^T,
//     and 64 of the 128 columns of dV += P^T dO and dK += dS^T Q), so a product reads 6 or 2 KB a step instead of 8 or 4;
//   * dQ of a chunk is formed once per pair: the CTAs exchange half of their dS through distributed shared memory, CTA r then
//     holds dS [256 keys x queries 64 r .. 64 r + 63] and dQ = dS K is one product of M = 128 over the pair (64 rows a CTA, at the
//     full rate: 32 clocks a step), so each CTA reduces 32 KB instead of 64.
//
// Tensor memory (both CTAs): T1 = [0, 128) S^T, T2 = [128, 256) dP^T then dS^T, [256, 384) dV, [384, 512) dK.  Once every softmax
// warp has read S(c), bf16 P(c) goes to T1's first 64 columns and dQ(c-1) (64 rows of 128 columns: lanes 0 - 63 hold columns
// 0 - 63, lanes 64 - 127 columns 64 - 127) to its last 64.  So dQ waits for nothing but its own operands, and the chain
// dP(c+1) -> dS(c+1) runs beside the exchange.
//
//   tensor core:  dK(c) dP(c+1) | dQ(c) dV(c+1) | S(c+2) ...
//   softmax:      P(c+1) ................ | dS(c+1) ... | P(c+2)        dQ warps:  read out dQ(c), stage it
//
// Shared memory holds exactly one copy of each streamed operand (Q as the operand of S and of dK, dO as that of dP and of dV: four
// tiles of 16 KB), refilled as soon as its product has retired, a whole chunk before it is needed again.
//
// What bounds it (~3300 clocks a chunk; 1000 W under sustained load): two chains of that length, dS stored -> exchange (~1600: bulk copy and
// the hop back to the leader) -> dQ -> next dS stored, and P -> dS in the softmax warps (the exponentials alone take 1024).  So what does
// not have to be on them is kept off: eight warps of their own read dQ out of tensor memory (the softmax warps doing it: 32.6 ms); the
// exchange is a bulk copy from a buffer (stores to the peer's memory from the softmax warps held up every other shared-memory access for
// ~1000 clocks a chunk); statistics come scaled and padded, one ld.shared each.  Registers are split by role (setmaxnreg): spills
// in the MMA or the read-out warps cost up to 10 ms.  24 heads x 32656 tokens: 28.4 ms, 29.0 under sustained load (single CTAs: 32.7 and
// 34.2); 3 heads x 119056: 47.4 (55.8); 24 x 6144: 1.00 (1.15).
//
// Synchronisation (mbarriers, bounded waits): "leader" barriers live in CTA 0, whose MMA thread issues for the pair; commits arrive
// in both CTAs.  The bytes of the exchange complete, at cluster scope, on a barrier of the receiving CTA.  CTA 1's relay thread passes that
// on to the leader, and with it its softmax warps' own half of dS, which they have stored for products that the leader issues: for those
// it fences at cluster scope, while the exchange is under way.  (Released by the arrival itself, behind the exchange: 30.6 ms instead of
// 28.4 at 24 heads x 32656 tokens, 52.3 instead of 47.4 at 3 x 119056; by arrivals of the softmax warps: 14 ms more.)
// utils/pair_pipeline_model.py checks the protocol.
#include "common.cuh"
#include "sm100.cuh"
#include "teletron_b200.h"

namespace {

using namespace sm100;

constexpr int D = 128;
constexpr int BK = 128;                     // keys per CTA
constexpr int BC = 128;                     // queries per chunk
constexpr int kSlab = 128 * 128;            // [128 rows x 64 columns] bf16: 16 KB
constexpr int kHalfSlab = 64 * 128;         // [64 rows x 64 columns] bf16: 8 KB
constexpr int kGroups = 4;                  // softmax warpgroups: 32 queries of every chunk each
constexpr int kThreads = 128 + 128 * kGroups + 256;     // TMA, MMA (CTA 1: relay), exchange, reductions; softmax; dQ read-out
constexpr int kFirstSoftmax = 4, kFirstDrain = kFirstSoftmax + 4 * kGroups;     // warps
// registers per thread: what the compiler launches the block with, then split (the launcher checks it)
constexpr int kRegsLaunch = 72, kRegsMisc = 56, kRegsSoftmax = 88, kRegsDrain = 48;
static_assert(128 * (kRegsMisc + kGroups * kRegsSoftmax + 2 * kRegsDrain) <= kThreads * kRegsLaunch, "register split");
constexpr int kStageFloats = 64 * 64;       // half of the dQ of one chunk and CTA
constexpr int kStatBytes = 2 * BC * 4;      // lse and delta of one chunk
// byte offsets in shared memory
constexpr int oK = 0;                       // K, own keys: two slabs (A of S, K-major)
constexpr int oV = 2 * kSlab;               // V, own keys (A of dP)
constexpr int oKB = 4 * kSlab;              // K, the pair's 256 keys, 64 columns (B of dQ, MN-major)
constexpr int oQs = 6 * kSlab;              // Q, 64 queries x 128 (B of S, K-major)
constexpr int oDOp = 7 * kSlab;             // dO, 64 queries x 128 (B of dP)
constexpr int oDOv = 8 * kSlab;             // dO, 128 queries x 64 columns (B of dV, MN-major)
constexpr int oQk = 9 * kSlab;              // Q, 128 queries x 64 columns (B of dK)
constexpr int oDS = 10 * kSlab;             // dS, the pair's 256 keys x 64 queries (A of dQ, MN-major)
constexpr int oStage = 12 * kSlab;          // half of a chunk's dQ on its way out, fp32
constexpr int oOut = 13 * kSlab;            // the dS of the peer's queries on its way there
constexpr int oBars = 14 * kSlab;
constexpr int oStat = oBars + 256;          // two slots
constexpr int kSmemBytes = oStat + 2 * kStatBytes;
static_assert(kSmemBytes <= 232448, "shared memory of one CTA");
constexpr float kLog2e = 1.4426950408889634f;

struct PairParams {
    __nv_bfloat16* dv;
    __nv_bfloat16* dk;
    const float* stats;     // [BH, chunks, 2, 128]: -lse * log2(e), then -delta; -inf and 0 for queries at and beyond S
    float* dq_acc;          // [BH, s_pad, 128] fp32, zeroed
    int S, kv_len, H;
    int mask_lo, mask_hi;
    int s_pad;
    float scale;
    int* status;
};

__device__ __forceinline__ void bulk_reduce_add(float* dst, uint32_t smem_src, uint32_t bytes) {
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst), "r"(smem_src), "r"(bytes)
                 : "memory");
}

template <int N>
__device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// column of T1 where group g's 32 bf16 pairs of P begin: its own first 16 columns for groups 0 and 1, the second 16 of those for
// groups 2 and 3, which therefore wait until groups 0 and 1 have read their scores
__device__ __forceinline__ constexpr int p_col(int g) { return (g & 1) * 32 + (g >> 1) * 16; }

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
attn_bwd_pair_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO, const PairParams p) {
    extern __shared__ __align__(1024) uint8_t pair_smem[];
    volatile int& abort_flag = *reinterpret_cast<volatile int*>(pair_smem + oBars + 248);
    uint32_t& tmem_base_slot = *reinterpret_cast<uint32_t*>(pair_smem + oBars + 252);
    uint32_t base = smem_u32(pair_smem);
    if ((base & 1023u) != 0) {               // both CTAs of a pair see the same offset
        if (threadIdx.x == 0) atomicExch(p.status, TT_ERR_ARG);
        return;
    }
    enum : int {
        // in the leader
        kvFull, qsFull, qkFull, dopFull, dovFull,
        sRead,                   // S(c) is in registers everywhere: T1 takes P(c) and dQ(c-1)
        pReady, dsReady, dqRead,
        exPeer,                  // CTA 1's dS tile is complete, both halves
        // in both CTAs, reached by commits
        qsEmpty, qkEmpty, dopEmpty, dovEmpty, sFull, dpFull, dqFull, accFinal,
        // each CTA's own
        dsOwn,                   // its own half of dS(c) is in the dS tile
        exIn,                    // the peer's half of dS has arrived in the dS tile
        exStaged,                // the peer's half of dS(c) is complete in oOut
        staged, stageFree,       // [2]: that half of dQ(c) has left the staging buffer
        stFull = stageFree + 2,  // [2]
        quadRead = stFull + 2,   // [4]: groups 0, 1 of this quadrant have read their scores
        nBars = quadRead + 4
    };
    static_assert(8 * nBars <= 248, "barriers");
    auto bar = [&](int i) { return base + (uint32_t)(oBars + 8 * i); };

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int bh = blockIdx.y;
    const int r0 = blockIdx.x * BK;                  // first key of this CTA (at and beyond S in the last pair of an odd count)
    const int pair0 = (int)(blockIdx.x >> 1) * 2 * BK;
    const int n_chunks = (p.S + BC - 1) / BC;
    // pairs of a head start at different chunks, so their reductions land on different rows of the accumulator
    const int c0 = (int)(blockIdx.x >> 1) % n_chunks;
    auto chunk_of = [&](int c) { const int e = c + c0; return e >= n_chunks ? e - n_chunks : e; };

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int i = 0; i < nBars; ++i) {
            int count = 1;
            if (i == sRead || i == pReady || i == dsReady) count = 2 * 4 * kGroups;      // every softmax warp of both CTAs
            if (i == dqRead) count = 2 * 8;
            if (i == dsOwn || i == exStaged) count = 2 * kGroups;
            if (i == staged) count = 4;
            if (i >= quadRead) count = 2;
            mbar_init(bar(i), (uint32_t)count);
        }
        fence_barrier_init();
        fence_proxy_async();
    }
    if (warp == 1) {
        tmem_alloc2(smem_u32(&tmem_base_slot), 512);
        tmem_relinquish2();
    }
    tc_fence_before();
    __syncthreads();
    cluster_arrive();
    cluster_wait();
    tc_fence_after();
    const uint32_t tmem = tmem_base_slot;
    constexpr uint32_t kT1 = 0, kDQ = 64, kT2 = 128, kAccV = 256, kAccK = 384;
    // barrier addresses are computed anew from here on: kept from the initialisation they would be spilled
    asm volatile("mov.u32 %0, %0;" : "+r"(base));
    // The split stands inside the branches that the roles share: ahead of them, where the paths meet again, the compiler holds every role
    // to the smallest share and spills (24 heads x 32656 tokens: 28.7 -> 28.3 ms).
    if (warp < kFirstSoftmax) {
    reg_dec<kRegsMisc>();
    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer (one per CTA: its halves)
        if (elect_one()) {
            const int b = bh / p.H, head = bh - b * p.H;
            const int d0 = (int)rank * 64;           // this CTA's columns of dV, dK, dQ
            const int qh = (int)rank * 64;           // and its queries of S, dP
            if (rank == 0) mbar_arrive_expect_tx(bar(kvFull), 2 * 6 * kSlab);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                tma_load_3d_pair(base + oK + h * kSlab, &tmK, bar(kvFull), h * 64, r0, bh);
                tma_load_3d_pair(base + oV + h * kSlab, &tmV, bar(kvFull), h * 64, r0, bh);
                tma_load_3d_pair(base + oKB + h * kSlab, &tmK, bar(kvFull), d0, pair0 + h * BK, bh);
            }
            auto load_stats = [&](int c) {
                mbar_arrive_expect_tx(bar(stFull + (c & 1)), kStatBytes);
                bulk_load_1d(base + oStat + (uint32_t)(c & 1) * kStatBytes, p.stats + ((long)bh * p.s_pad + chunk_of(c) * BC) * 2, kStatBytes,
                             bar(stFull + (c & 1)));
            };
            auto load_qk = [&](int c) {
                if (rank == 0) mbar_arrive_expect_tx(bar(qkFull), 2 * kSlab);
#pragma unroll
                for (int h = 0; h < 2; ++h) tma_load_3d_pair(base + oQk + h * kHalfSlab, &tmQ, bar(qkFull), d0, chunk_of(c) * BC + h * 64, bh);
            };
            load_stats(0);
            if (n_chunks > 1) load_stats(1);
            for (int c = 0; c <= n_chunks; ++c) {
                const uint32_t wpar = ((uint32_t)c & 1u) ^ 1u;       // the product of chunk c - 1 has retired
                if (c < n_chunks) {
                    if (!mbar_wait(bar(qsEmpty), wpar, &abort_flag)) goto done;
                    if (rank == 0) mbar_arrive_expect_tx(bar(qsFull), 2 * kSlab);
#pragma unroll
                    for (int h = 0; h < 2; ++h) tma_load_3d_pair(base + oQs + h * kHalfSlab, &tmQ, bar(qsFull), h * 64, chunk_of(c) * BC + qh, bh);
                }
                if (c > 0) {                                         // Q for dK(c - 1), after dK(c - 2)
                    if (!mbar_wait(bar(qkEmpty), wpar ^ 1u, &abort_flag)) goto done;
                    load_qk(c - 1);
                    // every warp has read the statistics of chunk c - 2 before dK(c - 2) was issued
                    if (c >= 2 && c < n_chunks) load_stats(c);
                }
                if (c < n_chunks) {
                    if (!mbar_wait(bar(dopEmpty), wpar, &abort_flag)) goto done;
                    if (rank == 0) mbar_arrive_expect_tx(bar(dopFull), 2 * kSlab);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        tma_load_4d_pair(base + oDOp + h * kHalfSlab, &tmDO, bar(dopFull), h * 64, head, chunk_of(c) * BC + qh, b);
                    if (!mbar_wait(bar(dovEmpty), wpar, &abort_flag)) goto done;
                    if (rank == 0) mbar_arrive_expect_tx(bar(dovFull), 2 * kSlab);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        tma_load_4d_pair(base + oDOv + h * kHalfSlab, &tmDO, bar(dovFull), d0, head, chunk_of(c) * BC + h * 64, b);
                }
            }
        }
    } else if (warp == 1 && rank == 1) {
        // ------------------------------------------------------------ relay: the dS tile of this CTA is complete
        if (elect_one()) {
            for (int c = 0; c < n_chunks; ++c) {
                mbar_arrive_expect_tx(bar(exIn), kSlab);
                if (!mbar_wait(bar(dsOwn), (uint32_t)c & 1u, &abort_flag)) goto done;
                fence_cluster();
                if (!mbar_wait(bar(exIn), (uint32_t)c & 1u, &abort_flag)) goto done;
                mbar_arrive_leader_relaxed(bar(exPeer));
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (leader)
        if (elect_one()) {
            constexpr uint32_t idesc_t = idesc_bf16(2 * BK, BC, false, false);   // T = A B^T, both K-major
            constexpr uint32_t idesc_a = idesc_bf16(2 * BK, D, false, true);     // acc += (tensor-memory A) B, B MN-major
            constexpr uint32_t idesc_q = idesc_bf16(BC, D, true, true);          // dQ = dS K: both operands MN-major
            // with all ~100 descriptors hoisted out of the chunk loop they are spilled, and every issue waits for loads
            auto issue_t = [&](uint32_t t_col, int oa, int ob) {
                const uint64_t da = fresh_desc(smem_desc_sw128(base + oa, 16, 1024)), db = fresh_desc(smem_desc_sw128(base + ob, 16, 1024));
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk)
                    umma2_bf16_ss(tmem + t_col, da + (uint64_t)(((kk >> 2) * kSlab + (kk & 3) * 32) >> 4),
                                  db + (uint64_t)(((kk >> 2) * kHalfSlab + (kk & 3) * 32) >> 4), idesc_t, kk ? 1u : 0u);
            };
            auto issue_s = [&](int c) -> bool {
                if (!mbar_wait(bar(qsFull), (uint32_t)c & 1u, &abort_flag)) return false;
                tc_fence_after();
                issue_t(kT1, oK, oQs);
                umma2_commit_both(bar(sFull));
                umma2_commit_both(bar(qsEmpty));
                return true;
            };
            auto issue_dp = [&](int c) -> bool {
                if (!mbar_wait(bar(dopFull), (uint32_t)c & 1u, &abort_flag)) return false;
                tc_fence_after();
                issue_t(kT2, oV, oDOp);
                umma2_commit_both(bar(dpFull));
                umma2_commit_both(bar(dopEmpty));
                return true;
            };
            auto issue_dv = [&](int c) -> bool {
                if (!mbar_wait(bar(dovFull), (uint32_t)c & 1u, &abort_flag)) return false;
                if (!mbar_wait(bar(pReady), (uint32_t)c & 1u, &abort_flag)) return false;
                tc_fence_after();
                const uint64_t db = fresh_desc(smem_desc_sw128(base + oDOv, kSlab, 1024));
#pragma unroll
                for (int kk = 0; kk < BC / 16; ++kk)
                    umma2_bf16_ts(tmem + kAccV, tmem + kT1 + p_col(kk >> 1) + (kk & 1) * 8, db + (uint64_t)(kk * (2048 >> 4)),
                                  idesc_a, (c == 0 && kk == 0) ? 0u : 1u);
                umma2_commit_both(bar(dovEmpty));
                return true;
            };
            if (!mbar_wait(bar(kvFull), 0, &abort_flag)) goto done;
            if (!issue_s(0) || !issue_dp(0) || !issue_dv(0)) goto done;
            if (n_chunks > 1 && !issue_s(1)) goto done;
            for (int c = 0; c < n_chunks; ++c) {
                const uint32_t par = (uint32_t)c & 1u;
                const bool more = c + 1 < n_chunks;
                mbar_arrive_expect_tx(bar(exIn), kSlab);
                if (!mbar_wait(bar(qkFull), par, &abort_flag)) goto done;
                if (!mbar_wait(bar(dsReady), par, &abort_flag)) goto done;      // dS(c) in T2
                tc_fence_after();
                const uint64_t dqk = fresh_desc(smem_desc_sw128(base + oQk, kSlab, 1024));
#pragma unroll
                for (int kk = 0; kk < BC / 16; ++kk)                                // dK += dS^T Q
                    umma2_bf16_ts(tmem + kAccK, tmem + kT2 + (kk >> 1) * 32 + (kk & 1) * 8, dqk + (uint64_t)(kk * (2048 >> 4)),
                                  idesc_a, (c == 0 && kk == 0) ? 0u : 1u);
                umma2_commit_both(bar(qkEmpty));
                if (more && !issue_dp(c + 1)) goto done;                            // T2: dK(c) has read dS before (issue order)
                // T1's last columns: S(c+1) has been read (and dQ(c-1) before it was issued); behind the last chunk only dQ(c-1) is left
                if (more && !mbar_wait(bar(sRead), par ^ 1u, &abort_flag)) goto done;
                if (!more && c > 0 && !mbar_wait(bar(dqRead), par ^ 1u, &abort_flag)) goto done;
                if (!mbar_wait(bar(dsOwn), par, &abort_flag)) goto done;        // dS(c) in the dS tile here: own half
                if (!mbar_wait(bar(exIn), par, &abort_flag)) goto done;         // and the other one
                if (!mbar_wait<true>(bar(exPeer), par, &abort_flag)) goto done; // and both in CTA 1
                tc_fence_after();
                const uint64_t dds = fresh_desc(smem_desc_sw128(base + oDS, kSlab, 1024)), dkb = fresh_desc(smem_desc_sw128(base + oKB, kSlab, 1024));
#pragma unroll
                for (int kk = 0; kk < 2 * BK / 16; ++kk)                            // dQ(c) = dS K over the pair's 256 keys
                    umma2_bf16_ss(tmem + kDQ, dds + (uint64_t)(kk * (2048 >> 4)), dkb + (uint64_t)(kk * (2048 >> 4)), idesc_q, kk ? 1u : 0u);
                umma2_commit_both(bar(dqFull));
                if (more && !issue_dv(c + 1)) goto done;
                if (c + 2 < n_chunks) {                                             // T1: P(c+1) consumed (issue order), dQ(c) read out
                    if (!mbar_wait(bar(dqRead), par, &abort_flag)) goto done;
                    if (!issue_s(c + 2)) goto done;
                }
            }
            umma2_commit_both(bar(accFinal));
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------ exchange: half of dS(c) into the peer's dS tile
        if (elect_one()) {
            const uint32_t dst = mapa(base + oDS, rank ^ 1u) + rank * (uint32_t)kSlab, dst_bar = mapa(bar(exIn), rank ^ 1u);
            for (int c = 0; c < n_chunks; ++c) {
                if (!mbar_wait(bar(exStaged), (uint32_t)c & 1u, &abort_flag)) goto done;
                bulk_copy_to_cta(dst, base + oOut, kSlab, dst_bar);
            }
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------ dQ reductions
        if (elect_one()) {
            for (int i = 0; i < 2 * n_chunks; ++i) {
                if (!mbar_wait(bar(staged), (uint32_t)i & 1u, &abort_flag)) goto done;
                bulk_reduce_add(p.dq_acc + ((long)bh * p.s_pad + chunk_of(i >> 1) * BC) * D + (rank * 2 + (i & 1)) * kStageFloats, base + oStage,
                                kStageFloats * 4);
                bulk_commit();
                bulk_wait_read<0>();
                mbar_arrive(bar(stageFree + (i & 1)));
            }
            bulk_wait_all();
        }
    }
    } else if (warp >= kFirstDrain) {
        reg_dec<kRegsDrain>();
        // ------------------------------------------------------------ dQ read-out: two halves of 32 columns through one buffer
        // lane l of the CTA holds query 64 rank + l % 64, columns 64 (l / 64) + 0 .. 63
        const int quad = warp & 3, half = (warp - kFirstDrain) >> 2;
        const uint32_t tq = tmem + ((uint32_t)(quad * 32) << 16) + kDQ + half * 32;
        const uint32_t stage = base + oStage + ((uint32_t)quad << 12) + (uint32_t)lane * 128u + (((uint32_t)lane & 7u) << 4);
        for (int c = 0; c < n_chunks; ++c) {
            if (!mbar_wait(bar(dqFull), (uint32_t)c & 1u, &abort_flag)) goto done;
            tc_fence_after();
            uint32_t r[32];
            tmem_ld_32x32(tq, r);
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(bar(dqRead));
            // the half before this one has left the buffer
            if ((c > 0 || half > 0) && !mbar_wait(bar(stageFree + (half ^ 1)), (uint32_t)(half ? c : c - 1) & 1u, &abort_flag)) goto done;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage ^ (uint32_t)(j << 4)), "r"(r[4 * j]),
                             "r"(r[4 * j + 1]), "r"(r[4 * j + 2]), "r"(r[4 * j + 3])
                             : "memory");
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(staged));
        }
    } else {
        reg_inc<kRegsSoftmax>();
        // ------------------------------------------------------------ softmax / dS
        const int part = (warp - kFirstSoftmax) >> 2;                  // queries [32 part, 32 part + 32) of every chunk
        const int quad = warp & 3;
        const int srow = quad * 32 + lane;                 // key row within the CTA's tile
        const int row = r0 + srow;
        const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
        const float c_log2 = p.scale * kLog2e;
        const uint32_t live_mask = row < p.kv_len && !(row >= p.mask_lo && row < p.mask_hi) ? 0xffffffffu : 0u;
        const uint32_t t1 = tmem + lane_sel + kT1 + part * 32, t2 = tmem + lane_sel + kT2 + part * 32;
        const uint32_t tp = tmem + lane_sel + kT1 + p_col(part);
        // dS row of this key: queries of this CTA go to its own dS tile (keys of both CTAs), those of the peer to the outgoing buffer;
        // 16-byte pieces 4 (part & 1) + 0 .. 3 of the row's 128 bytes, swizzled
        const bool mine = (uint32_t)(part >> 1) == rank;
        const uint32_t ds_row = base + (mine ? oDS + rank * (uint32_t)kSlab : (uint32_t)oOut) + (uint32_t)srow * 128u +
                                ((((uint32_t)(part & 1) << 2) ^ ((uint32_t)srow & 7u)) << 4);      // piece 0; piece j differs by j << 4
        const uint32_t stat = base + oStat + (uint32_t)part * 128u;
        uint32_t pk[16];

        // statistics of this thread's 32 queries of chunk c, four at a time
        auto stat4 = [&](int c, int which, int i) {
            float4 v;
            const uint32_t a = stat + (uint32_t)(c & 1) * kStatBytes + (uint32_t)(which * BC + i * 4) * 4u;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
            return v;
        };
        for (int c = 0; c < n_chunks; ++c) {
            const uint32_t par = (uint32_t)c & 1u;
            // ---- P(c)
            if (!mbar_wait(bar(stFull + (c & 1)), (uint32_t)(c >> 1) & 1u, &abort_flag)) goto done;
            if (!mbar_wait(bar(sFull), par, &abort_flag)) goto done;
            tc_fence_after();
            {
                uint32_t a[32];
                tmem_ld_32x32(t1, a);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (part < 2) mbar_arrive(bar(quadRead + quad));
                    mbar_arrive_leader(bar(sRead));
                }
                float4 lv;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    if ((i & 1) == 0) lv = stat4(c, 0, i >> 1);
                    const float2 nl2 = (i & 1) ? make_float2(lv.z, lv.w) : make_float2(lv.x, lv.y);
                    const float2 x = __ffma2_rn(make_float2(__uint_as_float(a[2 * i]), __uint_as_float(a[2 * i + 1])),
                                                make_float2(c_log2, c_log2), nl2);
                    const __nv_bfloat162 pb = __floats2bfloat162_rn(exp2f(x.x), exp2f(x.y));
                    pk[i] = *reinterpret_cast<const uint32_t*>(&pb) & live_mask;     // masked keys: 0, whatever their score
                }
            }
            if (part >= 2) {
                if (!mbar_wait(bar(quadRead + quad), par, &abort_flag)) goto done;
                tc_fence_after();
            }
            tmem_st_32x16(tp, pk);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(bar(pReady));
            // ---- dS(c) from dP(c) and the P kept in registers
            if (!mbar_wait(bar(dpFull), par, &abort_flag)) goto done;
            tc_fence_after();
            {
                uint32_t dk[16];
#pragma unroll
                for (int h = 0; h < 2; ++h) {              // 16 columns at a time: fewer registers
                    uint32_t g[16];
                    tmem_ld_32x16(t2 + h * 16, g);
                    tmem_ld_wait();
                    float4 dv;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int i = h * 8 + k;
                        if ((i & 1) == 0) dv = stat4(c, 1, i >> 1);
                        const float2 d2 = (i & 1) ? make_float2(dv.z, dv.w) : make_float2(dv.x, dv.y);
                        const float2 pr = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&pk[i]));
                        const float2 dp = __fadd2_rn(d2, make_float2(__uint_as_float(g[2 * k]), __uint_as_float(g[2 * k + 1])));
                        const float2 ds = __fmul2_rn(pr, dp);
                        const __nv_bfloat162 db = __floats2bfloat162_rn(ds.x, ds.y);
                        dk[i] = *reinterpret_cast<const uint32_t*>(&db);
                    }
                }
                tmem_st_32x16(t2, dk);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_leader(bar(dsReady));
                // dQ(c - 1) is complete: the dS tiles of both CTAs, and the outgoing buffers, take dS(c)
                if (c > 0 && !mbar_wait(bar(dqFull), par ^ 1u, &abort_flag)) goto done;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(ds_row ^ (uint32_t)(j << 4)), "r"(dk[4 * j]),
                                 "r"(dk[4 * j + 1]), "r"(dk[4 * j + 2]), "r"(dk[4 * j + 3])
                                 : "memory");
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(bar(mine ? dsOwn : exStaged));
                }
            }
        }
        // ------------------------------------------------------------ epilogue: dV (unscaled), dK (x softmax scale)
        if (!mbar_wait(bar(accFinal), 0, &abort_flag)) goto done;
        tc_fence_after();
        const bool store = row < p.S;
        const long orow = ((long)bh * p.S + row) * D;
#pragma unroll 1
        for (int which = 0; which < 2; ++which) {
            __nv_bfloat16* dst = (which == 0 ? p.dv : p.dk) + orow;
            const float mul = which == 0 ? 1.f : p.scale;
            uint32_t r[32];
            tmem_ld_32x32(tmem + lane_sel + kAccV + which * 128 + part * 32, r);
            tmem_ld_wait();
            if (store) {
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    float o[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) o[i] = __uint_as_float(r[g * 8 + i]) * mul;
                    tt::st8(dst + part * 32 + g * 8, tt::pack8(o));
                }
            }
        }
    }

done:
    tc_fence_before();
    __syncthreads();
    if (abort_flag) {
        if (threadIdx.x == 0) atomicExch(p.status, TT_ERR_TIMEOUT);
        for (int i = 0; i < 200; ++i) __nanosleep(1000);        // let copies in flight land
    }
    // both CTAs are done with each other's shared and tensor memory before either frees it
    cluster_arrive();
    cluster_wait();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc2(tmem, 512);
    }
}

// dq[bh, s, :] = bf16(scale * acc[bh, s, :]); eight elements per thread.  The accumulator of a 128-query chunk is the byte image of
// the two CTAs' staging buffers: [query / 64][column / 32 % 2][lane of the CTA] rows of 32 floats whose 16-byte pieces are XOR-swizzled.
__global__ void __launch_bounds__(256) dq_pair_finish_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, long BH, int S,
                                                             int s_pad, float scale) {
    const long n8 = BH * S * (D / 8);
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (long)gridDim.x * blockDim.x) {
        const long rowi = i / (D / 8);
        const int c8 = (int)(i - rowi * (D / 8));
        const long bhi = rowi / S, s = rowi - bhi * S;
        const int r = (int)(s & (BC - 1)), l = (c8 >> 3) * 64 + (r & 63), j = (c8 & 3) * 2;
        const float4* src = reinterpret_cast<const float4*>(acc + (bhi * s_pad + s - r) * D + ((r >> 6) * 2 + ((c8 >> 2) & 1)) * kStageFloats + l * 32);
        const int x = l & 7;
        const float4 a = __ldg(src + (j ^ x)), e = __ldg(src + ((j + 1) ^ x));
        float o[8] = {a.x * scale, a.y * scale, a.z * scale, a.w * scale, e.x * scale, e.y * scale, e.z * scale, e.w * scale};
        tt::st8(dq + rowi * D + c8 * 8, tt::pack8(o));
    }
}

}  // namespace

// The pair kernel and the pass that scales and rounds dQ; arguments have been checked and stats / dq_acc prepared by tt_attn_bwd_fused.
int tt_attn_bwd_pair(const void* q, const void* k, const void* v, const void* dout, const float* stats, float* dq_acc, void* dq, void* dk,
                     void* dv, int B, int H, int S, int kv_len, int mask_lo, int mask_hi, float scale, int* status, cudaStream_t st) {
    const uint64_t BH = (uint64_t)B * H;
    const int s_pad = (S + BC - 1) / BC * BC;
    CUtensorMap tq, tk, tv, tdo;
    int rc;
    if ((rc = tt_make_tmap_3d(&tq, q, BH, (uint64_t)S, D, D, (uint64_t)S * D, 64, 64)) != TT_OK) return rc;
    if ((rc = tt_make_tmap_3d(&tk, k, BH, (uint64_t)S, D, D, (uint64_t)S * D, BK, 64)) != TT_OK) return rc;
    if ((rc = tt_make_tmap_3d(&tv, v, BH, (uint64_t)S, D, D, (uint64_t)S * D, BK, 64)) != TT_OK) return rc;
    if ((rc = tt_make_tmap_bshd(&tdo, dout, (uint64_t)B, (uint64_t)S, (uint64_t)H, 64)) != TT_OK) return rc;
    static bool configured[64] = {false};
    const int dev = tt_device().dev;
    if (!configured[dev]) {
        // setmaxnreg.inc waits, without a bound, for registers that the block was launched with
        cudaFuncAttributes at;
        cudaError_t e = cudaFuncGetAttributes(&at, attn_bwd_pair_kernel);
        if (e != cudaSuccess) return tt_record_cuda(e);
        if (at.numRegs < kRegsLaunch) return TT_ERR_LIMIT;
        e = cudaFuncSetAttribute(attn_bwd_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (e != cudaSuccess) return tt_record_cuda(e);
        configured[dev] = true;
    }
    PairParams p;
    p.dv = (__nv_bfloat16*)dv;
    p.dk = (__nv_bfloat16*)dk;
    p.stats = stats;
    p.dq_acc = dq_acc;
    p.S = S;
    p.kv_len = kv_len;
    p.H = H;
    p.mask_lo = mask_lo;
    p.mask_hi = mask_lo < mask_hi ? mask_hi : mask_lo;
    p.s_pad = s_pad;
    p.scale = scale;
    p.status = status;
    const unsigned pairs = (unsigned)((S + 2 * BK - 1) / (2 * BK));
    attn_bwd_pair_kernel<<<dim3(2 * pairs, (unsigned)BH), kThreads, kSmemBytes, st>>>(tq, tk, tv, tdo, p);
    TT_CHECK_LAUNCH();
    const long n8 = (long)BH * S * (D / 8);
    const long blocks = (n8 + 255) / 256;
    dq_pair_finish_kernel<<<(int)(blocks < 148L * 16 ? blocks : 148L * 16), 256, 0, st>>>(dq_acc, (__nv_bfloat16*)dq, (long)BH, S, s_pad, scale);
    TT_CHECK_LAUNCH();
    return TT_OK;
}
