// bf16 GEMM on CTA pairs: two CTAs of a thread-block cluster share one 256 x 256 x 64 tile and one
// tcgen05.mma.cta_group::2 instruction stream.  CTA r of the pair loads rows [128 r, 128 r + 128) of the A tile and
// rows [128 r, 128 r + 128) of the B tile (its half of N) into its own shared memory, with its own non-multicast TMA
// loads; the leader CTA (rank 0) issues every MMA, which reads both CTAs' shared memory and writes each CTA's half of
// the accumulator (128 rows x 256 fp32 columns, double buffered) into that CTA's tensor memory.  Per CTA and k-block
// 32 KB come through L2 instead of the 48 KB of the single-CTA 128 x 256 tile: the short-K products of the model
// (K = 3072: QKV, fc1, projections), which sit at the L2 / epilogue limit with the single-CTA kernel, gain the most.
//
// Synchronisation (all mbarrier waits bounded, sm100.cuh):
//   full[s]   in the leader: armed by the leader's producer with the bytes of BOTH CTAs; each CTA's TMA loads complete
//             on it (the .cta_group::2 form of the load addresses the leader's barrier);
//   empty[s]  in each CTA: the leader's tcgen05.commit multicasts the "stage consumed" arrival to both;
//   tfull[b]  in each CTA: commit multicast when an accumulator buffer is complete;
//   tempty[b] in the leader: the four epilogue warps of both CTAs arrive (8 arrivals) once a buffer has been drained.
// Tensor memory is allocated and freed by warp 1 of both CTAs (cta_group::2), the free after a cluster barrier.
//
// Split-K (tt_gemm2_bf16_splitk): a product with few tiles and a long K leaves most pairs idle, so the k-blocks of a tile are
// shared by `splits` pairs; each writes its fp32 accumulator to its own slice of a scratch buffer (EPI 7) and a second kernel
// adds the slices in a fixed order and applies the epilogue.
//
// Two A operands (tt_gemm2_bf16_two): [a | a2] B^T with the K columns from k1 on taken from a second tensor, so that the
// single-stream block's [attention | MLP] never has to be concatenated.
//
// Layouts and epilogues are those of gemm_tcgen05.cu (nt / nn / tn; bias, GELU erf / tanh with pre-activation,
// GELU backward), and one more for weight gradients: epilogue 5 (tn) adds the bf16 tile to what C holds, in the TMA unit
// (cp.reduce.async.bulk.tensor), so that a gradient buffer takes a product without a temporary and a pass that adds it.  In the reference these products are TransformerEngine -> cuBLASLt calls
// (teletron/models/dit/dit_attention.py:65-104, dit_layerspec.py:266-298, 438-445).
#include "common.cuh"
#include "sm100.cuh"
#include "teletron_b200.h"

#include <string.h>

namespace {

using namespace sm100;

constexpr int BMH = 128;            // rows of A per CTA (half of the pair's 256)
constexpr int BNH = 128;            // rows of B (columns of C) loaded per CTA (half of the pair's 256)
constexpr int BN = 256;             // columns of the accumulator
constexpr int BK = 64;
constexpr int kStages = 6;
constexpr int kABytes = BMH * BK * 2;
constexpr int kBBytes = BNH * BK * 2;
constexpr int kStageBytes = kABytes + kBBytes;          // 32 KB per CTA
constexpr int kThreads = 192;
constexpr int kGroupM = 8;
constexpr int kEpiBytes = 4 * 8192;                      // two 32 x 64 boxes per epilogue warp
constexpr int kSmemBytes = kStages * kStageBytes + kEpiBytes + 1024 + 256;

struct Params2 {
    int M, N, K;
    long ldc;                   // of aux, which the epilogues 3 / 4 read directly
    const __nv_bfloat16* bias;
    __nv_bfloat16* aux;
    int* status;
    int tiles_m, tiles_n;       // in 256 x 256 tiles
    int splits, kb_split;       // k-block ranges per tile, and their length
    int k1;                     // K columns >= k1 come from the second A tensor (a multiple of BK, or >= K: there is none)
    int part_rows;              // rows of one split's slice of the scratch buffer (M rounded up to whole 32-row boxes)
};

template <int EPI>
__device__ __forceinline__ float epi2(float acc, float b, float u) {
    if (EPI == 0 || EPI == 5) return acc + b;
    if (EPI == 1) return tt::gelu_erf(acc + b);
    if (EPI == 2) return tt::gelu_tanh(acc + b);
    if (EPI == 3) return acc * tt::gelu_erf_grad(u);
    return acc * tt::gelu_tanh_grad(u);
}

template <bool A_MN, bool B_MN, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
gemm2_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC,
             const __grid_constant__ CUtensorMap tmAux, const __grid_constant__ CUtensorMap tmA2, const Params2 p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ volatile int abort_flag;
    __shared__ uint32_t tmem_base_slot;

    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t epi_stage = base + kStages * kStageBytes;
    const uint32_t bar_base = epi_stage + kEpiBytes;
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (kStages + s); };
    auto tfull_bar = [&](int b) { return bar_base + 8u * (2 * kStages + b); };
    auto tempty_bar = [&](int b) { return bar_base + 8u * (2 * kStages + 2 + b); };

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();            // 0 = leader
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(tfull_bar(b), 1);
            mbar_init(tempty_bar(b), 8);                  // four epilogue warps of each CTA
        }
        fence_barrier_init();
        fence_proxy_async();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
    }
    if (warp == 1) {
        tmem_alloc2(smem_u32(&tmem_base_slot), 512);
        tmem_relinquish2();
    }
    tc_fence_before();
    __syncthreads();
    // nobody may signal the other CTA's barriers before they exist
    cluster_arrive();
    cluster_wait();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;

    const int num_tiles = p.tiles_m * p.tiles_n * p.splits;       // units of work: (tile, k-block range)
    const int kblocks = (p.K + BK - 1) / BK;
    auto k_first = [&](int u) { return (u % p.splits) * p.kb_split; };
    auto k_end = [&](int u) { return min(kblocks, (u % p.splits + 1) * p.kb_split); };
    auto tile_coords = [&](int u, int& m0, int& n0) {
        const int t = u / p.splits;
        const int per_group = kGroupM * p.tiles_n;
        const int g = t / per_group;
        const int first_m = g * kGroupM;
        const int gm = min(kGroupM, p.tiles_m - first_m);
        const int r = t - g * per_group;
        m0 = (first_m + r % gm) * 256;
        n0 = (r / gm) * 256;
    };

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer (one per CTA: its halves of A and B)
        if (elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            for (int t = pair; t < num_tiles; t += n_pairs) {
                int m0, n0;
                tile_coords(t, m0, n0);
                const int am = m0 + (int)rank * BMH, bn = n0 + (int)rank * BNH;
                const int kb1 = k_end(t);
                for (int kb = k_first(t); kb < kb1; ++kb) {
                    if (!mbar_wait(empty_bar(stage), phase ^ 1u, &abort_flag)) goto done;
                    const uint32_t sa = base + stage * kStageBytes;
                    const uint32_t sb = sa + kABytes;
                    if (rank == 0) mbar_arrive_expect_tx(full_bar(stage), 2 * kStageBytes);      // both CTAs' bytes
                    const int k0 = kb * BK;
                    if (!A_MN) {
                        const bool second = k0 >= p.k1;
                        tma_load_2d_pair(sa, second ? &tmA2 : &tmA, full_bar(stage), second ? k0 - p.k1 : k0, am);
                    } else {
#pragma unroll
                        for (int j = 0; j < BMH / 64; ++j) tma_load_2d_pair(sa + j * 8192, &tmA, full_bar(stage), am + 64 * j, k0);
                    }
                    if (!B_MN) {
                        tma_load_2d_pair(sb, &tmB, full_bar(stage), k0, bn);
                    } else {
#pragma unroll
                        for (int j = 0; j < BNH / 64; ++j) tma_load_2d_pair(sb + j * 8192, &tmB, full_bar(stage), bn + 64 * j, k0);
                    }
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (leader CTA only)
        if (rank == 0 && elect_one()) {
            constexpr uint32_t idesc = idesc_bf16(256, BN, A_MN, B_MN);
            int stage = 0;
            uint32_t phase = 0;
            int it = 0;
            for (int t = pair; t < num_tiles; t += n_pairs, ++it) {
                const int buf = it & 1;
                const uint32_t acc_phase = (uint32_t)(it >> 1) & 1u;
                if (!mbar_wait(tempty_bar(buf), acc_phase ^ 1u, &abort_flag)) goto done;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(buf * BN);
                const int kb0 = k_first(t), kb1 = k_end(t);
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!mbar_wait(full_bar(stage), phase, &abort_flag)) goto done;
                    tc_fence_after();
                    const uint32_t sa = base + stage * kStageBytes;
                    const uint32_t sb = sa + kABytes;
#pragma unroll
                    for (int kk = 0; kk < BK / 16; ++kk) {
                        const uint64_t da = A_MN ? smem_desc_sw128(sa + kk * 2048, 8192, 1024) : smem_desc_sw128(sa + kk * 32, 16, 1024);
                        const uint64_t db = B_MN ? smem_desc_sw128(sb + kk * 2048, 8192, 1024) : smem_desc_sw128(sb + kk * 32, 16, 1024);
                        umma2_bf16_ss(d_tmem, da, db, idesc, (kb > kb0 || kk) ? 1u : 0u);
                    }
                    umma2_commit_both(empty_bar(stage));        // frees this stage in both CTAs when the MMAs retire
                    if (++stage == kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                umma2_commit_both(tfull_bar(buf));              // accumulator complete, both halves
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue (warps 2..5 of each CTA: its 128 rows)
        const int quad = warp & 3;
        uint32_t nbox = 0;       // boxes alternate across tiles too: a tile may store an odd number of them
        int it = 0;
        for (int t = pair; t < num_tiles; t += n_pairs, ++it) {
            int m0, n0;
            tile_coords(t, m0, n0);
            const int buf = it & 1;
            const uint32_t acc_phase = (uint32_t)(it >> 1) & 1u;
            if (!mbar_wait(tfull_bar(buf), acc_phase, &abort_flag)) goto done;
            tc_fence_after();
            const int row0 = m0 + (int)rank * BMH + quad * 32;
            const int row = row0 + lane;
            const bool row_ok = row < p.M;
            const uint32_t tacc = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * BN);
            const __nv_bfloat16* arow = (EPI == 3 || EPI == 4) ? p.aux + (long)row * p.ldc : nullptr;
            // Through shared memory and the TMA unit: a lane holds a row, so direct 16-byte stores touch 32 rows per instruction and
            // the epilogue of a tile, not its products, set the pace of short-K products (12288 x 3072 x 256, 75 MB written: 43.8 us direct, 25.2 us this way; 32656 x 12288 x 3072:
            // 1676 and 1625 us).
            const uint32_t box = epi_stage + (uint32_t)(warp - 2) * 8192u;
            if (EPI == 7) {
                const int prow = (t % p.splits) * p.part_rows + row0;
#pragma unroll 1
                for (int c = 0; c < BN / 32; ++c) {
                    const int col0 = n0 + c * 32;
                    if (col0 >= p.N || row0 >= p.M) break;
                    uint32_t r[32];
                    tmem_ld_32x32(tacc + c * 32, r);
                    tmem_ld_wait();
                    store_box_32x64(box + 4096u * (nbox++ & 1u), &tmC, col0, prow, lane,
                                    [&](int g) { return make_uint4(r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]); });
                }
            } else
#pragma unroll 1
            for (int c = 0; c < BN / 64; ++c) {
                const int col0 = n0 + c * 64;
                if (col0 >= p.N || row0 >= p.M) break;
                uint32_t r[64];
                tmem_ld_32x32(tacc + c * 64, r);
                tmem_ld_32x32(tacc + c * 64 + 32, r + 32);
                tmem_ld_wait();
                auto packed = [&](int g, bool pre) -> uint4 {
                    const int col = col0 + g * 8;
                    float bv[8], uv[8], o[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) bv[j] = uv[j] = 0.f;
                    if (EPI <= 2 && p.bias != nullptr && col + 8 <= p.N) tt::unpack8(tt::ld8(p.bias + col), bv);
                    if ((EPI == 3 || EPI == 4) && row_ok && col + 8 <= p.N) tt::unpack8(tt::ld8(arow + col), uv);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        o[j] = pre ? __uint_as_float(r[g * 8 + j]) + bv[j] : epi2<EPI>(__uint_as_float(r[g * 8 + j]), bv[j], uv[j]);
                    const tt::bf16x8 pk = tt::pack8(o);
                    return *reinterpret_cast<const uint4*>(&pk);
                };
                if (EPI == 1 || EPI == 2) store_box_32x64(box + 4096u * (nbox++ & 1u), &tmAux, col0, row0, lane, [&](int g) { return packed(g, true); });
                store_box_32x64<EPI == 5>(box + 4096u * (nbox++ & 1u), &tmC, col0, row0, lane,
                                          [&](int g) { return packed(g, false); });
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(tempty_bar(buf));
        }
        if (lane == 0) bulk_wait_read<0>();        // the boxes outlive the copies that read them
    }

done:
    tc_fence_before();
    __syncthreads();
    if (abort_flag) {
        if (threadIdx.x == 0) atomicExch(p.status, TT_ERR_TIMEOUT);
        for (int i = 0; i < 200; ++i) __nanosleep(1000);        // let TMA copies in flight land
    }
    // both CTAs are done with each other's shared and tensor memory before either frees it
    cluster_arrive();
    cluster_wait();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc2(tmem_base, 512);
    }
}

template <bool A_MN, bool B_MN, int EPI>
int launch2(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const CUtensorMap& tmAux, const CUtensorMap& tmA2,
            const Params2& p, const tt_device_info& on, cudaStream_t st) {
    auto kern = gemm2_kernel<A_MN, B_MN, EPI>;
    static bool configured[64] = {false};
    if (!configured[on.dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
        if (e != cudaSuccess) return tt_record_cuda(e);
        configured[on.dev] = true;
    }
    const int tiles = p.tiles_m * p.tiles_n * p.splits;
    int pairs = on.sms / 2;
    if (pairs > tiles) pairs = tiles;
    if (pairs < 1) pairs = 1;
    kern<<<2 * pairs, kThreads, kSmemBytes, st>>>(tmA, tmB, tmC, tmAux, tmA2, p);      // cluster shape comes from __cluster_dims__
    TT_CHECK_LAUNCH();
    return TT_OK;
}

// out = epilogue(sum of the splits' slices): 8 columns per thread, slices added in order
template <int EPI>
__global__ void __launch_bounds__(256) splitk_finish_kernel(const float* __restrict__ part, int splits, long slice, int M, int N, long ldc,
                                                           const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ aux,
                                                           __nv_bfloat16* __restrict__ C) {
    const int nvec = N >> 3;
    const long total = (long)M * nvec;
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const long row = i / nvec;
        const int col = (int)(i - row * nvec) * 8;
        const float* src = part + row * N + col;
        float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int s = 0; s < splits; ++s) {
            const float4 x = __ldcs(reinterpret_cast<const float4*>(src + s * slice)), y = __ldcs(reinterpret_cast<const float4*>(src + s * slice) + 1);
            a[0] += x.x; a[1] += x.y; a[2] += x.z; a[3] += x.w;
            a[4] += y.x; a[5] += y.y; a[6] += y.z; a[7] += y.w;
        }
        float bv[8], uv[8], o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) bv[j] = uv[j] = 0.f;
        if (EPI <= 2 && bias != nullptr) tt::unpack8(tt::ld8(bias + col), bv);
        if (EPI >= 3) tt::unpack8(tt::ld8(aux + row * ldc + col), uv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = epi2<EPI>(a[j], bv[j], uv[j]);
        if (EPI == 1 || EPI == 2) {
#pragma unroll
            for (int j = 0; j < 8; ++j) a[j] += bv[j];
            tt::st8(aux + row * ldc + col, tt::pack8(a));
        }
        tt::st8(C + row * ldc + col, tt::pack8(o));
    }
}

// The product of every entry point.  a2 (or nullptr) supplies the K columns from k1 on; splits > 1 needs `scratch`.
int run2(const void* a, const void* a2, int k1, long lda2, const void* b, void* c, const void* bias, void* aux, int M, int N, int K, long lda,
         long ldb, long ldc, int a_mn, int b_mn, int epi, int splits, float* scratch, int* status, void* stream) {
    // epilogue 5 (both operands K x MN) takes any K, there a row count: the rows beyond it load as zeros
    if (M <= 0 || N <= 0 || K <= 0 || (N & 7) || ((K & 7) && epi != 5) || (ldc & 7) || status == nullptr) return TT_ERR_ARG;
    if (a_mn && (M & 7)) return TT_ERR_ARG;
    if (epi < 0 || epi > 5 || (epi >= 1 && epi <= 4 && aux == nullptr)) return TT_ERR_ARG;
    if (epi == 5 && (!a_mn || !b_mn || bias != nullptr || splits != 1)) return TT_ERR_ARG;
    if (((uintptr_t)c & 15) || (bias && ((uintptr_t)bias & 15)) || (aux && ((uintptr_t)aux & 15))) return TT_ERR_ARG;
    if (a_mn && !b_mn) return TT_ERR_ARG;
    if (a2 != nullptr && (a_mn || k1 <= 0 || k1 >= K || (k1 % BK))) return TT_ERR_ARG;
    const int kblocks = (K + BK - 1) / BK;
    if (splits < 1 || splits > kblocks || (splits > 1 && (scratch == nullptr || ((uintptr_t)scratch & 15)))) return TT_ERR_ARG;
    const tt_device_info on = tt_device();
    int rc;
    CUtensorMap tmA, tmA2, tmB, tmC, tmAux;
    if (!a_mn) rc = tt_make_tmap_2d(&tmA, a, (uint64_t)M, (uint64_t)(a2 != nullptr ? k1 : K), (uint64_t)lda, BMH, BK);
    else rc = tt_make_tmap_2d(&tmA, a, (uint64_t)K, (uint64_t)M, (uint64_t)lda, 64, 64);
    if (rc != TT_OK) return rc;
    tmA2 = tmA;
    if (a2 != nullptr && (rc = tt_make_tmap_2d(&tmA2, a2, (uint64_t)M, (uint64_t)(K - k1), (uint64_t)lda2, BMH, BK)) != TT_OK) return rc;
    if (!b_mn) rc = tt_make_tmap_2d(&tmB, b, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, BNH, BK);
    else rc = tt_make_tmap_2d(&tmB, b, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, 64, 64);
    if (rc != TT_OK) return rc;
    Params2 p;
    memset(&p, 0, sizeof(p));
    p.M = M; p.N = N; p.K = K;
    p.ldc = ldc;
    p.bias = (const __nv_bfloat16*)bias;
    p.aux = (__nv_bfloat16*)aux;
    p.status = status;
    p.tiles_m = (M + 255) / 256;
    p.tiles_n = (N + 255) / 256;
    p.k1 = a2 != nullptr ? k1 : K;
    p.kb_split = (kblocks + splits - 1) / splits;
    p.splits = (kblocks + p.kb_split - 1) / p.kb_split;           // no empty range
    p.part_rows = (M + 31) / 32 * 32;
    cudaStream_t st = (cudaStream_t)stream;
    const bool amn = a_mn != 0, bmn = b_mn != 0;
    if (splits == 1) {
        if ((rc = tt_make_tmap_2d(&tmC, c, (uint64_t)M, (uint64_t)N, (uint64_t)ldc, 32, 64)) != TT_OK) return rc;
        tmAux = tmC;
        if ((epi == 1 || epi == 2) && (rc = tt_make_tmap_2d(&tmAux, aux, (uint64_t)M, (uint64_t)N, (uint64_t)ldc, 32, 64)) != TT_OK) return rc;
#define GO(A_, B_, E_) return launch2<A_, B_, E_>(tmA, tmB, tmC, tmAux, tmA2, p, on, st)
        if (!amn && !bmn) {
            if (epi == 0) GO(false, false, 0);
            if (epi == 1) GO(false, false, 1);
            if (epi == 2) GO(false, false, 2);
        } else if (!amn && bmn) {
            if (epi == 0) GO(false, true, 0);
            if (epi == 3) GO(false, true, 3);
            if (epi == 4) GO(false, true, 4);
        } else if (amn && bmn) {
            if (epi == 0) GO(true, true, 0);
            if (epi == 5) GO(true, true, 5);
        }
#undef GO
        return TT_ERR_ARG;
    }
    if ((rc = tt_make_tmap_2d_f32(&tmC, scratch, (uint64_t)p.part_rows * p.splits, (uint64_t)N, (uint64_t)N, 32, 32)) != TT_OK) return rc;
    if (!amn && !bmn) rc = launch2<false, false, 7>(tmA, tmB, tmC, tmC, tmA2, p, on, st);
    else if (!amn) rc = launch2<false, true, 7>(tmA, tmB, tmC, tmC, tmA2, p, on, st);
    else rc = launch2<true, true, 7>(tmA, tmB, tmC, tmC, tmA2, p, on, st);
    if (rc != TT_OK) return rc;
    const long want = ((long)M * (N >> 3) + 255) / 256;
    const int grid = (int)(want < 148L * 8 ? want : 148L * 8);
    const long slice = (long)p.part_rows * N;
#define FIN(E_)                                                                                                          \
    splitk_finish_kernel<E_><<<grid, 256, 0, st>>>(scratch, p.splits, slice, M, N, ldc, (const __nv_bfloat16*)bias,        \
                                                   (__nv_bfloat16*)aux, (__nv_bfloat16*)c)
    if (epi == 0) FIN(0);
    else if (epi == 1) FIN(1);
    else if (epi == 2) FIN(2);
    else if (epi == 3) FIN(3);
    else FIN(4);
#undef FIN
    TT_CHECK_LAUNCH();
    return TT_OK;
}

}  // namespace

// Same contract as tt_gemm_bf16 (gemm_tcgen05.cu); returns TT_ERR_ARG for shapes this kernel does not take, so that the
// caller can fall back to the single-CTA kernel.
extern "C" int tt_gemm2_bf16(const void* a, const void* b, void* c, const void* bias, void* aux, int M, int N, int K,
                             long lda, long ldb, long ldc, int a_mn, int b_mn, int epi, int* status, void* stream) {
    return run2(a, nullptr, 0, 0, b, c, bias, aux, M, N, K, lda, ldb, ldc, a_mn, b_mn, epi, 1, nullptr, status, stream);
}

// The product with its k-blocks shared by `splits` pairs per tile.  scratch: fp32, splits * roundup(M, 32) * N entries.
extern "C" int tt_gemm2_bf16_splitk(const void* a, const void* b, void* c, const void* bias, void* aux, int M, int N, int K, long lda, long ldb,
                                    long ldc, int a_mn, int b_mn, int epi, int splits, float* scratch, int* status, void* stream) {
    return run2(a, nullptr, 0, 0, b, c, bias, aux, M, N, K, lda, ldb, ldc, a_mn, b_mn, epi, splits, scratch, status, stream);
}

// c = [a | a2] b^T + bias: a [M, k1] (k1 a multiple of 64), a2 [M, K - k1], b [N, K]; splits and scratch as above.
extern "C" int tt_gemm2_bf16_two(const void* a, const void* a2, const void* b, void* c, const void* bias, int M, int N, int K, int k1, long lda,
                                 long lda2, long ldb, long ldc, int splits, float* scratch, int* status, void* stream) {
    if (a2 == nullptr) return TT_ERR_ARG;
    return run2(a, a2, k1, lda2, b, c, bias, nullptr, M, N, K, lda, ldb, ldc, 0, 0, 0, splits, scratch, status, stream);
}
