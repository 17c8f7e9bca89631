// Projections of long prompt blocks: C[M][N] = A[M][K] . B[N][K]^T as one persistent kernel, one CTA per SM, tiles of
// 128 x 256 (SwiGLU: 128 gate + 128 up columns) handed out round robin.  Same arithmetic and epilogues as gemm_tc.cu.
//
// Bound: tensor pipe, under the power cap.  A 128 x 128 tile reads its two operands from shared memory at 128 bytes per
// cycle while it multiplies, all that shared memory gives; a 128 x 256 tile reads 96.  Prompt of 4096 tokens (8B shape)
// 67.3 ms with 128 x 128 tiles, 60.0 with these (59.9 -> 59.0 with the two halves of K below in place of one tile's and the
// next one's accumulators).  CTA pairs (cta_group::2, 256 x 256
// tiles, 64 bytes per cycle) gained 3 % from 3000 rows on and lost 2 % at 2000 to 2384; cutting the last wave's tiles along
// K with FP32 parts in a workspace lost 6 % at 4096 rows and 20 % at 517 (a chain of L2 round trips per tile).
// The two accumulators (all 512 columns of tensor memory) are the two halves of K: tcgen05.mma truncates where it adds to its
// accumulator, an error that grows with the length of the chain (results that are not the nearest FP16 at k = 4096 / 14336:
// 1.7 % / 5.1 % in one chain, 1.0 % / 2.8 % in two).  The epilogue warps take the first half into registers while the second
// is multiplied, and finish with the second while the next tile's first is: the main loop never waits for them.  The ring
// runs on across tiles.
//
//   warp 0    TMA producer: 4 stages of 16 KB of A + 32 KB of B
//   warp 1    tensor-memory owner, MMA issue (M 128, N 256, K 16)
//   warps 2-9 epilogue, thread = output row and half of the tile's columns
// Row tiles vary fastest, so the CTAs that run together share weight tiles.  Every wait is bounded.
#include "gemm_common.cuh"

namespace llmb {

constexpr int kWideN = 256, kWideStages = 4;
constexpr int kWideEpilogueWarps = 8, kWideThreads = 64 + 32 * kWideEpilogueWarps;
constexpr uint32_t kWideBBytes = kWideN * kBK * 2, kWideStageBytes = kATileBytes + kWideBBytes;

template <bool DUAL>
__global__ void __launch_bounds__(kWideThreads, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                 const __grid_constant__ CUtensorMap map_b2, const GemmParams p) {
    extern __shared__ __align__(1024) unsigned char wide_smem[];
    __shared__ __align__(8) uint64_t full_bar[kWideStages], empty_bar[kWideStages], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint64_t drain_bar;
    __shared__ int prior_status;
    constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(kWideN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
    constexpr int kTileN = DUAL ? kWideN / 2 : kWideN;  // output columns of a tile

    unsigned char *ring = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(wide_smem) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m_tiles = (p.M + kBM - 1) / kBM, tiles = m_tiles * ((p.N + kTileN - 1) / kTileN), k_tiles = p.K / kBK;
    const int chains = k_tiles > 1 ? 2 : 1, half = (k_tiles + 1) / 2;  // K steps of the first accumulator

    if (threadIdx.x == 0) {
        prior_status = *reinterpret_cast<volatile int *>(p.status);
        for (int s = 0; s < kWideStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], kWideEpilogueWarps);
        }
        fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();  // this CTA has its tensor memory (see gemm_tc.cu)

    if (prior_status != 0) {
        pdl_wait();
    } else if (warp == 0) {
        if (lane == 0) {
            auto load_b = [&](unsigned char *st, int kt, int n0, uint64_t *bar) {
                tma_load_2d(st + kATileBytes, &map_b, kt * kBK, n0, bar);
                if (DUAL) tma_load_2d(st + kATileBytes + kWideBBytes / 2, &map_b2, kt * kBK, n0, bar);
            };
            bool ok = true;
            uint32_t it = 0;
            int head = 0;  // stages of the first tile whose weights are asked for before the previous kernel is complete
            if ((int)blockIdx.x < tiles) {
                head = min(kWideStages, k_tiles);
                for (int i = 0; i < head; ++i) {
                    mbar_arrive_expect_tx(&full_bar[i], kWideStageBytes);
                    load_b(ring + (size_t)i * kWideStageBytes, i, (int)blockIdx.x / m_tiles * kTileN, &full_bar[i]);
                }
            }
            pdl_wait();  // the activations are the previous kernel's output
            for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
                const int m0 = tile % m_tiles * kBM, n0 = tile / m_tiles * kTileN;
                for (int kt = 0; kt < k_tiles; ++kt, ++it) {
                    const int s = it % kWideStages;
                    unsigned char *st = ring + (size_t)s * kWideStageBytes;
                    if ((int)it >= head) {
                        if (it >= kWideStages) ok = mbar_wait(&empty_bar[s], ((it / kWideStages) - 1) & 1, p.status, 351);
                        if (!ok) break;
                        mbar_arrive_expect_tx(&full_bar[s], kWideStageBytes);
                        load_b(st, kt, n0, &full_bar[s]);
                    }
                    tma_load_2d(st, &map_a, kt * kBK, m0, &full_bar[s]);
                }
            }
            if (!ok) drain_copies(full_bar, kWideStages, max(0, (int)it - kWideStages), (int)it);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            bool ok = true;
            uint32_t it = 0;
            int n = 0;
            for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, ++n) {
                for (int b = 0; b < chains && ok; ++b) {
                    if (n >= 1) ok = mbar_wait(&acc_empty[b], (n - 1) & 1, p.status, 352);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const int kt_end = b + 1 < chains ? half : k_tiles;
                    for (int kt = b * half; kt < kt_end && ok; ++kt, ++it) {
                        const int s = it % kWideStages;
                        ok = mbar_wait(&full_bar[s], (it / kWideStages) & 1, p.status, 353);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const unsigned char *st = ring + (size_t)s * kWideStageBytes;
                        const uint64_t adesc = umma_desc(st), bdesc = umma_desc(st + kATileBytes);
#pragma unroll
                        for (int k = 0; k < kBK / 16; ++k)
                            umma_f16(tmem + b * kWideN, adesc + 2 * k, bdesc + 2 * k, kIdesc, kt > b * half || k > 0 ? 1u : 0u);
                        umma_commit(&empty_bar[s]);
                    }
                    umma_commit(&acc_full[b]);
                }
            }
            if (!ok) {
                const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;  // tiles of this CTA
                wind_down_mma(full_bar, kWideStages, (int)it, min((int)it + kWideStages, mine * k_tiles), &drain_bar);
            }
        }
    } else {
        bool ok = true;
        pdl_wait();  // the epilogue reads and writes global memory of earlier kernels
        const int lane_group = (warp & 3) * 32, part = (warp - 2) >> 2;
        // this thread's 128 accumulator columns, in groups of 32: one run of the output row's, or gate columns and the up
        // columns that belong to them
        const uint32_t taddr = tmem + ((uint32_t)lane_group << 16);
        auto column = [&](int g) { return DUAL ? (g >> 1) * kTileN + part * 64 + (g & 1) * 32 : part * 128 + g * 32; };
        auto wait_acc = [&](int b, int n) {
            ok = mbar_wait_warp(&acc_full[b], n & 1, p.status, 354, lane);
            if (!ok) mbar_wait(&acc_full[b], n & 1, nullptr, 0);
            // a wait of another warp that gave up has set the status word: its accumulators are incomplete
            ok = __all_sync(0xffffffffu, ok && *reinterpret_cast<volatile int *>(p.status) == 0);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            return ok;
        };
        auto release = [&](int b) {  // every column of this warp has been read: the accumulator may be overwritten
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[b]);
        };
        int n = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++n) {
            const int m0 = tile % m_tiles * kBM, n0 = tile / m_tiles * kTileN, row = m0 + lane_group + lane;
            uint32_t v[4][32];
            if (!wait_acc(0, n)) break;
#pragma unroll
            for (int g = 0; g < 4; ++g) tmem_ld32_async(taddr + column(g), v[g]);
#pragma unroll
            for (int g = 0; g < 4; ++g) tmem_wait_ld32(v[g]);
            release(0);
            if (chains > 1 && !wait_acc(1, n)) break;
            auto add_second = [&](int g) {
                __syncwarp();  // see tmem_ld32
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t w[16];
                    tmem_ld16(taddr + kWideN + column(g) + h * 16, w);
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[g][h * 16 + i] = __float_as_uint(__uint_as_float(v[g][h * 16 + i]) + __uint_as_float(w[i]));
                }
            };
#pragma unroll
            for (int g = 0; g < (DUAL ? 2 : 4); ++g) {
                if (chains > 1) {
                    add_second(g);
                    if (DUAL) add_second(2 + g);
                    if (g + 1 == (DUAL ? 2 : 4)) release(1);
                }
                const int col = n0 + column(g);
                if (row < p.M && col < p.N) finish_cols<DUAL>(p, row, col, v[g], v[DUAL ? 2 + g : g]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// From 6/7 of a wave on: prompts of 1000 and 1024 tokens (o_proj and down_proj of the 8B shape: 128 tiles on 148 SMs) 16.6 ->
// 15.6 ms against a whole wave; from half a wave on, 450 and 512 tokens lose 4 to 6 % and 800 gain 3.
bool gemm_wide_takes(const LlmbGemmArgs *a) {
    if (a->tile_n != 0) return false;
    const int sms = sm_count_cached(), m_tiles = (a->m + kBM - 1) / kBM;
    const int tile_n = a->epilogue == LLMB_EPI_SWIGLU ? kWideN / 2 : kWideN;
    const long long wide = (long long)m_tiles * ((a->n + tile_n - 1) / tile_n);
    return wide * 7 >= 6LL * sms;
}

int launch_gemm_wide(const LlmbGemmArgs *a, int rows_per_seq, bool pdl, cudaStream_t stream) {
    const bool dual = a->epilogue == LLMB_EPI_SWIGLU;
    const int sms = sm_count_cached(), tile_n = dual ? kWideN / 2 : kWideN;
    CUtensorMap ma, mb, mb2;
    int rc;
    if ((rc = make_map(&ma, a->a, a->m, a->k, kBM))) return rc;
    if ((rc = make_map(&mb, a->b, a->n, a->k, tile_n))) return rc;
    if ((rc = make_map(&mb2, dual ? a->b2 : a->b, a->n, a->k, tile_n))) return rc;
    GemmParams p = {};
    if ((rc = fill_gemm_params(p, a, rows_per_seq))) return rc;
    const long long tiles = (long long)((a->m + kBM - 1) / kBM) * ((a->n + tile_n - 1) / tile_n);
    if (tiles > 0x7fffffff - 65536) return LLMB_ERR_UNSUPPORTED;
    const size_t smem = (size_t)kWideStages * kWideStageBytes + 1024;
    auto kernel = dual ? gemm_wide_kernel<true> : gemm_wide_kernel<false>;
    static size_t attr_set[2][kMaxDevices] = {};  // per instantiation and device
    LLMB_CUDA_OK(ensure_dynamic_smem(kernel, attr_set[dual ? 1 : 0], smem));
    LLMB_CUDA_OK(launch_pdl(kernel, dim3((unsigned)(tiles < sms ? tiles : sms)), dim3(kWideThreads), smem, stream, pdl, ma, mb, mb2, p));
    return LLMB_OK;
}

}  // namespace llmb
