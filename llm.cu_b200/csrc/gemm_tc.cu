// Prompt-phase projections: C[M][N] = A[M][K] . B[N][K]^T on the 5th-generation tensor cores.
//
// Replaces kernel_standard_tiled_gemm / kernel_standard_tiled_gemm_ffn_swiglu of the reference
// (inference.cu:393-519) for M > 1 rows, with the same FP16 inputs, FP32 accumulation and FP16
// rounding points, and the neighbouring element-wise kernels fused into the epilogue.
//
// Bound: tensor pipe (2 * M * N * K flops); A and B are both K-major, which is how the
// activations and the checkpoint's [out][in] weights already sit in memory.
//
//   tile     128 x BN output per CTA (BN = 128, 64 or 32: the widest that still gives every SM a CTA),
//            K in steps of 64 (one 128-byte swizzle span of FP16); two CTAs share an SM, so one's
//            epilogue overlaps the other's main loop
//   warp 0   producer: TMA (cp.async.bulk.tensor.2d, 128B swizzle, no multicast) fills a shared-memory
//            ring, completion on mbarriers; 3 stages (SwiGLU: 2) when CTAs share an SM, up to 8 when
//            the grid is a single partial wave and only the ring can hide the copy latency
//   warp 1   allocates tensor memory and issues tcgen05.mma (kind::f16, M = 128, N = BN, K = 16)
//            from one elected lane; tcgen05.commit releases ring stages and signals the epilogue
//   warps 2-5 epilogue: tcgen05.ld the FP32 accumulators (one output row per thread), apply
//            store / residual add / RoPE + KV-cache append / SiLU(gate) * up, write FP16
// The SwiGLU variant keeps two accumulators (gate and up, 2 x BN TMEM columns) fed by two B tiles.  The others use two as
// well, one for each half of the CTA's K, and the epilogue adds them: tcgen05.mma truncates where it adds to its
// accumulator, an error that grows with the length of the chain (results that are not the nearest FP16 at k = 4096 / 14336:
// 1.7 % / 5.1 % with one chain).  Two CTAs' columns fill the SM's tensor memory either way.
// Rows of A beyond M are zero-filled by TMA and masked in the epilogue; N and K must be multiples
// of 128 and 64.  Every mbarrier wait is bounded (status word, see llmb_device_status).
// A launch with few output tiles and a caller-provided workspace splits K over blockIdx.z: partial
// accumulators are written to the workspace in FP32, and the last CTA of a tile to arrive adds them in
// slice order and runs the epilogue.
#include "gemm_common.cuh"

namespace llmb {

template <bool DUAL, int kBN>
__global__ void __launch_bounds__(kGemmThreads, 2)
gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               const __grid_constant__ CUtensorMap map_b2, const GemmParams p) {
    extern __shared__ __align__(1024) unsigned char gemm_smem[];
    __shared__ __align__(8) uint64_t full_bar[kGemmMaxStages];
    __shared__ __align__(8) uint64_t empty_bar[kGemmMaxStages];
    __shared__ __align__(8) uint64_t acc_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint64_t drain_bar;
    __shared__ int prior_status;
    __shared__ int split_last;

    const int kGemmStages = p.stages;
    constexpr uint32_t kBTileBytes = kBN * kBK * 2;
    constexpr uint32_t kStageBytes = gemm_stage_bytes(DUAL, kBN);  // every tile a multiple of 1024 bytes
    constexpr uint32_t kTmemCols = 2 * kBN;
    // kind::f16: D = F32 (bit 4), A = B = F16 (0), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
    constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(kBN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);

    // the dynamic shared memory window is only 16-byte aligned by contract: align the ring to 1024 bytes
    unsigned char *ring = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(gemm_smem) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // row tiles vary fastest across the grid: the CTAs that share a weight tile run together and it
    // comes from DRAM once
    const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * kBN;
    const int k_tiles = p.K / kBK;
    const int kt_begin = (int)((long long)blockIdx.z * k_tiles / p.splits);
    const int kt_end = (int)((long long)(blockIdx.z + 1) * k_tiles / p.splits);

    // a wait that gave up earlier (here or in another kernel) leaves the status word set: do not queue
    // up more bounded waits behind it
    if (threadIdx.x == 0) prior_status = *reinterpret_cast<volatile int *>(p.status);
    __syncthreads();
    if (prior_status != 0) {
        pdl_wait();
        return;
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < kGemmStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&acc_bar, 1);
        fence_mbar_init();
    }
    if (warp == 1) {  // one warp allocates the accumulator columns
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_slot;
    // not before the accumulator columns are allocated: a CTA of the next kernel that took them first would wait for
    // this one (griddepcontrol.wait) while this one waits for the columns
    pdl_launch_dependents();

    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            // the head of the weight stream does not depend on the previous kernel: ask for it first
            const int head = min(kGemmStages, kt_end - kt_begin);
            for (int i = 0; i < head; ++i) {
                unsigned char *st = ring + (size_t)i * kStageBytes;
                mbar_arrive_expect_tx(&full_bar[i], kStageBytes);
                tma_load_2d(st + kATileBytes, &map_b, (kt_begin + i) * kBK, n0, &full_bar[i]);
                if (DUAL) tma_load_2d(st + kATileBytes + kBTileBytes, &map_b2, (kt_begin + i) * kBK, n0, &full_bar[i]);
            }
            pdl_wait();  // the activations are the previous kernel's output
            for (int i = 0; i < head; ++i) tma_load_2d(ring + (size_t)i * kStageBytes, &map_a, (kt_begin + i) * kBK, m0, &full_bar[i]);
            int i = head;
            for (int kt = kt_begin + head; kt < kt_end && ok; ++kt, ++i) {
                const int s = i % kGemmStages;
                ok = mbar_wait(&empty_bar[s], ((i / kGemmStages) - 1) & 1, p.status, 301);
                if (!ok) break;
                unsigned char *st = ring + (size_t)s * kStageBytes;
                mbar_arrive_expect_tx(&full_bar[s], kStageBytes);
                tma_load_2d(st, &map_a, kt * kBK, m0, &full_bar[s]);
                tma_load_2d(st + kATileBytes, &map_b, kt * kBK, n0, &full_bar[s]);
                if (DUAL) tma_load_2d(st + kATileBytes + kBTileBytes, &map_b2, kt * kBK, n0, &full_bar[s]);
            }
            if (!ok) drain_copies(full_bar, kGemmStages, max(0, i - kGemmStages), i);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            bool ok = true;
            const int second = DUAL ? -1 : (kt_end - kt_begin + 1) / 2;  // first K step of the second accumulator
            int i = 0;
            for (int kt = kt_begin; kt < kt_end && ok; ++kt, ++i) {
                const int s = i % kGemmStages;
                ok = mbar_wait(&full_bar[s], (i / kGemmStages) & 1, p.status, 302);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                unsigned char *st = ring + (size_t)s * kStageBytes;
                const uint64_t adesc = umma_desc(st), bdesc = umma_desc(st + kATileBytes);
                const uint64_t b2desc = DUAL ? umma_desc(st + kATileBytes + kBTileBytes) : 0;
#pragma unroll
                for (int k = 0; k < kBK / 16; ++k) {
                    const uint32_t acc = ((i > 0 && i != second) || k > 0) ? 1u : 0u;
                    // 16 FP16 along K = 32 bytes = 2 descriptor address units inside the swizzle span
                    umma_f16(tmem_base + (!DUAL && i >= second ? kBN : 0), adesc + 2 * k, bdesc + 2 * k, kIdesc, acc);
                    if (DUAL) umma_f16(tmem_base + kBN, adesc + 2 * k, b2desc + 2 * k, kIdesc, acc);
                }
                umma_commit(&empty_bar[s]);  // the stage may be refilled once these MMAs have read it
            }
            umma_commit(&acc_bar);  // arrives even after a failed wait, so the epilogue never waits forever
            if (!ok) wind_down_mma(full_bar, kGemmStages, i, min(i + kGemmStages, kt_end - kt_begin), &drain_bar);
        }
    } else {
        // ---- epilogue: thread = one row of the tile, TMEM lanes (warp % 4) * 32 .. + 32 ----
        const bool ok = mbar_wait(&acc_bar, 0, p.status, 303);
        if (!ok) mbar_wait(&acc_bar, 0, nullptr, 0);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        pdl_wait();  // from here on global memory of earlier kernels is read and written
        const int lane_group = (warp & 3) * 32;
        const int row = m0 + lane_group + lane;
        const bool row_ok = ok && row < p.M;
        constexpr int kAccCols = (DUAL ? 2 : 1) * kBN;
        const bool two_chains = !DUAL && kt_end - kt_begin > 1;
        // 32 columns of the accumulator, the two chains added; warp-collective
        auto load_acc = [&](uint32_t taddr, uint32_t (&v)[32]) {
            __syncwarp();  // see tmem_ld32
            if (!two_chains) {
                tmem_ld32(taddr, v);
                return;
            }
            uint32_t w[32];
            tmem_ld32_async(taddr, v);
            tmem_ld32_async(taddr + kBN, w);
            tmem_wait_ld32(v);
            tmem_wait_ld32(w);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) + __uint_as_float(w[i]));
        };
        const int tile_id = blockIdx.y * gridDim.x + blockIdx.x;
        bool finish = true;  // this CTA runs the epilogue
        if (p.splits > 1) {
            float *mine = p.ws_part + (((size_t)tile_id * p.splits + blockIdx.z) * kBM + lane_group + lane) * kAccCols;
#pragma unroll 1
            for (int c = 0; c < kBN / 32; ++c) {
                uint32_t v[32];
                const uint32_t taddr = tmem_base + ((uint32_t)lane_group << 16) + (uint32_t)(c * 32);
                load_acc(taddr, v);  // every lane takes part, rows past M are not stored
                if (row_ok) {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        reinterpret_cast<uint4 *>(mine + c * 32)[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                }
                if (DUAL) {
                    __syncwarp();
                    tmem_ld32(taddr + kBN, v);
                    if (row_ok) {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            reinterpret_cast<uint4 *>(mine + kBN + c * 32)[i] = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    }
                }
            }
            __threadfence();  // this thread's partials are visible device-wide before the arrival is counted
            named_bar_sync(1, 128);
            if (threadIdx.x == 64) {
                const int arrived = atomicAdd(p.ws_count + tile_id, 1);
                split_last = (arrived == p.splits - 1) ? 1 : 0;
                if (split_last) p.ws_count[tile_id] = 0;  // ready for the next launch
                __threadfence();
            }
            named_bar_sync(1, 128);
            finish = split_last != 0;
        }
#pragma unroll 1
        for (int c = 0; c < kBN / 32 && finish; ++c) {
            uint32_t v[32], u[32];
            if (p.splits > 1) {
                if (!row_ok) continue;  // no collective below on this path
                // partial sums in slice order: the result does not depend on which CTA arrived last
                float fv[32], fu[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) fv[i] = fu[i] = 0.0f;
                for (int z = 0; z < p.splits; ++z) {
                    const float *part = p.ws_part + (((size_t)tile_id * p.splits + z) * kBM + lane_group + lane) * kAccCols + c * 32;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float4 t = __ldcg(reinterpret_cast<const float4 *>(part) + i);
                        fv[4 * i] += t.x; fv[4 * i + 1] += t.y; fv[4 * i + 2] += t.z; fv[4 * i + 3] += t.w;
                    }
                    if (DUAL) {
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float4 t = __ldcg(reinterpret_cast<const float4 *>(part + kBN) + i);
                            fu[4 * i] += t.x; fu[4 * i + 1] += t.y; fu[4 * i + 2] += t.z; fu[4 * i + 3] += t.w;
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    v[i] = __float_as_uint(fv[i]);
                    u[i] = __float_as_uint(fu[i]);
                }
            } else {
                const uint32_t taddr = tmem_base + ((uint32_t)lane_group << 16) + (uint32_t)(c * 32);
                load_acc(taddr, v);
                if (DUAL) tmem_ld32(taddr + kBN, u);
            }
            if (row_ok) finish_cols<DUAL>(p, row, n0 + c * 32, v, u);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
    return fn;
}

// [rows][k] FP16 row-major as a 2-D tensor map with a 64 x box_rows box and 128-byte swizzle.
int make_map(CUtensorMap *map, const void *base, int rows, int k, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_last_error("cuTensorMapEncodeTiled is not available from this driver");
        return LLMB_ERR_UNSUPPORTED;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)k * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_last_error("cuTensorMapEncodeTiled failed (base must be 16-byte aligned, k a multiple of 8)");
        return LLMB_ERR_INVALID;
    }
    return LLMB_OK;
}

int make_map_3d(CUtensorMap *map, const void *base, int d0, int d1, int d2, size_t stride1, size_t stride2, int box1, int box2) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_last_error("cuTensorMapEncodeTiled is not available from this driver");
        return LLMB_ERR_UNSUPPORTED;
    }
    const cuuint64_t dims[3] = {(cuuint64_t)d0, (cuuint64_t)d1, (cuuint64_t)d2};
    const cuuint64_t strides[2] = {(cuuint64_t)stride1 * 2, (cuuint64_t)stride2 * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)box1, (cuuint32_t)box2};
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_last_error("cuTensorMapEncodeTiled failed (base must be 16-byte aligned, strides multiples of 8 elements)");
        return LLMB_ERR_INVALID;
    }
    return LLMB_OK;
}

int fill_gemm_params(GemmParams &p, const LlmbGemmArgs *a, int rows_per_seq) {
    p.c = reinterpret_cast<__half *>(a->c);
    p.rope_cs = reinterpret_cast<const float2 *>(a->rope_cs);
    p.k_cache = reinterpret_cast<__half *>(a->k_cache);
    p.v_cache = reinterpret_cast<__half *>(a->v_cache);
    p.status = device_status_ptr();
    if (!p.status) return LLMB_ERR_CUDA;
    p.M = a->m; p.N = a->n; p.K = a->k; p.epilogue = a->epilogue;
    p.n_q = a->n_q; p.n_kv = a->n_kv; p.head_dim = a->head_dim; p.pos0 = a->pos0; p.max_pos = a->max_pos;
    p.row_pos = a->row_pos;
    p.seq_stride = a->seq_stride;
    p.rows_per_seq = rows_per_seq > 0 ? rows_per_seq : a->m;
    p.splits = 1;
    return LLMB_OK;
}

}  // namespace llmb

extern "C" int llmb_gemm_f16(const LlmbGemmArgs *a, llmb_stream_t stream_) {
    return llmb::launch_gemm(a, 0, a && a->use_pdl != 0 && a->m <= 32 && a->tile_n == 0, static_cast<cudaStream_t>(stream_));
}

int llmb::launch_gemm(const LlmbGemmArgs *a, int rows_per_seq, bool pdl, cudaStream_t stream) {
    if (!a || !a->a || !a->b || (!a->c && a->epilogue != LLMB_EPI_TP_SCATTER) || a->m <= 0 || a->n <= 0 || a->k <= 0) return LLMB_ERR_INVALID;
    const bool small_m = a->m <= kSmallM && a->tile_n == 0;
    // the weight-streaming kernel masks the tail of its last tile, so STORE / TP_SCATTER take any multiple of 8 there
    const bool any_n = small_m && (a->epilogue == LLMB_EPI_STORE || a->epilogue == LLMB_EPI_TP_SCATTER) && a->n % 8 == 0;
    if ((a->n % 128 && !any_n) || a->k % kBK) {
        set_last_error("llmb_gemm_f16: n must be a multiple of 128 and k a multiple of 64");
        return LLMB_ERR_UNSUPPORTED;
    }
    if (a->epilogue == LLMB_EPI_TP_SCATTER && (a->m > 32 || a->tile_n != 0)) {
        set_last_error("llmb_gemm_f16: LLMB_EPI_TP_SCATTER needs m <= 32");
        return LLMB_ERR_UNSUPPORTED;
    }
    const bool dual = a->epilogue == LLMB_EPI_SWIGLU;
    if (dual && !a->b2) return LLMB_ERR_INVALID;
    if (a->epilogue == LLMB_EPI_ROPE_KV) {
        if (!a->rope_cs || !a->k_cache || !a->v_cache || a->head_dim <= 0 || (a->head_dim & 1) ||
            a->n != a->n_q + 2 * a->n_kv || a->n_q % 32 || a->n_kv % 32)
            return LLMB_ERR_INVALID;
    } else if (a->epilogue != LLMB_EPI_STORE && a->epilogue != LLMB_EPI_RESIDUAL && a->epilogue != LLMB_EPI_TP_SCATTER && !dual) {
        return LLMB_ERR_INVALID;
    }
    // A handful of rows (batched decode): the weight-streaming kernel with the operands swapped
    if (small_m) return launch_gemm_smallm(a, rows_per_seq, pdl, stream);
    if (gemm_mid_takes(a)) return launch_gemm_mid(a, rows_per_seq, pdl, stream);
    if (gemm_wide_takes(a)) return launch_gemm_wide(a, rows_per_seq, pdl, stream);
    // Small grids: with a workspace, 128-wide tiles and K split across CTAs until the SMs are covered
    // (every CTA then streams its own weights and only its slice of the activations); without one, the
    // widest tile that still gives every SM a CTA.
    const int m_tiles = (a->m + kBM - 1) / kBM;
    const int sms = sm_count_cached();
    const bool have_ws = a->workspace && a->workspace_bytes > 4096 && (((uintptr_t)a->workspace) & 15) == 0;
    int bn = a->tile_n;
    if (bn == 0) {
        bn = 128;
        if (!have_ws)
            while (bn > 32 && (a->n / bn) * m_tiles < sms) bn >>= 1;
    }
    if (bn != 128 && bn != 64 && bn != 32) {
        set_last_error("llmb_gemm_f16: tile_n must be 0, 32, 64 or 128");
        return LLMB_ERR_INVALID;
    }
    CUtensorMap ma, mb, mb2;
    int rc;
    if ((rc = make_map(&ma, a->a, a->m, a->k, kBM))) return rc;
    if ((rc = make_map(&mb, a->b, a->n, a->k, bn))) return rc;
    if ((rc = make_map(&mb2, dual ? a->b2 : a->b, a->n, a->k, bn))) return rc;
    GemmParams p = {};
    if ((rc = fill_gemm_params(p, a, rows_per_seq))) return rc;
    dim3 grid(m_tiles, a->n / bn);
    const int tiles = (int)(grid.x * grid.y), k_tiles = a->k / kBK;
    if (have_ws && tiles * 2 <= sms && tiles <= 1024) {
        int splits = sms / tiles;
        if (splits > 8) splits = 8;
        if (splits > k_tiles / 8) splits = k_tiles / 8;
        const size_t need = 4096 + (size_t)tiles * splits * kBM * (dual ? 2 : 1) * bn * sizeof(float);
        if (splits > 1 && need <= a->workspace_bytes) p.splits = splits;
    }
    p.ws_count = static_cast<int *>(a->workspace);
    p.ws_part = reinterpret_cast<float *>(static_cast<unsigned char *>(a->workspace) + 4096);
    grid.z = p.splits;
    p.stages = gemm_stages(dual);
    if (tiles * p.splits <= sms) {
        p.stages = (int)((size_t)200 * 1024 / gemm_stage_bytes(dual, bn));
        if (p.stages > kGemmMaxStages) p.stages = kGemmMaxStages;
    }
    const size_t smem = (size_t)p.stages * gemm_stage_bytes(dual, bn) + 1024;
    void (*kernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const GemmParams) =
        dual ? (bn == 128 ? gemm_tc_kernel<true, 128> : bn == 64 ? gemm_tc_kernel<true, 64> : gemm_tc_kernel<true, 32>)
             : (bn == 128 ? gemm_tc_kernel<false, 128> : bn == 64 ? gemm_tc_kernel<false, 64> : gemm_tc_kernel<false, 32>);
    static size_t attr_set[2][3][kMaxDevices] = {};  // per instantiation and device
    LLMB_CUDA_OK(ensure_dynamic_smem(kernel, attr_set[dual ? 1 : 0][bn == 128 ? 0 : bn == 64 ? 1 : 2], smem));
    LLMB_CUDA_OK(launch_pdl(kernel, grid, dim3(kGemmThreads), smem, stream, pdl, ma, mb, mb2, p));
    return LLMB_OK;
}
