// Projections for a handful of rows (batched decode: one new row per sequence; short prompts; m <= 128):
// C[m][n] = X[m][k] . W[n][k]^T with the roles of the two operands swapped on the tensor cores.
//
// Replaces kernel_standard_tiled_gemm / kernel_standard_tiled_gemm_ffn_swiglu of the reference
// (inference.cu:393-519) at small m, with the same FP16 inputs, FP32 accumulation, FP16 rounding points and
// fused element-wise neighbours as gemm_tc.cu.
//
// Bound: HBM.  Every weight byte is streamed once per launch; the m activation rows (a few KB per K step)
// come from L2.  So the kernel is shaped as a weight stream, like the batch-1 projections, not as a GEMM:
//
//   operands  the WEIGHT tile is the 128-row (M) operand of tcgen05.mma, the activation rows are the nx-column
//             (N) operand, nx = m rounded up to 32: D[128 weight rows][nx activation rows] in tensor memory.  A ring
//             stage is 16 KB of weights + 4 KB per 32 activation rows (32 KB of weights for the gate/up pair), so most
//             of the shared memory in flight is weight bytes, and an MMA step costs nx / 128 of the 128-wide one.
//   grid      x = 128-row weight tile, y = slice of K.  K is split in 2, 4 or 8 until about two CTAs per SM
//             exist (each slice at least 8 K steps).  The CTAs of one tile form a thread-block cluster: each
//             leaves its partial accumulators (128 x nx FP32) in its own shared memory, and after a
//             cluster barrier CTA r adds the partials of activation rows r * nx/S .. through distributed
//             shared memory, in slice order, and runs the epilogue for those rows.  No workspace, no atomic,
//             no last CTA that reduces alone.
//   ring      about 100 KB per CTA, so that two CTAs share an SM: two of this launch, or the tail of this
//             launch and the head of the next one.
//   overlap   programmatic dependent launch: a CTA releases its dependents at entry and asks for its first
//             ring-full of WEIGHT tiles at once (weights never depend on an earlier kernel); only then does
//             it wait for the previous kernel (griddepcontrol.wait) and ask for the activation tiles.  The
//             epilogue warps wait too before they touch global memory.
//   warps     0 = TMA producer, 1 = MMA issuer (one lane) + tensor-memory owner, 2-5 = epilogue; thread =
//             tensor-memory lane = one weight row n, holding the values of all activation rows for it.
// Every mbarrier wait is bounded (status word, see llmb_device_status).
#include <type_traits>

#include "gemm_common.cuh"
#include "tp_common.cuh"

namespace llmb {

constexpr int kNX = 32;                                   // the activation rows of a launch (N of the MMA) are a multiple of this
constexpr uint32_t kWTileBytes = kBM * kBK * 2;           // 16 KB
constexpr int kSmallMaxStages = 8;
__host__ __device__ constexpr uint32_t small_stage_bytes(bool dual, int nx) { return (dual ? 2 : 1) * kWTileBytes + nx * kBK * 2; }

// The sum of S slices' partial sums in slice order.
template <int S>
__device__ __forceinline__ float add_slices(const float (&t)[S]) {
    float sum = 0.0f;
#pragma unroll
    for (int z = 0; z < S; ++z) sum += t[z];
    return sum;
}

template <bool DUAL>
__global__ void __launch_bounds__(kGemmThreads, 2)
gemm_smallm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_w2,
                   const __grid_constant__ CUtensorMap map_x, const GemmParams p) {
    extern __shared__ __align__(1024) unsigned char small_smem[];
    __shared__ __align__(8) uint64_t full_bar[kSmallMaxStages];
    __shared__ __align__(8) uint64_t empty_bar[kSmallMaxStages];
    __shared__ __align__(8) uint64_t acc_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint64_t drain_bar;
    __shared__ int prior_status;

    constexpr uint32_t kXOff = (DUAL ? 2 : 1) * kWTileBytes;
    const int nx = p.nx;
    const uint32_t stage_bytes = small_stage_bytes(DUAL, nx);
    // an allocation is a power of two from 32 on: (DUAL ? 2 : 1) * nx columns rounded up
    const uint32_t tmem_cols = (DUAL ? 2u : 1u) * (nx <= 32 ? 32u : nx <= 64 ? 64u : 128u);
    // kind::f16: D = F32 (bit 4), A = B = F16, both K-major, N >> 3 at bit 17, M >> 4 at bit 24
    const uint32_t idesc = (1u << 4) | ((uint32_t)(nx >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);

    unsigned char *ring = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(small_smem) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int stages = p.stages;
    const int n0 = blockIdx.x * kBM;
    const int k_tiles = p.K / kBK;
    const bool clustered = p.splits > 1;  // then the p.splits CTAs of a tile are one cluster along y
    const int slice = clustered ? (int)cluster_cta_rank() : 0;
    const int kt_begin = (int)((long long)slice * k_tiles / p.splits);
    const int kt_end = (int)((long long)(slice + 1) * k_tiles / p.splits);

    const int cta = blockIdx.y * gridDim.x + blockIdx.x;
    auto stamp = [&](int which) {
        if (p.trace) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
            p.trace[(size_t)cta * 8 + which] = t;
        }
    };
    if (threadIdx.x == 0) stamp(0);  // entry
    // The next kernel may start its own weight stream as soon as an SM has room (and this CTA has its accumulator
    // columns, see gemm_tc.cu).  After a scattering projection the next kernel is the gather, which takes no wait of its
    // own and reads the exchange counter and the residual rows at once: it is let go only after this kernel's wait, when
    // every earlier kernel is complete.
    const bool scatter = !DUAL && p.epilogue == LLMB_EPI_TP_SCATTER;
    // a wait that gave up earlier (here or in another kernel) leaves the status word set: take no wait at all,
    // but still let the previous kernel finish first so that the order of the chain holds
    if (threadIdx.x == 0) prior_status = *reinterpret_cast<volatile int *>(p.status);
    __syncthreads();  // one read for the whole CTA: every thread takes the same way out
    if (prior_status != 0) {
        pdl_wait();
        if (clustered) {  // the other CTAs of the cluster may still read this one's shared memory: leave with them
            cluster_sync_all();
            cluster_sync_all();
        }
        return;
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&acc_bar, 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_slot;
    if (!scatter) pdl_launch_dependents();
    if (threadIdx.x == 0) stamp(1);  // barriers and tensor memory ready

    if (warp == 0) {
        if (lane == 0) {
            // the head of the weight stream does not depend on the previous kernel: ask for it first
            const int head = min(stages, kt_end - kt_begin);
            for (int i = 0; i < head; ++i) {
                unsigned char *st = ring + (size_t)i * stage_bytes;
                mbar_arrive_expect_tx(&full_bar[i], stage_bytes);
                tma_load_2d(st, &map_w, (kt_begin + i) * kBK, n0, &full_bar[i]);
                if (DUAL) tma_load_2d(st + kWTileBytes, &map_w2, (kt_begin + i) * kBK, n0, &full_bar[i]);
            }
            pdl_wait();  // the activations are the previous kernel's output
            if (scatter) pdl_launch_dependents();
            stamp(2);    // previous kernel complete
            // a wait that gave up earlier leaves the status word set: do not queue more bounded waits behind it
            bool ok = *reinterpret_cast<volatile int *>(p.status) == 0;
            for (int i = 0; i < head; ++i)
                tma_load_2d(ring + (size_t)i * stage_bytes + kXOff, &map_x, (kt_begin + i) * kBK, 0, &full_bar[i]);
            int i = head;
            for (int kt = kt_begin + head; kt < kt_end && ok; ++kt, ++i) {
                const int s = i % stages;
                ok = mbar_wait(&empty_bar[s], ((i / stages) - 1) & 1, p.status, 311);
                if (!ok) break;
                unsigned char *st = ring + (size_t)s * stage_bytes;
                mbar_arrive_expect_tx(&full_bar[s], stage_bytes);
                tma_load_2d(st, &map_w, kt * kBK, n0, &full_bar[s]);
                if (DUAL) tma_load_2d(st + kWTileBytes, &map_w2, kt * kBK, n0, &full_bar[s]);
                tma_load_2d(st + kXOff, &map_x, kt * kBK, 0, &full_bar[s]);
            }
            if (!ok) drain_copies(full_bar, stages, max(0, i - stages), i);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            bool ok = true;
            int i = 0;
            for (int kt = kt_begin; kt < kt_end && ok; ++kt, ++i) {
                const int s = i % stages;
                ok = mbar_wait(&full_bar[s], (i / stages) & 1, p.status, 312);
                if (!ok) break;
                if (i == 0) stamp(3);  // first stage landed
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                unsigned char *st = ring + (size_t)s * stage_bytes;
                const uint64_t wdesc = umma_desc(st), xdesc = umma_desc(st + kXOff);
                const uint64_t w2desc = DUAL ? umma_desc(st + kWTileBytes) : 0;
#pragma unroll
                for (int k = 0; k < kBK / 16; ++k) {
                    const uint32_t acc = (i > 0 || k > 0) ? 1u : 0u;
                    umma_f16(tmem_base, wdesc + 2 * k, xdesc + 2 * k, idesc, acc);
                    if (DUAL) umma_f16(tmem_base + nx, w2desc + 2 * k, xdesc + 2 * k, idesc, acc);
                }
                umma_commit(&empty_bar[s]);
            }
            stamp(4);  // last MMA issued
            umma_commit(&acc_bar);  // arrives even after a failed wait, so the epilogue never waits forever
            if (!ok) wind_down_mma(full_bar, stages, i, min(i + stages, kt_end - kt_begin), &drain_bar);
        }
    }
    // ---- epilogue: thread = weight row n0 + lane_group + lane.  Loops over four or eight rows that are NOT unrolled over
    // all of them: a CTA runs its epilogue once, so every instruction of it is fetched cold, and the fully unrolled form
    // (five epilogues x 32 rows) cost 5-19 us of instruction fetch per launch.  With a test per possible slice and
    // everything through shared memory it took 14 / 11 / 37 / 10 us of the four projections of a layer at 96 rows (last
    // accumulator to last store); this form 14 / 10 / 12 / 9.
    const int lane_group = (warp & 3) * 32;
    const int nl = lane_group + lane;
    const int n = n0 + nl;
    uint32_t *red_own = reinterpret_cast<uint32_t *>(ring);
    bool ok = false;
    if (warp >= 2) {
        const bool got = mbar_wait(&acc_bar, 0, p.status, 313);
        if (!got) mbar_wait(&acc_bar, 0, nullptr, 0);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (threadIdx.x == 64) stamp(5);  // accumulators complete
        pdl_wait();  // from here on global memory of earlier kernels is read and written
        ok = got && *reinterpret_cast<volatile int *>(p.status) == 0;
    }
    // every load of the ring has landed and every MMA has read it (acc_bar): the ring is free
    const uint32_t taddr = tmem_base + ((uint32_t)lane_group << 16);
    // Split K: every slice leaves its partial sums in its shared memory as [accumulator][activation row][weight row].
    if (clustered) {
        if (warp >= 2) {
#pragma unroll 1
            for (int b0 = 0; b0 < (DUAL ? 2 : 1) * nx; b0 += 32) {
                uint32_t v[32];
                __syncwarp();  // see tmem_ld32
                tmem_ld32(taddr + b0, v);
#pragma unroll
                for (int b = 0; b < 32; ++b) red_own[(b0 + b) * kBM + nl] = v[b];
            }
        }
        cluster_sync_all();  // all slices of the tile are in shared memory
    }
    if (threadIdx.x == 64) stamp(6);
    if (warp >= 2) {
        // Output element (b, n): the 32 lanes of a warp hold 32 consecutive n, so each store of a warp is one 64-byte run of
        // row b.  R rows at a time: their loads first, then their stores (a load after a store to the same array would have
        // to wait for it).
        const bool valid = ok && n < p.N;  // the last weight tile may reach past N (its rows are zero-filled by TMA)
        const int half_dim = p.head_dim >> 1;
        const bool is_q = n < p.n_q, is_v = n >= p.n_q + p.n_kv;
        const int local = is_q ? n : (is_v ? n - p.n_q - p.n_kv : n - p.n_q);
        const int pair = half_dim > 0 ? (local >> 1) % half_dim : 0;
        const unsigned int tag = p.epilogue == LLMB_EPI_TP_SCATTER ? __ldg(p.tp_seq) + (unsigned int)p.tp_index + 1u : 0u;
        auto finish = [&](int b0, int b_hi, auto &val, auto &val2) {
            constexpr int R = sizeof(val) / sizeof(float);
            if (!DUAL && p.epilogue == LLMB_EPI_TP_SCATTER) {
                // tensor parallel: this rank's partial sums go, tagged, to every rank's receive buffer
                const size_t slot0 = tp_rows_slot(p.tp_size, p.N, p.tp_index, p.tp_rank, 0, n);
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    if (valid && b0 + i < b_hi) {
                        const size_t off = slot0 + (size_t)(b0 + i) * p.N * 8;
                        for (int r = 0; r < p.tp_size; ++r)
                            asm volatile("st.relaxed.sys.global.v2.b32 [%0], {%1, %2};" ::"l"(p.tp_peer[r] + off), "r"(__float_as_uint(val[i])),
                                         "r"(tag)
                                         : "memory");
                    }
                }
            } else if (DUAL) {
#pragma unroll
                for (int i = 0; i < R; ++i)
                    if (valid && b0 + i < b_hi) p.c[(size_t)(b0 + i) * p.N + n] = __float2half_rn(silu_gemm(val[i]) * val2[i]);
            } else if (p.epilogue == LLMB_EPI_STORE) {
#pragma unroll
                for (int i = 0; i < R; ++i)
                    if (valid && b0 + i < b_hi) p.c[(size_t)(b0 + i) * p.N + n] = __float2half_rn(val[i]);
            } else if (p.epilogue == LLMB_EPI_RESIDUAL) {
                __half res[R];
#pragma unroll
                for (int i = 0; i < R; ++i) res[i] = valid && b0 + i < b_hi ? __ldcg(p.c + (size_t)(b0 + i) * p.N + n) : __half(0.0f);
#pragma unroll
                for (int i = 0; i < R; ++i)
                    if (valid && b0 + i < b_hi)
                        p.c[(size_t)(b0 + i) * p.N + n] = __float2half_rn(__half2float(__float2half_rn(val[i])) + __half2float(res[i]));
            } else {  // LLMB_EPI_ROPE_KV: the pair (even n, n + 1) sits in neighbouring lanes
                float2 cs[R];
                int pos[R];
                size_t cache_row[R];
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    const int b = min(b0 + i, b_hi - 1);
                    cs[i] = is_v ? make_float2(1.0f, 0.0f) : __ldg(p.rope_cs + (size_t)b * half_dim + pair);
                    pos[i] = kv_position(p, b, cache_row[i]);
                }
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    const float mine = __half2float(__float2half_rn(val[i]));
                    const float other = __shfl_xor_sync(0xffffffffu, mine, 1);
                    __half out;
                    if (is_v) {
                        out = __float2half_rn(val[i]);
                    } else {
                        out = __float2half_rn((n & 1) ? __fmaf_rn(cs[i].y, other, __fmul_rn(cs[i].x, mine))
                                                      : __fmaf_rn(cs[i].x, mine, -__fmul_rn(cs[i].y, other)));
                    }
                    if (valid && b0 + i < b_hi) {
                        if (is_q) p.c[(size_t)(b0 + i) * p.n_q + n] = out;
                        else if (pos[i] >= 0 && pos[i] < p.max_pos) (is_v ? p.v_cache : p.k_cache)[cache_row[i] * p.n_kv + local] = out;
                    }
                }
            }
        };
        // CTA r of a cluster of S finishes activation rows r * nx/S ..: the loads of R rows x S slices go out together.
        auto gather = [&](auto s_const) {
            constexpr int S = decltype(s_const)::value, R = S >= 4 ? 4 : 8;  // eight with RoPE (S 4 as a rule): 3 us more of it, fetched cold
            const int nb = nx / S, first = slice * nb, b_hi = min(first + nb, p.M);
            uint32_t rbase[S];
#pragma unroll
            for (int z = 0; z < S; ++z) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(rbase[z]) : "r"(smem_u32(ring)), "r"(z));
#pragma unroll 1
            for (int b0 = first; b0 < b_hi; b0 += R) {
                float t[(DUAL ? 2 : 1) * R][S], val[R], val2[R];
#pragma unroll
                for (int i = 0; i < (DUAL ? 2 : 1) * R; ++i) {
                    const uint32_t off = (uint32_t)(((i / R * nx + min(b0 + i % R, b_hi - 1)) * kBM + nl) * 4);
#pragma unroll
                    for (int z = 0; z < S; ++z) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(t[i][z]) : "r"(rbase[z] + off));
                }
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    val[i] = add_slices<S>(t[i]);
                    val2[i] = DUAL ? add_slices<S>(t[(DUAL ? R : 0) + i]) : 0.0f;
                }
                finish(b0, b_hi, val, val2);
            }
        };
        if (p.splits == 8) gather(std::integral_constant<int, 8>());
        else if (p.splits == 4) gather(std::integral_constant<int, 4>());
        else if (p.splits == 2) gather(std::integral_constant<int, 2>());
        else {  // no split: straight from tensor memory
#pragma unroll 1
            for (int b0 = 0; b0 < p.M; b0 += 8) {
                uint32_t v[8], u[8];
                float val[8], val2[8];
                __syncwarp();  // see tmem_ld32
                tmem_ld8(taddr + b0, v);
                if (DUAL) tmem_ld8(taddr + nx + b0, u);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    val[i] = __uint_as_float(v[i]);
                    val2[i] = DUAL ? __uint_as_float(u[i]) : 0.0f;
                }
                finish(b0, p.M, val, val2);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (clustered) cluster_sync_all();  // no CTA leaves while another may still read its partial sums
    if (threadIdx.x == 0) stamp(7);  // epilogue done
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    }
}

int launch_gemm_smallm(const LlmbGemmArgs *a, int rows_per_seq, bool pdl, cudaStream_t stream) {
    const bool dual = a->epilogue == LLMB_EPI_SWIGLU;
    const int nx = (a->m + kNX - 1) / kNX * kNX;
    CUtensorMap mw, mw2, mx;
    int rc;
    if ((rc = make_map(&mw, a->b, a->n, a->k, kBM))) return rc;
    if ((rc = make_map(&mw2, dual ? a->b2 : a->b, a->n, a->k, kBM))) return rc;
    if ((rc = make_map(&mx, a->a, a->m, a->k, nx))) return rc;
    GemmParams p = {};
    if ((rc = fill_gemm_params(p, a, rows_per_seq))) return rc;
    p.trace = reinterpret_cast<unsigned long long *>(a->trace);
    p.tp_seq = nullptr;
    if (a->epilogue == LLMB_EPI_TP_SCATTER) {
        if (dual || a->tp_size < 2 || a->tp_size > 8 || a->tp_rank < 0 || a->tp_rank >= a->tp_size || a->tp_index < 0) return LLMB_ERR_INVALID;
        for (int r = 0; r < a->tp_size; ++r) {
            if (!a->tp_peers[r]) return LLMB_ERR_INVALID;
            p.tp_peer[r] = static_cast<unsigned char *>(a->tp_peers[r]);
        }
        p.tp_rank = a->tp_rank; p.tp_size = a->tp_size; p.tp_index = a->tp_index;
        p.tp_seq = reinterpret_cast<const unsigned int *>(p.tp_peer[a->tp_rank] + tp_rows_seq_off(a->tp_size, a->n));
    }
    const int tiles = (a->n + kBM - 1) / kBM, k_tiles = a->k / kBK, sms = sm_count_cached();
    // K is split (2, 4 or 8 slices = the CTAs of one cluster) until about two CTAs per SM stream weights, each
    // slice at least 8 K steps long.  The gate/up pair moves two weight tiles per CTA: it is split only while
    // the tiles alone leave half of the SMs without a CTA.
    p.nx = nx;
    p.splits = 1;
    // More than 32 rows of the gate/up pair: its two blocks of partial sums (128 KB at 128 rows) leave room for one CTA per
    // SM where K is split; tiles enough for every SM are not split and keep two.
    const bool one_per_sm = dual && nx > kNX && tiles <= sms;
    const int ctas = one_per_sm ? sms : 2 * sms;
    if (tiles < ctas && !(dual && nx > kNX && !one_per_sm)) {
        int want = ctas / tiles;  // never more CTAs than can be resident at once
        if (want > k_tiles / 8) want = k_tiles / 8;
        p.splits = want >= 8 ? 8 : want >= 4 ? 4 : want >= 2 ? 2 : 1;
    }
    p.ws_count = nullptr;
    p.ws_part = nullptr;
    // about 100 KB of ring per CTA: two CTAs (of this launch, or of this and the next one) share an SM.  The ring also
    // holds the partial sums: (dual ? 2 : 1) * nx * 512 bytes with a split, 32 rows at a time without.
    const uint32_t stage = small_stage_bytes(dual, nx);
    p.stages = (int)((dual ? 108u : 100u) * 1024u / stage);
    if (dual && nx == kNX && tiles * p.splits <= sms) p.stages = 5;  // one CTA per SM anyway: a deeper ring (180 KB)
    if (one_per_sm) p.stages = (int)(196u * 1024u / stage);
    if (p.stages > kSmallMaxStages) p.stages = kSmallMaxStages;
    const size_t smem = (size_t)p.stages * stage + 1024;
    static size_t attr_set[2][kMaxDevices] = {};  // per instantiation and device
    if (dual) {
        LLMB_CUDA_OK(ensure_dynamic_smem(gemm_smallm_kernel<true>, attr_set[1], smem));
        LLMB_CUDA_OK(launch_pdl_cluster(gemm_smallm_kernel<true>, dim3(tiles, p.splits), dim3(kGemmThreads), smem, stream, pdl,
                                        dim3(1, p.splits, 1), mw, mw2, mx, p));
    } else {
        LLMB_CUDA_OK(ensure_dynamic_smem(gemm_smallm_kernel<false>, attr_set[0], smem));
        LLMB_CUDA_OK(launch_pdl_cluster(gemm_smallm_kernel<false>, dim3(tiles, p.splits), dim3(kGemmThreads), smem, stream, pdl,
                                        dim3(1, p.splits, 1), mw, mw2, mx, p));
    }
    return LLMB_OK;
}

}  // namespace llmb
