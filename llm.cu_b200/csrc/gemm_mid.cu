// Projections of middling prompt blocks (of the 8B shape 129 to 672 rows of QKV, to 896 of o_proj and down_proj; not SwiGLU):
// C[M][N] = A[M][K] . B[N][K]^T where the tiles are one wave: a CTA per tile and SM.  Same arithmetic as gemm_tc.cu.
//
// The WEIGHTS are the 128-row operand of tcgen05.mma and the block's rows are its columns, as in gemm_smallm.cu, because the
// number of columns can be any multiple of 16: with 128-row tiles of the block 517 rows are 640, and the 160 tiles of o_proj
// are a second wave of 12.  Here the rows are cut into as many tiles of equal height (nt) as one wave takes.
//
// Bound: L2 to shared memory.  Per K step of 16 an SM loads (128 + nt) x 32 bytes, at 62 to 64 bytes a cycle, and the MMA takes
// max(nt / 2, 32 + nt / 4) cycles (both measured): 64 + nt / 2 cycles a step, and no less than 120 with a stage of four steps, the
// time of the waits, copies and MMAs of a stage.  So lower tiles than about 96 rows (M in ceil(M / 96) tiles, at the least 80 rows each)
// gain nothing; where that leaves half of the SMs idle, K is cut in two
// and the two CTAs of a tile are a cluster: each leaves the sums of half of the columns in its shared memory (the ring, free by
// then) for the other, which adds them in slice order and finishes them.  us at m = 200 / 384 / 517 rows (8B shape, weights from HBM, a graph of
// launches) against gemm_tc: QKV 31.9 / 31.6 / 34.8 -> 24.0 / 29.2 / 32.5, o_proj 29.3 / 30.1 / 31.5 -> 19.3 / 22.3 / 28.7, down_proj 61.4 / 92.8 / 95.6 ->
// 41.0 / 49.2 / 73.0.
// The K of a CTA is summed in two accumulators, four up to 128 columns (all 512 columns of tensor memory), which the epilogue adds: tcgen05.mma
// truncates where it adds to its accumulator, an error that grows with the length of the chain.
//
//   warps 0, 10  TMA: 16 KB of weights / 128 bytes per row of the block to a stage
//   warp 1       tensor-memory owner, MMA issue
//   warps 2-9    epilogue, thread = weight row and half of the tile's columns, straight from tensor memory
// The copy and MMA warps run as whole warps with one elected lane at the copies and MMAs, and look at the next stage's barrier while
// they work on this one: single threads that waited stage by stage took 620 cycles a stage, more than most tiles' MMAs.
// Every wait is bounded.
#include <algorithm>

#include "gemm_common.cuh"

namespace llmb {

constexpr int kMidMaxStages = 8, kMidRing = 216 * 1024, kMidEpilogueWarps = 8, kMidThreads = 96 + 32 * kMidEpilogueWarps;
__host__ __device__ constexpr uint32_t mid_stage_bytes(int nt) { return kATileBytes + (uint32_t)nt * kBK * 2; }

__device__ __forceinline__ bool mid_elect() {
    uint32_t one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(one));
    return one != 0;
}
__device__ __forceinline__ bool mid_peek(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(smem_u32(bar)), "r"(parity)
                 : "memory");
    return __all_sync(0xffffffffu, ok != 0);
}
__device__ __forceinline__ bool mid_wait(uint64_t *bar, uint32_t parity, int *status, int code, int lane) {
    return __all_sync(0xffffffffu, mbar_wait_warp(bar, parity, status, code, lane));
}

__global__ void __launch_bounds__(kMidThreads, 1)
gemm_mid_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const GemmParams p) {
    extern __shared__ __align__(1024) unsigned char mid_smem[];
    __shared__ __align__(8) uint64_t full_bar[kMidMaxStages], empty_bar[kMidMaxStages], acc_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint64_t drain_bar;
    __shared__ int prior_status;

    unsigned char *ring = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(mid_smem) + 1023) & ~uintptr_t(1023));
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const bool clustered = p.splits > 1;  // K in two halves, the two CTAs of a tile are a cluster along y
    const int slice = clustered ? (int)cluster_cta_rank() : 0, kt0 = slice * (p.K / kBK) / p.splits;
    const int nt = p.nx, stages = p.stages, k_tiles = (slice + 1) * (p.K / kBK) / p.splits - kt0;
    const uint32_t stage_bytes = mid_stage_bytes(nt);
    const uint32_t idesc = (1u << 4) | ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
    // row tiles vary fastest: the CTAs of a weight tile run together and it comes from HBM once
    const int m_tiles = (p.M + nt - 1) / nt, m0 = (int)blockIdx.x % m_tiles * nt, n0 = (int)blockIdx.x / m_tiles * kBM;
    // K in `chains` accumulators of `acc_cols` columns, `part` K steps each (the last one the rest)
    const int most = nt <= 128 ? 4 : 2, acc_cols = 512 / most, part = (k_tiles + most - 1) / most, chains = (k_tiles + part - 1) / part;

    if (threadIdx.x == 0) {
        prior_status = *reinterpret_cast<volatile int *>(p.status);
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full_bar[s], 2);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&acc_bar, 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
    pdl_launch_dependents();  // this CTA has its tensor memory (see gemm_tc.cu)

    // of 16 columns: what this CTA finishes (the other half of them the cluster's other CTA)
    const int groups = nt / 16, middle = (groups + 1) / 2;
    const int own_begin = slice == 0 ? 0 : middle, own_end = !clustered || slice == 1 ? groups : middle;
    const int lane_group = (warp & 3) * 32, side = (warp - 2) >> 2;
    const uint32_t taddr = tmem + ((uint32_t)lane_group << 16);
    float *sums = reinterpret_cast<float *>(ring);  // [column of the other half][weight row], once the ring is free
    bool done = false;                              // the accumulators are complete
    // sixteen columns of all accumulators
    auto add = [&](int c, float (&v)[16]) {
#pragma unroll 1
        for (int b = 0; b < chains; ++b) {
            uint32_t w[16];
            tmem_ld16(taddr + b * acc_cols + c * 16, w);
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = b == 0 ? __uint_as_float(w[i]) : v[i] + __uint_as_float(w[i]);
        }
    };
    // Of two rows the even lanes take the first, the odd ones the second: features col, col + 1.
    const bool odd = lane & 1;
    const int col0 = n0 + lane_group, col = col0 + (lane & 30), half_dim = p.head_dim >> 1;
    const bool is_q = col0 < p.n_q, is_v = col0 >= p.n_q + p.n_kv;
    const int local = is_q ? col : (is_v ? col - p.n_q - p.n_kv : col - p.n_q), pair = half_dim > 0 ? (local >> 1) % half_dim : 0;
    const bool residual = p.epilogue == LLMB_EPI_RESIDUAL, rope = p.epilogue == LLMB_EPI_ROPE_KV && !is_v;
    const int own_middle = own_begin + (own_end - own_begin + 1) / 2;
    const int c_begin = side == 0 ? own_begin : own_middle, c_end = side == 0 ? own_middle : own_end;
    // What a group of rows needs besides the sums (residual: x, RoPE: y too) is asked for one group ahead.
    float2 next[8];
    auto ask = [&](int c) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int row = min(m0 + c * 16 + 2 * i + (odd ? 1 : 0), p.M - 1);
            next[i] = make_float2(0.0f, 0.0f);
            if (residual && col0 < p.N) next[i].x = __uint_as_float(__ldcg(reinterpret_cast<const unsigned int *>(p.c + (size_t)row * p.N + col)));
            if (rope) next[i] = __ldg(p.rope_cs + (size_t)row * half_dim + pair);
        }
    };

    if (prior_status != 0) {
        pdl_wait();
    } else if (warp == 0 || warp == 10) {
        // ---- copies: warp 0 the weights, warp 10 the block's rows ----
        const bool rows = warp == 10;
        const uint32_t bytes = rows ? stage_bytes - kATileBytes : kATileBytes;
        unsigned char *base = rows ? ring + kATileBytes : ring;
        const CUtensorMap *map = rows ? &map_x : &map_w;
        const int y = rows ? m0 : n0;
        bool ok = true, free = true;         // `free`: stage s has been seen to be free already
        uint32_t s = 0, parity = 1;          // parity of the round before: complete at once in the first one
        if (rows) pdl_wait();                // the activations are the previous kernel's output; the weights nobody's
        int kt = 0;
#pragma unroll 1
        for (; kt < k_tiles; ++kt) {
            if (!free) ok = mid_wait(&empty_bar[s], parity, p.status, 361, lane);
            if (!ok) break;
            const uint32_t s2 = s + 1 == (uint32_t)stages ? 0 : s + 1, parity2 = s2 ? parity : parity ^ 1;
            free = mid_peek(&empty_bar[s2], parity2);  // the answer comes while this stage is asked for
            if (mid_elect()) {
                mbar_arrive_expect_tx(&full_bar[s], bytes);
                tma_load_2d(base + (size_t)s * stage_bytes, map, (kt0 + kt) * kBK, y, &full_bar[s]);
            }
            __syncwarp();
            s = s2;
            parity = parity2;
        }
        // A wait gave up: no copy of this CTA's is under way when it leaves (a stage that the other warp has not asked for never
        // completes: that wait ends at its limit).
        if (!ok && lane == 0) drain_copies(full_bar, stages, max(0, kt - stages), kt);
    } else if (warp == 1) {
        const uint64_t ring_desc = umma_desc(ring);  // a stage further: its bytes / 16 more
        bool ok = true, full = false;                // `full`: stage s has been seen to be full already
        uint32_t s = 0, parity = 0, acc = tmem;
        int kt = 0, left = part;                     // K steps that the accumulator still takes
#pragma unroll 1
        for (; kt < k_tiles; ++kt) {
            if (!full) ok = mid_wait(&full_bar[s], parity, p.status, 362, lane);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t s2 = s + 1 == (uint32_t)stages ? 0 : s + 1, parity2 = s2 ? parity : parity ^ 1;
            full = mid_peek(&full_bar[s2], parity2);  // the answer comes while this stage's MMAs are issued
            const uint64_t wdesc = ring_desc + s * (stage_bytes >> 4), xdesc = wdesc + (kATileBytes >> 4);
            if (mid_elect()) {
#pragma unroll
                for (int k = 0; k < kBK / 16; ++k) umma_f16(acc, wdesc + 2 * k, xdesc + 2 * k, idesc, left < part || k > 0 ? 1u : 0u);
                umma_commit(&empty_bar[s]);
            }
            __syncwarp();
            if (--left == 0) {
                left = part;
                acc += acc_cols;
            }
            s = s2;
            parity = parity2;
        }
        if (mid_elect()) umma_commit(&acc_bar);  // also after a wait that gave up: the epilogue never waits forever
        __syncwarp();
        if (!ok && lane == 0) wind_down_mma(full_bar, stages, kt, min(kt + stages, k_tiles), &drain_bar);
    } else {
        // ---- epilogue ----
        pdl_wait();  // it reads and writes global memory of earlier kernels
        if (c_begin < c_end) ask(c_begin);
        done = mbar_wait_warp(&acc_bar, 0, p.status, 363, lane);
        if (!done) mbar_wait(&acc_bar, 0, nullptr, 0);
        // a wait of another warp that gave up has set the status word: the accumulators are incomplete
        done = __all_sync(0xffffffffu, done && *reinterpret_cast<volatile int *>(p.status) == 0);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (clustered) {  // the other CTA's columns: through this one's shared memory
            const int begin = slice == 0 ? middle : 0, end = slice == 0 ? groups : middle;
#pragma unroll 1
            for (int c = begin + side; c < end; c += 2) {
                float v[16];
                add(c, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) sums[((c - begin) * 16 + i) * kBM + lane_group + lane] = v[i];
            }
        }
    }
    if (clustered) cluster_sync_all();  // both halves of K are there
    if (warp >= 2 && warp < 10) {
        uint32_t other_sums = 0;
        if (clustered) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(other_sums) : "r"(smem_u32(sums)), "r"(slice ^ 1));
        // Not unrolled: a CTA runs its epilogue once, so every instruction of it is fetched cold.
#pragma unroll 1
        for (int c = c_begin; c < c_end && done; ++c) {
            __syncwarp();  // see tmem_ld32; before the loads below, which it would wait for
            float2 now[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) now[i] = next[i];
            if (c + 1 < c_end) ask(c + 1);
            float v[16];
            add(c, v);
            if (clustered) {
                float w[16];
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(w[i]) : "r"(other_sums + (uint32_t)(((c - own_begin) * 16 + i) * kBM + lane_group + lane) * 4));
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] += w[i];
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int row = m0 + c * 16 + 2 * i + (odd ? 1 : 0);
                const float other = __shfl_xor_sync(0xffffffffu, odd ? v[2 * i] : v[2 * i + 1], 1);
                const float e = odd ? other : v[2 * i], o = odd ? v[2 * i + 1] : other;
                __half2 out = __halves2half2(__float2half_rn(e), __float2half_rn(o));
                if (row >= p.M || col0 >= p.N) continue;
                const float2 x = __half22float2(out);
                __half *dst = p.c + (size_t)row * p.N + col;
                if (residual) {
                    const uint32_t bits = __float_as_uint(now[i].x);
                    const float2 old = __half22float2(*reinterpret_cast<const __half2 *>(&bits));
                    out = __halves2half2(__float2half_rn(x.x + old.x), __float2half_rn(x.y + old.y));
                } else if (p.epilogue == LLMB_EPI_ROPE_KV) {
                    if (rope)
                        out = __halves2half2(__float2half_rn(__fmaf_rn(now[i].x, x.x, -__fmul_rn(now[i].y, x.y))),
                                             __float2half_rn(__fmaf_rn(now[i].y, x.x, __fmul_rn(now[i].x, x.y))));
                    dst = p.c + (size_t)row * p.n_q + col;
                    if (!is_q) {
                        size_t cache_row;
                        const int pos = kv_position(p, row, cache_row);
                        if (pos < 0 || pos >= p.max_pos) continue;
                        dst = (is_v ? p.v_cache : p.k_cache) + cache_row * p.n_kv + local;
                    }
                }
                *reinterpret_cast<__half2 *>(dst) = out;
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (clustered) cluster_sync_all();  // no CTA leaves while the other may still read its sums
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// Rows of a tile and slices of K where all tiles are one wave of at least 3/8 of the SMs; 0 rows where they are not.  Of the cuts of
// the rows and the one or two slices the pair whose CTAs take least time, a step of 16 at max(121, 64 + nt / 2) cycles.  Prompts of 129 /
// 200 / 256 tokens without slices 6.40 / 6.42 / 6.57 ms, with them 5.39 / 5.60 / 5.85.
// Two slices from k = 2048 on (32 K steps): below, the exchange can cost more than the shorter K saves.  us with two slices / one,
// n = 4096, m = 200: k = 512 10.5 / 11.4, 1024 11.5 / 13.6, 2048 14.0 / 18.0, 4096 18.6 / 26.0; m = 384: 11.9 / 10.4, 13.3 / 12.6, 16.2 / 16.7, 21.9 / 24.9.
// 3/8 of the SMs keeps the cost honest where one slice would leave most of them idle: 300 x 2176 x 1024 in 3 cuts (51 CTAs) 13.3 us, in 4 11.9.
// It only decides below k = 2048 (above, two slices double the CTAs), and there also leaves a few sizes to gemm_tc.cu that this kernel
// would do faster (n 3200 to 3456 at up to 192 rows, 2176 and 2304 at 257 to 288: 160 x 3200 x 1024 19.1 us there, 12.0 here).
// From 225 rows a tile on gemm_wide.cu is as fast or faster: prompts of 1000 / 1024 tokens (o_proj and down_proj in tiles of 256) 15.6 / 15.6 ->
// 15.9 / 16.2 ms with this kernel.  At 224 rows in one slice the kernel alone is slower than gemm_wide.cu and gemm_tc.cu (672 x 6144 x 4096
// 36.9 us against 31.9, 896 x 4096 x 4096 36.3 against 33.4: the part that does not grow with K, 7.5 us against 5, counts), but not behind another kernel whose
// end hides that: prompts of 640 / 672 / 896 tokens take 11.0 / 11.9 / 14.5 ms either way.  For the same reason it is slower alone at
// k below about 1200 (484 x 1920 x 192 9.3 us against 6.2); its four accumulators of up to 128 rows are the more exact there.
// Where gemm_tc.cu cuts K into three and more parts, its sums are in shorter chains than here: it keeps those.
static int mid_tile_rows(int m, int n, int k, int sms, int &splits) {
    const int w_tiles = (n + kBM - 1) / kBM;
    int best = 0, least = 0;
    splits = 1;
    if (w_tiles * ((m + 127) / 128) * 3 <= sms) return 0;
    for (int s = 1; s <= (k / kBK >= 32 ? 2 : 1); ++s)
        for (int cuts = 1; w_tiles * cuts * s <= sms && cuts <= (m + 95) / 96; ++cuts) {
            const int nt = ((m + cuts - 1) / cuts + 15) / 16 * 16, cost = std::max(242, 128 + nt) / s;
            if (nt > 224 || w_tiles * cuts * s * 8 < 3 * sms || (best && cost >= least)) continue;
            best = nt;
            least = cost;
            splits = s;
        }
    return best;
}

bool gemm_mid_takes(const LlmbGemmArgs *a) {
    int splits;
    return a->tile_n == 0 && a->epilogue != LLMB_EPI_SWIGLU && mid_tile_rows(a->m, a->n, a->k, sm_count_cached(), splits) > 0;
}

int launch_gemm_mid(const LlmbGemmArgs *a, int rows_per_seq, bool pdl, cudaStream_t stream) {
    CUtensorMap mw, mx;
    int rc;
    GemmParams p = {};
    if ((rc = fill_gemm_params(p, a, rows_per_seq))) return rc;
    p.nx = mid_tile_rows(a->m, a->n, a->k, sm_count_cached(), p.splits);
    p.stages = std::min(kMidMaxStages, (int)(kMidRing / mid_stage_bytes(p.nx)));
    if ((rc = make_map(&mw, a->b, a->n, a->k, kBM))) return rc;
    if ((rc = make_map(&mx, a->a, a->m, a->k, p.nx))) return rc;
    const int tiles = ((a->m + p.nx - 1) / p.nx) * ((a->n + kBM - 1) / kBM);
    const size_t smem = (size_t)p.stages * mid_stage_bytes(p.nx) + 1024;
    static size_t attr_set[kMaxDevices] = {};
    LLMB_CUDA_OK(ensure_dynamic_smem(gemm_mid_kernel, attr_set, smem));
    LLMB_CUDA_OK(launch_pdl_cluster(gemm_mid_kernel, dim3((unsigned)tiles, (unsigned)p.splits), dim3(kMidThreads), smem, stream, pdl,
                                    dim3(1, (unsigned)p.splits, 1), mw, mx, p));
    return LLMB_OK;
}

}  // namespace llmb
