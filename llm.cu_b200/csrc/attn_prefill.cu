// Causal attention of a block of new rows against the KV cache on the 5th-generation tensor cores (replaces
// compute_attention's three kernels, inference.cu:698-947, for many rows): scores (q.k)/sqrtf(head_dim) in FP32 from
// FP16, softmax in FP32 (online, the N x N matrix is never materialised), P.V with FP32 accumulation, FP16 out.  K and V
// come from the cache rows that the QKV projection has just appended, so a block that starts at position pos0 > 0 attends
// to the earlier rows as well.
//
// Bound: tensor pipe.  Per 128 query rows and 128 keys: Q K^T 512 cycles and P V twice 512 cycles (head_dim 128), since P
// enters the product as an FP16 head plus an FP16 remainder (~22 bits, as the reference's FP32 P does).  The softmax of
// that tile takes 1024 cycles of the SM's exponential units and about 800 of its issue slots, so two tiles take turns:
// the tensor pipe works on one while the other's softmax runs.
//
//   tile      128 rows = 128/G positions x the G query heads of one KV head (row = position * G + head), so that a K/V tile
//             is fetched once for all heads that share it and a ragged end wastes at most 128/G positions.  G that does not
//             divide 128: one head per tile.  A CTA works on two consecutive tiles.
//   warps     0-3 and 4-7 softmax of tile 0 / 1, thread = row = tensor-memory lane (no shuffles); 8 TMA; 9 MMA issue
//   tensor memory   S0 | S1 (128 columns each) | O0 | O1.  P overwrites S: head in columns 0-63, remainder in 64-127 (two FP16
//             per column), and is the A operand of P V straight from tensor memory; V is the MN-major B operand as it lies.
//   rescale   the running reference maximum of a row moves only when the tile's maximum exceeds it by more than 2^8: P stays
//             below 256 (FP16 has the same relative precision there), and O is rescaled rarely instead of once per tile (the
//             idea, and that of two row tiles in turn, are FlashAttention-4's as published).
//   precision results that are not the nearest FP16 of the float64 ones, against the warp-level kernel before it (IEEE division
//             and expf): 0.97 to 1.00 of its count at scores of standard deviation 0.1 to 4 (8B heads, 16 to 4096 rows), 0.99 at 9.
//   order     P V of tile t, then Q K^T of tile t's next keys, in issue order: when S is ready, O and P of the previous keys
//             are done with, so S and P can share columns and no further barrier is needed.
//   grid      (sequence, KV head) fastest, then pairs of tiles, most keys first; one dimension, since a launch may have more
//             than 65535 pairs (2 M rows with eight heads to a tile).
// Every mbarrier wait is bounded (status word, see llmb_device_status).
#include "gemm_common.cuh"
#include "mma_common.cuh"  // pack_half2

namespace llmb {

constexpr int kPaThreads = 320;
constexpr int kPaRows = 128;      // rows of a tile
constexpr int kPaKeys = 128;      // keys of a K/V tile
constexpr int kPaStages = 2;      // K and V ring depth
constexpr float kPaLazy = 8.0f;   // log2 of the growth that P may show before the reference maximum moves

struct PrefillAttnParams {
    const __half *q;  // where it is copied without TMA
    __half *out;
    int rows;         // n_seqs * len
    int *status;
    int len;         // rows per sequence in this launch
    int pos0;        // cache position of the first of them
    int n_q_heads;
    int group;       // heads per tile (rows of a tile = 128 / group positions x group heads)
    int kv_div;      // tiles' first head / kv_div = KV head
    int head_groups; // n_q_heads / group
    int columns;     // n_seqs * head_groups
    int pairs;       // pairs of tiles per column
};

__device__ __forceinline__ void tma_load_3d(void *smem_dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

// D[128][N] += A (tensor memory, K-major) . B (shared memory)
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// MN-major operand in the 128-byte swizzle: 64 elements of MN per 128-byte row, 8 rows of K per 1024-byte group
// (stride between groups = SBO), the next 64 elements of MN `mn_stride` bytes on (LBO).
__device__ __forceinline__ uint64_t umma_desc_mn(const void *smem_tile, uint32_t mn_stride) {
    const uint64_t addr = smem_u32(smem_tile);
    return ((addr & 0x3FFFFull) >> 4) | ((uint64_t)(mn_stride >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// (a + b) and (a * b) of two FP32 values at once
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

// PLAIN: q or out does not lie on a 16-byte boundary (4 suffice): q is copied without TMA, out stored in words.  A kernel of its
// own, since the instructions that it adds are fetched cold by every launch (1.1 us of it at 37 rows).
template <int HD, bool PLAIN>
__global__ void __launch_bounds__(kPaThreads, 1)
attn_prefill_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const PrefillAttnParams p) {
    constexpr int HB = HD / 64;                                  // 64-dim boxes per row
    constexpr uint32_t kBox = kPaRows * 128;                     // 16 KB: 128 rows x 64 dims
    constexpr uint32_t kTile = HB * kBox;
    constexpr uint32_t kIdescS = (1u << 4) | ((uint32_t)(kPaKeys >> 3) << 17) | ((uint32_t)(kPaRows >> 4) << 24);
    constexpr uint32_t kIdescO = (1u << 4) | (1u << 16) | ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(kPaRows >> 4) << 24);

    extern __shared__ __align__(1024) unsigned char pa_smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(pa_smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char *q_s = smem;                                   // two tiles
    unsigned char *k_s = q_s + 2 * kTile;
    unsigned char *v_s = k_s + kPaStages * kTile;
    __shared__ __align__(8) uint64_t q_full, k_full[kPaStages], k_empty[kPaStages], v_full[kPaStages], v_empty[kPaStages];
    __shared__ __align__(8) uint64_t s_full[2], p_full[2], o_full[2];
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) uint64_t drain_bar;
    __shared__ int prior_status;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col = blockIdx.x % p.columns, pair = blockIdx.x / p.columns;
    const int seq = col / p.head_groups, hg = col % p.head_groups;
    const int head0 = hg * p.group, kvh = head0 / p.kv_div;
    const int pt = kPaRows / p.group;                            // positions per tile
    const int i0 = (p.pairs - 1 - pair) * 2 * pt;                // first row (within the sequence) of tile 0
    // tile t: rows i0 + t * pt ..; n_tiles key tiles up to its last row's own position (0: past the end)
    auto key_tiles = [&](int t) {
        const int first = i0 + t * pt, last = min(first + pt, p.len) - 1;
        return first < p.len ? (p.pos0 + last) / kPaKeys + 1 : 0;
    };
    const int n_tiles0 = key_tiles(0), n_tiles1 = key_tiles(1), n_max = max(n_tiles0, n_tiles1);

    if (threadIdx.x == 0) {
        prior_status = *reinterpret_cast<volatile int *>(p.status);
        mbar_init(&q_full, 1);
        for (int s = 0; s < kPaStages; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
        }
        for (int t = 0; t < 2; ++t) {
            mbar_init(&s_full[t], 1);
            mbar_init(&p_full[t], 4);
            mbar_init(&o_full[t], 1);
        }
        fence_mbar_init();
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    pdl_launch_dependents();                                     // this CTA has its tensor memory (see gemm_tc.cu)
    const uint32_t tmem_o = tmem + 2 * kPaKeys;                  // O tile t at + t * HD
    pdl_wait();                                                  // q and the new cache rows are the previous kernel's output
    if (PLAIN) {  // what the boxes of map_q bring, 16 bytes at a time by all threads; rows past the last one are zero
        for (int i = threadIdx.x; i < 2 * kPaRows * (HD / 8); i += kPaThreads) {
            const int t = i / (kPaRows * (HD / 8)), r = i / (HD / 8) % kPaRows, c = i % (HD / 8);
            const int row = seq * p.len + i0 + t * pt + r / p.group;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (row < p.rows) {
                const uint32_t *src = reinterpret_cast<const uint32_t *>(p.q + ((size_t)row * p.n_q_heads + head0 + r % p.group) * HD + c * 8);
                v = make_uint4(__ldcg(src), __ldcg(src + 1), __ldcg(src + 2), __ldcg(src + 3));
            }
            *reinterpret_cast<uint4 *>(q_s + t * kTile + (c >> 3) * kBox + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = v;
        }
        fence_proxy_async();
        __syncthreads();
    }

    if (prior_status != 0) {
        // a wait that gave up earlier leaves the status word set: do not queue more bounded waits behind it
    } else if (warp == 8) {
        if (lane == 0) {
            bool ok = true;
            if (PLAIN) {
                mbar_arrive(&q_full);
            } else {
                const int used = n_tiles1 > 0 ? 2 : 1;
                mbar_arrive_expect_tx(&q_full, (uint32_t)used * kTile);
                for (int t = 0; t < used; ++t)
                    for (int b = 0; b < HB; ++b)  // 128 / group positions x group heads = 128 rows
                        tma_load_3d(q_s + t * kTile + b * kBox, &map_q, b * 64, head0, seq * p.len + i0 + t * pt, &q_full);
            }
            int j = 0;
            for (; j < n_max && ok; ++j) {
                const int s = j % kPaStages;
                if (j >= kPaStages) ok = mbar_wait(&k_empty[s], ((j / kPaStages) - 1) & 1, p.status, 341);
                if (!ok) break;
                mbar_arrive_expect_tx(&k_full[s], kTile);
                for (int b = 0; b < HB; ++b) tma_load_3d(k_s + s * kTile + b * kBox, &map_k, kvh * HD + b * 64, j * kPaKeys, seq, &k_full[s]);
                if (j >= kPaStages) ok = mbar_wait(&v_empty[s], ((j / kPaStages) - 1) & 1, p.status, 342);
                if (!ok) break;
                mbar_arrive_expect_tx(&v_full[s], kTile);
                for (int b = 0; b < HB; ++b) tma_load_3d(v_s + s * kTile + b * kBox, &map_v, kvh * HD + b * 64, j * kPaKeys, seq, &v_full[s]);
            }
            if (!ok) {  // winding down: no copy of this CTA may still be in flight when it leaves
                mbar_wait(&q_full, 0, nullptr, 0);
                for (int i = max(0, j - kPaStages + 1); i <= j && i < n_max; ++i) {
                    const int s = i % kPaStages;
                    if (i < j) mbar_wait(&v_full[s], (i / kPaStages) & 1, nullptr, 0);
                    mbar_wait(&k_full[s], (i / kPaStages) & 1, nullptr, 0);
                }
            }
        }
    } else if (warp == 9) {
        if (lane == 0) {
            bool ok = mbar_wait(&q_full, 0, p.status, 343);
            auto scores = [&](int t, int j) {  // S_t = Q_t K_j^T
                const unsigned char *qt = q_s + t * kTile, *kt = k_s + (j % kPaStages) * kTile;
                const uint64_t qd = umma_desc(qt), kd = umma_desc(kt);
#pragma unroll
                for (int ks = 0; ks < HD / 16; ++ks) {
                    const uint64_t off = (uint64_t)((ks / 4) * (kBox >> 4) + (ks % 4) * 2);
                    umma_f16(tmem + t * kPaKeys, qd + off, kd + off, kIdescS, ks > 0 ? 1u : 0u);
                }
                umma_commit(&s_full[t]);
            };
            if (ok) ok = mbar_wait(&k_full[0], 0, p.status, 344);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (ok) {
                scores(0, 0);
                if (n_tiles1 > 0) scores(1, 0);
                umma_commit(&k_empty[0]);
            }
            int j = 0;
            for (; j < n_max && ok; ++j) {
                const int s = j % kPaStages;
                ok = mbar_wait(&v_full[s], (j / kPaStages) & 1, p.status, 345);
                if (ok && j + 1 < n_max) ok = mbar_wait(&k_full[(j + 1) % kPaStages], ((j + 1) / kPaStages) & 1, p.status, 346);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t vd = umma_desc_mn(v_s + s * kTile, kBox);
#pragma unroll 1
                for (int t = 0; t < 2 && ok; ++t) {
                    const int n_tiles = t ? n_tiles1 : n_tiles0;
                    if (j >= n_tiles) continue;
                    ok = mbar_wait(&p_full[t], j & 1, p.status, 347);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int ks = 0; ks < kPaKeys / 16; ++ks) {   // 16 keys = 8 columns of P = two 1024-byte groups of V
                        const uint32_t pa = tmem + t * kPaKeys + ks * 8;
                        umma_f16_ts(tmem_o + t * HD, pa, vd + (uint64_t)ks * 128, kIdescO, (j > 0 || ks > 0) ? 1u : 0u);
                        umma_f16_ts(tmem_o + t * HD, pa + 64, vd + (uint64_t)ks * 128, kIdescO, 1u);
                    }
                    if (j + 1 < n_tiles) scores(t, j + 1);
                    else umma_commit(&o_full[t]);
                }
                umma_commit(&v_empty[s]);
                if (j + 1 < n_max) umma_commit(&k_empty[(j + 1) % kPaStages]);
            }
            if (!ok) {  // the producer may have requested tiles up to two ahead, and left
                const int end = min(j + kPaStages, n_max);
                mbar_wait(&q_full, 0, nullptr, 0);
                drain_copies(k_full, kPaStages, max(0, j - 1), end);
                wind_down_mma(v_full, kPaStages, max(0, j - 1), end, &drain_bar);
            }
        }
    } else {
        // ---- softmax: thread = row of tile t ----
        const int t = warp >> 2, n_tiles = t ? n_tiles1 : n_tiles0, r = (warp & 3) * 32 + lane;
        const int i = i0 + t * pt + r / p.group;                 // row within the sequence
        const int qpos = p.pos0 + min(i, p.len - 1);
        const int qpos_first = __shfl_sync(0xffffffffu, qpos, 0);
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t ts = tmem + t * kPaKeys + lanes, to = tmem_o + t * HD + lanes;
        const float c = 1.4426950408889634f / sqrtf((float)HD);  // log2(e) / sqrt(head_dim)
        const float2 c2 = make_float2(c, c);
        float m_ref = 0.0f, l = 0.0f;
        bool ok = true;
        for (int j = 0; j < n_tiles && ok; ++j) {
            ok = mbar_wait_warp(&s_full[t], j & 1, p.status, 348, lane);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t sv[4][32];
#pragma unroll
            for (int q = 0; q < 4; ++q) tmem_ld32_async(ts + q * 32, sv[q]);
#pragma unroll
            for (int q = 0; q < 4; ++q) tmem_wait_ld32(sv[q]);
            float s[kPaKeys];
#pragma unroll
            for (int e = 0; e < kPaKeys; ++e) s[e] = __uint_as_float(sv[e >> 5][e & 31]);
            const int kv0 = j * kPaKeys;
            if (kv0 + kPaKeys - 1 > qpos_first) {                // causal mask, on the last tiles only
                const int lim = qpos - kv0;
#pragma unroll
                for (int e = 0; e < kPaKeys; ++e) s[e] = e <= lim ? s[e] : -INFINITY;
            }
            float mx[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) mx[q] = fmaxf(s[q], s[q + 4]);
#pragma unroll
            for (int e = 8; e < kPaKeys; ++e) mx[e & 3] = fmaxf(mx[e & 3], s[e]);
            const float tmax = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            if (j == 0) {
                m_ref = tmax;                                    // key 0 is visible to every row: finite
            } else if (__any_sync(0xffffffffu, (tmax - m_ref) * c > kPaLazy)) {
                // O and P of the earlier keys are complete: their MMAs were issued before this S
                const float m_new = (tmax - m_ref) * c > kPaLazy ? tmax : m_ref;
                const float scale = ex2((m_ref - m_new) * c);
                m_ref = m_new;
                l *= scale;
#pragma unroll 1
                for (int q = 0; q < HD / 16; ++q) {
                    uint32_t o[16];
                    tmem_ld16(to + q * 16, o);
#pragma unroll
                    for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * scale);
                    tmem_st16(to + q * 16, o);
                }
            }
            const float2 nm2 = make_float2(-m_ref, -m_ref);
            float2 sum0 = make_float2(0.0f, 0.0f), sum1 = sum0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    float2 a = mul2(add2(make_float2(s[q * 32 + 2 * e], s[q * 32 + 2 * e + 1]), nm2), c2);
                    a.x = ex2(a.x);
                    a.y = ex2(a.y);
                    if (e & 1) sum1 = add2(sum1, a);
                    else sum0 = add2(sum0, a);
                    const __half2 h = __floats2half2_rn(a.x, a.y);
                    const float2 f = __half22float2(h);
                    hi[e] = *reinterpret_cast<const uint32_t *>(&h);
                    lo[e] = pack_half2(a.x - f.x, a.y - f.y);
                }
                tmem_st16(ts + q * 16, hi);
                tmem_st16(ts + 64 + q * 16, lo);
            }
            l += (sum0.x + sum0.y) + (sum1.x + sum1.y);
            tmem_wait_st();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[t]);
        }
        if (n_tiles > 0 && ok) {
            ok = mbar_wait_warp(&o_full[t], 0, p.status, 349, lane);
            if (!ok) mbar_wait(&o_full[t], 0, nullptr, 0);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            __half *dst = p.out + ((size_t)(seq * p.len + min(i, p.len - 1)) * p.n_q_heads + head0 + r % p.group) * HD;
#pragma unroll 1
            for (int q = 0; q < HD / 32 && ok; ++q) {
                uint32_t o[32];
                __syncwarp();  // see tmem_ld32
                tmem_ld32(to + q * 32, o);
                if (i < p.len) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        uint4 w;
                        uint32_t *pw = reinterpret_cast<uint32_t *>(&w);
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            pw[u] = pack_half2(__fdiv_rn(__uint_as_float(o[8 * e + 2 * u]), l), __fdiv_rn(__uint_as_float(o[8 * e + 2 * u + 1]), l));
                        if (!PLAIN) {
                            reinterpret_cast<uint4 *>(dst + q * 32)[e] = w;
                        } else {
#pragma unroll
                            for (int u = 0; u < 4; ++u) reinterpret_cast<uint32_t *>(dst + q * 32 + 8 * e)[u] = pw[u];
                        }
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 9) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

int launch_attn_prefill(const __half *q, const __half *k_cache, const __half *v_cache, int n_seqs, size_t seq_stride, int len, int pos0,
                        int n_q_heads, int n_kv_heads, int head_dim, __half *out, bool pdl, cudaStream_t stream) {
    PrefillAttnParams p = {};
    p.out = out;
    p.q = q;
    p.rows = n_seqs * len;
    p.status = device_status_ptr();
    if (!p.status) return LLMB_ERR_CUDA;
    const int G = n_q_heads / n_kv_heads;
    p.len = len;
    p.pos0 = pos0;
    p.n_q_heads = n_q_heads;
    p.group = (G <= 8 && (G & (G - 1)) == 0) ? G : 1;  // 128 rows = whole positions; 8 consecutive rows stay one swizzle group
    p.kv_div = G;
    p.head_groups = n_q_heads / p.group;
    const int pt = kPaRows / p.group;
    // rows of a sequence past its last one (pos0 + len) lie outside the map and read as zero: what an earlier, longer
    // sequence left in the cache never meets the zero probabilities of the masked keys
    CUtensorMap mq, mk, mv;
    int rc;
    const int n_kv = n_kv_heads * head_dim;
    if ((rc = make_map_3d(&mk, k_cache, n_kv, pos0 + len, n_seqs, (size_t)n_kv, seq_stride, kPaKeys, 1))) return rc;
    if ((rc = make_map_3d(&mv, v_cache, n_kv, pos0 + len, n_seqs, (size_t)n_kv, seq_stride, kPaKeys, 1))) return rc;
    const bool plain = (((uintptr_t)q | (uintptr_t)out) & 15) != 0;
    if (plain) mq = mk;  // not used
    else if ((rc = make_map_3d(&mq, q, head_dim, n_q_heads, n_seqs * len, (size_t)head_dim, (size_t)n_q_heads * head_dim, p.group, pt))) return rc;
    p.columns = n_seqs * p.head_groups;
    p.pairs = (int)(((long long)len + 2 * pt - 1) / (2 * pt));
    if ((long long)p.columns * p.pairs > 0x7fffffffll) return LLMB_ERR_UNSUPPORTED;
    const dim3 grid((unsigned)(p.columns * p.pairs));
    const size_t smem = (size_t)(2 + 2 * kPaStages) * kPaRows * head_dim * sizeof(__half) + 1024;
    auto kernel = head_dim == 128 ? (plain ? attn_prefill_kernel<128, true> : attn_prefill_kernel<128, false>)
                                  : (plain ? attn_prefill_kernel<64, true> : attn_prefill_kernel<64, false>);
    static size_t attr_set[4][kMaxDevices] = {};  // per instantiation and device
    LLMB_CUDA_OK(ensure_dynamic_smem(kernel, attr_set[(head_dim == 128 ? 2 : 0) + (plain ? 1 : 0)], smem));
    LLMB_CUDA_OK(launch_pdl(kernel, grid, dim3(kPaThreads), smem, stream, pdl, mq, mk, mv, p));
    return LLMB_OK;
}

}  // namespace llmb

extern "C" int llmb_attn_prefill(const uint16_t *d_q, const uint16_t *d_k_cache, const uint16_t *d_v_cache, int m, int pos0,
                                 int n_q_heads, int n_kv_heads, int head_dim, uint16_t *d_out, llmb_stream_t stream_) {
    using namespace llmb;
    if (!d_q || !d_k_cache || !d_v_cache || !d_out || m <= 0 || pos0 < 0 || n_q_heads <= 0 || n_kv_heads <= 0 ||
        n_q_heads % n_kv_heads)
        return LLMB_ERR_INVALID;
    if (n_q_heads > 65535) return LLMB_ERR_UNSUPPORTED;
    if (head_dim != 64 && head_dim != 128) {
        set_last_error("llmb_attn_prefill: head_dim must be 64 or 128");
        return LLMB_ERR_UNSUPPORTED;
    }
    if ((((uintptr_t)d_q | (uintptr_t)d_out) & 3) || (((uintptr_t)d_k_cache | (uintptr_t)d_v_cache) & 15) || (long long)pos0 + m >= (1ll << 31)) {
        set_last_error("llmb_attn_prefill: the caches must be 16-byte aligned, q and out 4-byte aligned");
        return LLMB_ERR_UNSUPPORTED;
    }
    const size_t n_kv = (size_t)n_kv_heads * head_dim;
    return launch_attn_prefill(reinterpret_cast<const __half *>(d_q), reinterpret_cast<const __half *>(d_k_cache),
                               reinterpret_cast<const __half *>(d_v_cache), 1, (size_t)(pos0 + m) * n_kv, m, pos0, n_q_heads, n_kv_heads,
                               head_dim, reinterpret_cast<__half *>(d_out), false, static_cast<cudaStream_t>(stream_));
}
