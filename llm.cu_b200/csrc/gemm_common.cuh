// Pieces shared by the tensor-core projection kernels (gemm_tc.cu: blocks of rows; gemm_smallm.cu: a handful of
// rows with the weights as the 128-row operand): tile constants, the parameter block, tcgen05 / TMA wrappers
// and the host-side tensor-map builder.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace llmb {

constexpr int kBM = 128, kBK = 64;
constexpr int kGemmThreads = 192;
constexpr uint32_t kATileBytes = kBM * kBK * 2;  // 16 KB: the A tile of a stage
constexpr int kGemmMaxStages = 8;
// Ring depth: two CTAs share an SM when the grid has more CTAs than SMs (3 stages each, 2 for SwiGLU);
// a grid that leaves every CTA alone on its SM gets a ring as deep as shared memory allows, because
// then the copy latency is hidden by nothing but the ring.
__host__ __device__ constexpr int gemm_stages(bool dual) { return dual ? 2 : 3; }
__host__ __device__ constexpr uint32_t gemm_stage_bytes(bool dual, int bn) { return kATileBytes + (dual ? 2 : 1) * bn * kBK * 2; }

struct GemmParams {
    __half *c;              // STORE/RESIDUAL/SWIGLU: [M][N] (SWIGLU: N = ffn); ROPE_KV: q [M][n_q]
    const float2 *rope_cs;  // ROPE_KV: [M][head_dim / 2]
    __half *k_cache, *v_cache;
    int *status;
    int M, N, K, epilogue;
    int n_q, n_kv, head_dim, pos0, max_pos;
    const int *row_pos;  // ROPE_KV, batched decode: cache position of each row; row r belongs to sequence r
    long long seq_stride;  // cache rows between consecutive sequences
    int rows_per_seq;      // ROPE_KV without row_pos: row r = position pos0 + r % rows_per_seq of sequence r / rows_per_seq
    int nx;      // small-M kernel: columns of the MMA, the activation rows rounded up to 32
    int stages;  // ring depth of this launch (<= kGemmMaxStages)
    // split-K: blockIdx.z takes a slice of K, partial accumulators meet in the workspace and the last
    // CTA of a tile to arrive adds them in slice order and runs the epilogue
    int splits;
    float *ws_part;  // [tiles][splits][128][accumulator columns]
    int *ws_count;   // [tiles], zero between launches
    // LLMB_EPI_TP_SCATTER (small-M kernel): the output is this rank's partial sum of a row-parallel projection;
    // it goes, tagged, into every rank's exchange block instead of memory of its own (tp_common.cuh)
    unsigned char *tp_peer[8];
    const unsigned int *tp_seq;  // device: exchanges completed before this step
    int tp_rank, tp_size, tp_index;  // this exchange is number tp_index of the step
    unsigned long long *trace;  // optional profiling aid (small-M kernel): [CTA][8] global-timer stamps
};

__device__ __forceinline__ uint64_t umma_desc(const void *smem_tile) {
    // K-major, 128-byte swizzle: rows are 128 bytes, 8-row groups are 1024 bytes apart (SBO);
    // descriptor version 1 (sm_100), layout type 2 = SWIZZLE_128B.
    const uint64_t addr = smem_u32(smem_tile);
    return ((addr & 0x3FFFFull) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void tma_load_2d(void *smem_dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Winding down after a wait of this CTA gave up: no copy into its shared memory and no MMA on its tensor memory may be under
// way when it leaves, so whoever gave up waits again, without a status, for what may be: the thread that requests copies
// for the stages it has requested, the one that issues MMAs for those that may have been and for its MMAs, the
// epilogue for the accumulator.  Only where a wait has given up: the same waits on every launch, or a flag that all threads
// look at behind the last barrier, cost 0.3 to 0.4 us a launch (instructions fetched cold on the way out).
__device__ __forceinline__ void drain_copies(uint64_t *full_bar, int stages, int first, int end) {  // ring stages first .. end - 1
    for (int i = first; i < end; ++i) mbar_wait(&full_bar[i % stages], (i / stages) & 1, nullptr, 0);
}

// The MMA thread's: drain_bar is used for nothing else.
static __device__ __noinline__ void wind_down_mma(uint64_t *full_bar, int stages, int first, int end, uint64_t *drain_bar) {
    drain_copies(full_bar, stages, first, end);
    mbar_init(drain_bar, 1);
    fence_mbar_init();
    umma_commit(drain_bar);
    mbar_wait(drain_bar, 0, nullptr, 0);
}

// Tensor-memory loads are one instruction of a converged warp.  An epilogue that comes to one from masked stores, a `continue` for
// rows past the end or a wait that each lane polls for itself joins the warp first (__syncwarp or a vote), instead of leaving it
// to where the compiler brings the lanes together again.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The load alone; its registers hold nothing until tmem_wait_ld32 on them (the first such wait completes every load
// of the thread, the others only keep the compiler from using their registers earlier).
__device__ __forceinline__ void tmem_ld32_async(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void tmem_wait_ld32(uint32_t (&v)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]),
                   "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]), "+r"(v[16]),
                   "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]),
                   "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31])
                 :
                 : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ uint32_t cluster_cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// Every thread of every CTA of the cluster arrives; returns when all have (a hardware barrier: no spin of ours).
__device__ __forceinline__ void cluster_sync_all() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

__device__ __forceinline__ float silu_gemm(float x) { return __fdiv_rn(x, 1.0f + expf(-x)); }


// Position and cache row of row `row` of a ROPE_KV launch.
__device__ __forceinline__ int kv_position(const GemmParams &p, int row, size_t &cache_row) {
    if (p.row_pos) {
        const int pos = __ldg(p.row_pos + row);
        cache_row = (size_t)row * (size_t)p.seq_stride + (size_t)pos;
        return pos;
    }
    const int seq = row / p.rows_per_seq, pos = p.pos0 + (row - seq * p.rows_per_seq);
    cache_row = (size_t)seq * (size_t)p.seq_stride + (size_t)pos;
    return pos;
}

// Epilogue of 32 accumulator columns (col0 .. col0 + 31, a multiple of 32) of one output row; u = the second
// accumulator (up) of a SwiGLU projection.
template <bool DUAL>
__device__ __forceinline__ void finish_cols(const GemmParams &p, int row, int col0, const uint32_t (&v)[32], const uint32_t (&u)[32]) {
    __align__(16) __half out[32];
    if (DUAL) {
#pragma unroll
        for (int i = 0; i < 32; ++i) out[i] = __float2half_rn(silu_gemm(__uint_as_float(v[i])) * __uint_as_float(u[i]));
        uint4 *dst = reinterpret_cast<uint4 *>(p.c + (size_t)row * p.N + col0);
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = reinterpret_cast<const uint4 *>(out)[i];
    } else if (p.epilogue == LLMB_EPI_STORE) {
#pragma unroll
        for (int i = 0; i < 32; ++i) out[i] = __float2half_rn(__uint_as_float(v[i]));
        uint4 *dst = reinterpret_cast<uint4 *>(p.c + (size_t)row * p.N + col0);
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = reinterpret_cast<const uint4 *>(out)[i];
    } else if (p.epilogue == LLMB_EPI_RESIDUAL) {
        uint4 *dst = reinterpret_cast<uint4 *>(p.c + (size_t)row * p.N + col0);
        __align__(16) __half res[32];
#pragma unroll
        for (int i = 0; i < 4; ++i) reinterpret_cast<uint4 *>(res)[i] = dst[i];
#pragma unroll
        for (int i = 0; i < 32; ++i)
            out[i] = __float2half_rn(__half2float(__float2half_rn(__uint_as_float(v[i]))) + __half2float(res[i]));
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = reinterpret_cast<const uint4 *>(out)[i];
    } else {  // LLMB_EPI_ROPE_KV
        size_t cache_row;
        const int pos = kv_position(p, row, cache_row);
        const int half_dim = p.head_dim >> 1;
        const bool is_v = col0 >= p.n_q + p.n_kv;
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
            const float e = __half2float(__float2half_rn(__uint_as_float(v[i])));
            const float o = __half2float(__float2half_rn(__uint_as_float(v[i + 1])));
            if (is_v) {
                out[i] = __float2half_rn(__uint_as_float(v[i]));
                out[i + 1] = __float2half_rn(__uint_as_float(v[i + 1]));
            } else {
                const int local = (col0 < p.n_q ? col0 : col0 - p.n_q) + i;
                const float2 cs = p.rope_cs[(size_t)row * half_dim + ((local >> 1) % half_dim)];
                out[i] = __float2half_rn(__fmaf_rn(cs.x, e, -__fmul_rn(cs.y, o)));
                out[i + 1] = __float2half_rn(__fmaf_rn(cs.y, e, __fmul_rn(cs.x, o)));
            }
        }
        __half *dstp = nullptr;
        if (col0 < p.n_q) dstp = p.c + (size_t)row * p.n_q + col0;
        else if (pos >= 0 && pos < p.max_pos)
            dstp = (is_v ? p.v_cache + cache_row * p.n_kv + (col0 - p.n_q - p.n_kv)
                         : p.k_cache + cache_row * p.n_kv + (col0 - p.n_q));
        if (dstp) {
#pragma unroll
            for (int i = 0; i < 4; ++i) reinterpret_cast<uint4 *>(dstp)[i] = reinterpret_cast<const uint4 *>(out)[i];
        }
    }
}

// [rows][k] FP16 row-major as a 2-D tensor map with a 64 x box_rows box and 128-byte swizzle (gemm_tc.cu).  L2 fetches 256 bytes at a
// time: the next K step of a row is needed next, and HBM gives more in longer runs (a stream of 128-row boxes from two CTAs per
// SM 5.4 TB/s with 128 bytes, 5.9 with 256; batched steps of 5 x 333 / 32 x 1024 / 96 x 200 3.63 / 4.54 / 5.15 -> 3.43 / 4.39 / 5.08 ms).
int make_map(CUtensorMap *map, const void *base, int rows, int k, int box_rows);

// [d2][d1][d0] FP16 with strides of d1 and d2 in elements (d0 contiguous) as a 3-D tensor map, box 64 x box1 x box2 in
// the 128-byte swizzle; what lies outside reads as zero.
int make_map_3d(CUtensorMap *map, const void *base, int d0, int d1, int d2, size_t stride1, size_t stride2, int box1, int box2);

// llmb_gemm_f16 for callers inside the library.  rows_per_seq > 0 (ROPE_KV without row_pos): the m rows are the
// positions pos0 .. of m / rows_per_seq sequences, one after the other, whose caches are seq_stride rows apart.
// pdl: programmatic stream serialization at any m (the weights must not be the previous kernel's output).
int launch_gemm(const LlmbGemmArgs *a, int rows_per_seq, bool pdl, cudaStream_t stream);

// What every path of launch_gemm passes on of its arguments (gemm_tc.cu).
int fill_gemm_params(GemmParams &p, const LlmbGemmArgs *a, int rows_per_seq);

// The path for tiles that are one wave (gemm_mid.cu), and whether it takes this one.
bool gemm_mid_takes(const LlmbGemmArgs *a);
int launch_gemm_mid(const LlmbGemmArgs *a, int rows_per_seq, bool pdl, cudaStream_t stream);

// The path for grids of many tiles (gemm_wide.cu), and whether it takes this one.
bool gemm_wide_takes(const LlmbGemmArgs *a);
int launch_gemm_wide(const LlmbGemmArgs *a, int rows_per_seq, bool pdl, cudaStream_t stream);

// Its small-M path (gemm_smallm.cu): m <= kSmallM rows.
constexpr int kSmallM = 128;
int launch_gemm_smallm(const LlmbGemmArgs *a, int rows_per_seq, bool pdl, cudaStream_t stream);

// llmb_attn_decode_batch where no caller has chosen the length of a piece: pieces of `split_len` rows, but no shorter than the
// longest sequence if that has at most `whole_rows` (attn_decode.cu).
int launch_attn_decode_batch(const uint16_t *d_q, const uint16_t *d_k_cache, const uint16_t *d_v_cache, const int32_t *d_pos, int n_seqs,
                             size_t seq_stride_rows, int n_q_heads, int n_kv_heads, int head_dim, int n_splits, int split_len,
                             int whole_rows, uint16_t *d_out, void *d_scratch, int use_pdl, llmb_stream_t stream);

// Causal attention of `len` new rows of each of n_seqs sequences (attn_prefill.cu); the caches of consecutive
// sequences are seq_stride elements apart, q and out are [n_seqs * len][n_q_heads * head_dim].
int launch_attn_prefill(const __half *q, const __half *k_cache, const __half *v_cache, int n_seqs, size_t seq_stride, int len, int pos0,
                        int n_q_heads, int n_kv_heads, int head_dim, __half *out, bool pdl, cudaStream_t stream);

// llmb_rmsnorm_rows; gains_ready: no kernel of the stream writes gamma, so it may be read before the previous one is complete
// (prefill.cu).
int launch_rmsnorm_rows(const uint16_t *x, const uint16_t *gamma, uint16_t *y, int m, int d, double eps, bool gains_ready, bool pdl,
                        cudaStream_t stream);

// llmb_embed_rope for a block of n_seqs * len rows: positions pos0 .. pos0 + len - 1 of each sequence, sequence s with its
// ids (position 0 first) at tokens + s * token_stride (misc.cu).
int launch_embed_rows(const __half *embed, const int *tokens, size_t token_stride, int n_seqs, int len, int pos0, int d_model,
                      int vocab, int head_dim, float theta, __half *x, float *rope_cs, bool pdl, cudaStream_t stream);

}  // namespace llmb
