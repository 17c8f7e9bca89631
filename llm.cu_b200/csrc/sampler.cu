// Temperature / top-k / top-p sampling on the device: the reference's host chain sample_next_token ->
// temperature_softmax -> top_k_sampling -> top_p_sampling (src/inference/inference.cu:1030-1161) as one
// kernel over the FP16 logits a decode step leaves in device memory, so that a sampled decode needs no
// 256 KB device-to-host copy of the logits per token.
//
//   t_i = expf(float(logit_i) / temperature);  p_i = t_i / sum(t)             (:1041-1061, no maximum subtracted)
//   order by p descending, ties to the lower index                            (:1059, qsort with ties unspecified)
//   the first top_k entries are renormalised to sum 1                         (:1088-1096; its own pick is discarded)
//   the shortest prefix whose running sum reaches top_p is renormalised       (:1131-1148)
//   the first entry whose running sum exceeds u is returned, entry 0 if none  (:1154-1160)
//
// One cluster of 8 CTAs of 1024 threads (calls are one row each, so a row has to spread over several SMs itself).
// Bound: latency of a chain of dependent passes; the data (256 KB for the 8B vocabulary) is 1/8 per CTA.
//   t_i, sum   the vocabulary entries fall into 1024 classes i mod 1024; CTA c owns classes 128 c .. 128 c + 127 and keeps
//              their t_i in shared memory (the caller's scratch for vocabularies beyond kSamplerSmemRows rows).  A class is
//              added in index order by one thread, 32 classes by a warp butterfly, the 32 warps' sums by another: the
//              sum does not depend on how many CTAs share the work.
//   order      only the first `want` entries can matter: top_k of them, or kSamplerMaxSelect where top_p is so close to 1
//              that rounding may carry the prefix past the first top_k (see want_entries).  Whoever adds a class also keeps its
//              largest t_i; as many entries as classes reach the `want`th largest of these, so the entries that do (usually not
//              many more than wanted) go to CTA 0, which sorts them: one pass over the t_i without division or histogram.  Where
//              nearly all classes or more than kSamplerCap entries do, where more than half as many entries as classes are wanted or the
//              vocabulary is small, a radix select over the 64-bit key (bits of p, then inverted index, so that keys are unique and
//              equal p keep index order) finds a key prefix that between `want` and kSamplerCap entries reach.
//   chain      the reference's statements on CTA 0: the running sums are one thread's, in the reference's order; the
//              divisions between them are elementwise and use all threads.
// Taking the entries one at a time by a block-wide argmax on a single CTA (every round: two barriers, and the owner's
// rescan of its entries) took 495 us a draw at top_k 50 over 128256 entries; this form takes 14.4 us (18.5 with the radix
// select for all, whose time depends on how the logits are spread; 20 before short lists were ranked by counting and the running sums lost their load and branch per entry).
// Different from the host code: the sum of the t_i is a tree over classes, not a loop in index order, and expf is CUDA's,
// so probabilities can differ from the host's by a few FP32 ulps; the token differs only if u lies within that distance
// of a boundary between two entries.
#include <climits>

#include "common.cuh"
#include "../../include/llm_b200_synth.h"

namespace llmb {

constexpr int kSamplerThreads = 1024;
constexpr int kSamplerMaxSelect = 1024;
constexpr int kSamplerCtas = 8;                                        // one portable cluster
constexpr int kSamplerClasses = 1024;                                  // summation classes (index mod 1024)
constexpr int kClassesPerCta = kSamplerClasses / kSamplerCtas;         // 128
constexpr int kRowsPerPass = kSamplerThreads / kClassesPerCta;         // 8 rows of a CTA's classes at a time
constexpr int kSamplerCap = 2048;                                      // entries that CTA 0 sorts at most
constexpr int kSamplerSmemRows = 384;                                  // 192 KB of t_i per CTA: vocabularies up to 393216
constexpr int kSamplerBins = 1024;
constexpr int kClassBinWords = 1024;                                   // 4096 bins of the classes' largest t_i
constexpr int kClassesListed = 880;  // classes whose largest entry reaches the floor, at most, for the list to be tried (see the kernel)
constexpr int kRankThreads = 4, kSamplerRankCap = kSamplerThreads / kRankThreads;  // up to 256 keys are ranked by counting

struct SamplerParams {
    const __half *logits;
    float *probs;   // [vocab] scratch
    int *token_out;
    int *pos;       // optional: history[*pos] = token (the position the decode step has already advanced to)
    int *history;
    int history_len;
    int *result;    // 0 ok, 1 overflow, 2 prefix longer than kSamplerMaxSelect; then, where it is 0: entries ordered, 1 if the classes led to them
    int vocab, top_k;
    int want;       // entries of the order that may be needed, top_k <= want <= kSamplerMaxSelect
    int in_smem;    // t_i in shared memory (else in probs)
    float temperature, top_p, u;
};

// Entries of the descending order that the chain can need.  The first k are renormalised to sum 1: their running sum
// ends within 2 k 2^-24 < 1.3e-4 of 1 (k <= 1024 additions and as many divisions, each off by at most 2^-24), so the
// prefix that reaches a top_p below 0.99 ends inside them.
inline int want_entries(int vocab, int top_k, float top_p) {
    if (top_p < 0.99f) return top_k;
    return vocab < kSamplerMaxSelect ? vocab : kSamplerMaxSelect;
}

__device__ __forceinline__ uint32_t sampler_cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ void sampler_cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// A CTA's shared memory may be touched by another one only once it is known to have started: every thread arrives at entry,
// without ordering anything, and waits before the first access to a peer, by when all have long arrived.
__device__ __forceinline__ void sampler_cluster_started_arrive() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
}
__device__ __forceinline__ void sampler_cluster_started_wait() {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

__device__ __forceinline__ uint32_t peer_smem(const void *own, uint32_t cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(own)), "r"(cta));
    return r;
}

__device__ __forceinline__ uint64_t sample_key(float pr, int i) {
    return ((uint64_t)__float_as_uint(pr) << 32) | (uint32_t)(0xffffffffu - (uint32_t)i);
}

// Bins of the classes' largest t_i: 16 to an octave over all of FP32, so that the scale of the logits and the temperature do not
// matter.  A CTA has 128 classes: a bin's count is a byte, four bins a word.
constexpr int kClassBinShift = 19;
__device__ __forceinline__ int class_bin(float t) { return (int)(__float_as_uint(t) >> kClassBinShift); }

// Index of the first entry whose running sum (in order, one rounding per entry) satisfies `hit`, -1 if none does; `run` =
// the running sum up to it (or of all n).  No probability is negative, so a sum of eight is looked at only if its last
// running value hits: the chain is then one addition per entry, not a load, an addition and a branch.
template <typename Hit>
__device__ __forceinline__ int first_reaching(const float *v, int n, float &run, const Hit &hit) {
    int i = 0;
    for (; i + 8 <= n; i += 8) {
        float c[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) c[j] = v[i + j];
        c[0] += run;
#pragma unroll
        for (int j = 1; j < 8; ++j) c[j] += c[j - 1];
        if (hit(c[7])) break;
        run = c[7];
    }
    for (; i < n; ++i) {
        run += v[i];
        if (hit(run)) return i;
    }
    return -1;
}

// LOADS of a thread in flight at first: sixteen over 128256 entries take 2 us less than eight; a thread with fewer rows works through the
// empty ones, 0.8 us over 8193 entries with sixteen instead of four.  One instantiation each, and one without the classes: a draw runs
// through its code once, so code that it passes by costs too (0.1 to 0.2 us).
template <bool BY_CLASS, int LOADS>
__global__ void __launch_bounds__(kSamplerThreads) sample_kernel(const SamplerParams p) {
    extern __shared__ float t_smem[];               // [rows][128] t_i, then p_i, of this CTA's classes
    __shared__ float warp_sums[32];                 // of all CTAs
    __shared__ int hist[kSamplerBins];
    __shared__ unsigned int class_hist[kClassBinWords];
    __shared__ int scan_s[32];
    __shared__ int bin_s, above_s, count_s;         // threshold bin, entries above it, entries from it on
    __shared__ int n_list;                          // CTA 0: entries collected
    __shared__ int over_s;                          // the list is full
    __shared__ uint64_t list[kSamplerCap];          // CTA 0
    __shared__ float sel_p[kSamplerMaxSelect];
    __shared__ float sum_s;
    __shared__ int cutoff_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t cta = sampler_cta_rank();
    sampler_cluster_started_arrive();
    pdl_launch_dependents();
    pdl_wait();

    // ---- t_i of this CTA's classes: thread = class cls, rows row0, row0 + 8, ... ----
    const int cls = (int)cta * kClassesPerCta + (tid & (kClassesPerCta - 1)), row0 = tid / kClassesPerCta;
    const int rows = (p.vocab + kSamplerClasses - 1) / kSamplerClasses;
    // element (row, class) of the vocabulary: t[row * t_stride + (class within the CTA)]
    float *t = p.in_smem ? t_smem : p.probs + (size_t)cta * kClassesPerCta;
    const int t_stride = p.in_smem ? kClassesPerCta : kSamplerClasses, col = tid & (kClassesPerCta - 1);
    for (int base = row0; base < rows; base += LOADS * kRowsPerPass) {
        __half x[LOADS];
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int row = base + j * kRowsPerPass, i = row * kSamplerClasses + cls;
            x[j] = row < rows && i < p.vocab ? p.logits[i] : __half(0.0f);
        }
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int row = base + j * kRowsPerPass, i = row * kSamplerClasses + cls;
            if (row < rows && i < p.vocab) t[(size_t)row * t_stride + col] = expf(__fdiv_rn(__half2float(x[j]), p.temperature));
        }
    }
    hist[tid] = 0;
    if (BY_CLASS) class_hist[tid] = 0;
    if (tid == 0) {
        n_list = 0;
        over_s = 0;
    }
    __syncthreads();
    sampler_cluster_started_wait();
    float most = 0.0f;  // of the class `tid` (of the CTA)
    if (tid < kClassesPerCta) {  // here col == tid
        float local = 0.0f;
        const int n = cls < p.vocab ? (p.vocab - cls + kSamplerClasses - 1) / kSamplerClasses : 0;
#pragma unroll 8
        for (int row = 0; row < n; ++row) {
            const float v = t[(size_t)row * t_stride + col];
            local += v;
            most = fmaxf(most, v);
        }
        if (BY_CLASS && n > 0) {
            const int bin = class_bin(most);
            atomicAdd(&class_hist[bin >> 2], 1u << ((bin & 3) * 8));
        }
        local = warp_sum(local);
        if (lane < kSamplerCtas)  // the same value in all lanes: lane c tells CTA c
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(peer_smem(&warp_sums[cta * (kClassesPerCta / 32) + warp], lane)), "f"(local) : "memory");
    }
    sampler_cluster_sync();
    const float total = warp_sum(warp_sums[lane]);
    if (!(total > 0.0f) || isinf(total) || isnan(total)) {  // the same in every thread of the cluster
        if (cta == 0 && tid == 0) { p.token_out[0] = -1; p.result[0] = 1; }
        return;
    }

    int inc, cnt;
    auto scan = [&]() {  // inc = the sum of cnt over this thread and those before it
        inc = cnt;
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, inc, m);
            if (lane >= m) inc += o;
        }
        if (lane == 31) scan_s[warp] = inc;
        __syncthreads();
        inc += __reduce_add_sync(0xffffffffu, lane < warp ? scan_s[lane] : 0);
    };
    auto count_down = [&]() {  // thread b holds bin 1023 - b of all CTAs: the scan counts the entries of that bin and all higher ones
        cnt = 0;
#pragma unroll
        for (int z = 0; z < kSamplerCtas; ++z) {
            int v;
            asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(peer_smem(&hist[kSamplerBins - 1 - tid], z)) : "memory");
            cnt += v;
        }
        scan();
    };
    const uint32_t n_list0 = peer_smem(&n_list, 0), list0 = peer_smem(list, 0);
    auto take = [&](uint64_t key) {
        int at;
        asm volatile("atom.relaxed.cluster.shared::cluster.add.s32 %0, [%1], 1;" : "=r"(at) : "r"(n_list0) : "memory");
        if (at < kSamplerCap) {
            asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(list0 + (uint32_t)at * 8), "l"(key) : "memory");
        } else if (at == kSamplerCap) {  // one thread of the cluster tells all CTAs
            for (int z = 0; z < kSamplerCtas; ++z) asm volatile("st.shared::cluster.s32 [%0], 1;" ::"r"(peer_smem(&over_s, z)) : "memory");
        }
    };

    // ---- the entries that can matter, from the classes' largest ones ----
    // As many entries reach F as classes' largest ones do: F = the lower end of the bin that holds the `want`th largest of these.
    // Division by the total keeps the order but may join neighbours, so whoever reaches F / total as a probability is taken; the
    // division is left out where t_i is further below F than its rounding.
    // Entries fall into classes as if by lot, so where c of the 1024 classes reach F, about -1024 ln(1 - c / 1024) entries do.  CTA 0 ranks
    // up to 256 entries by counting (c = 226) and sorts more with a network of 512, 1024 (c = 403, 647) or 2048, 4 us and more each, so
    // where the bin lets more classes pass than the wanted entries need, the next ten bits of its classes' largest are counted too
    // (1.6 us).  Above kClassesListed (logits that are all alike; the list's 2048 entries are c = 885) the list is not tried.  us a
    // draw, graph of 50, with the radix select alone / so, top_k 50: deviation 1.3 at temperature 0.7 over 32768 / 65536 / 128256 / 200000 entries
    // 9.3 / 8.6, 11.7 / 10.5, 16.6 / 13.0, 22.1 / 16.8; over 128256 at temperature 0.1 18.0 / 12.5, about -20 16.5 / 12.8, deviation 0.05 21.3 / 14.7, 0.01 21.6 / 14.7,
    // all equal 41.2 / 44.0, 20 not masked 46.6 / 48.6, 3224 equal ones on top in 224 classes (the list is tried and full) 37.4 / 44.8.
    bool listed = false, finer = false;
    uint32_t floor_bits = 0;
    if (BY_CLASS) {
        uint32_t even = 0, odd = 0;  // of four bins: counts of the first and the third, of the second and the fourth
#pragma unroll
        for (int z = 0; z < kSamplerCtas; ++z) {
            uint32_t v;
            asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(peer_smem(&class_hist[kClassBinWords - 1 - tid], z)) : "memory");
            even += v & 0x00ff00ffu;
            odd += (v >> 8) & 0x00ff00ffu;
        }
        const int c[4] = {(int)(even & 0xffff), (int)(odd & 0xffff), (int)(even >> 16), (int)(odd >> 16)};
        cnt = c[0] + c[1] + c[2] + c[3];
        scan();
        if (inc >= p.want && inc - cnt < p.want) {
            int reach = inc - cnt, bin = 0, above = 0;
#pragma unroll
            for (int j = 3; j >= 0; --j) {
                if (reach < p.want) {
                    above = reach;
                    reach += c[j];
                    bin = 4 * (kClassBinWords - 1 - tid) + j;
                }
            }
            bin_s = bin;
            above_s = above;
            count_s = reach;
        }
        __syncthreads();
        // all of this the same in all CTAs
        floor_bits = (uint32_t)bin_s << kClassBinShift;
        int classes = count_s;
        if (bin_s > 0 && classes > (p.want <= 200 ? 220 : p.want <= 390 ? 400 : 640)) {
            finer = true;
            const int need = p.want - above_s, above = above_s;
            if (tid < kClassesPerCta && class_bin(most) == bin_s) atomicAdd(&hist[(__float_as_uint(most) >> (kClassBinShift - 10)) & (kSamplerBins - 1)], 1);
            sampler_cluster_sync();
            count_down();
            if (inc >= need && inc - cnt < need) {
                bin_s = kSamplerBins - 1 - tid;
                count_s = above + inc;
            }
            __syncthreads();
            floor_bits |= (uint32_t)bin_s << (kClassBinShift - 10);
            classes = count_s;
            if (classes > kClassesListed) sampler_cluster_sync();  // every CTA has read the histograms
        }
        listed = classes <= kClassesListed;
    }
    if (listed) {
        const float floor_t = __uint_as_float(floor_bits), floor_p = __fdiv_rn(floor_t, total);
        const float near_t = floor_p > 1e-30f ? floor_t * 0.999999f : 0.0f;  // a quotient with fewer bits joins more
        for (int base = row0; base < rows; base += 4 * kRowsPerPass) {
            if (*reinterpret_cast<volatile int *>(&over_s)) break;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = (base + j * kRowsPerPass) * kSamplerClasses + cls;
                const float v = i < p.vocab ? t[(size_t)(base + j * kRowsPerPass) * t_stride + col] : -1.0f;
                if (v >= near_t) {
                    const float pr = __fdiv_rn(v, total);
                    if (pr >= floor_p) take(sample_key(pr, i));
                }
            }
        }
        sampler_cluster_sync();
        if (over_s) {
            listed = false;
            if (tid == 0) n_list = 0;  // a cluster barrier or more before the next entry is taken
        }
    }
    if (!listed) {  // the general way
        if (finer) {
            hist[tid] = 0;
            __syncthreads();
        }
        // ---- p_i, and a key prefix that enough entries reach ----
        for (int row = row0; row < rows; row += kRowsPerPass) {
            if (row * kSamplerClasses + cls >= p.vocab) break;
            const float pr = __fdiv_rn(t[(size_t)row * t_stride + col], total);
            t[(size_t)row * t_stride + col] = pr;
            atomicAdd(&hist[__float_as_uint(pr) >> 20], 1);  // p <= 1: the bin is at most 0x3f8
        }
        uint64_t floor_key = 0;  // prefix of the keys that are taken, at `shift`
        int shift = 52, need = p.want;
        for (;;) {
            sampler_cluster_sync();  // the histograms of all CTAs are complete
            count_down();
            if (inc >= need && inc - cnt < need) {
                bin_s = kSamplerBins - 1 - tid;
                above_s = inc - cnt;
                count_s = inc;
            }
            __syncthreads();
            floor_key += (uint64_t)bin_s;
            // entries above the bins of this level were counted out of `need` already: they are among the taken ones too
            if (p.want - need + count_s <= kSamplerCap || shift == 0) break;
            need -= above_s;
            const int bits = shift >= 10 ? 10 : shift;
            const int next = shift - bits;
            sampler_cluster_sync();  // every CTA has read the histograms
            hist[tid] = 0;
            __syncthreads();
            for (int row = row0; row < rows; row += kRowsPerPass) {
                const int i = row * kSamplerClasses + cls;
                if (i >= p.vocab) break;
                const uint64_t key = sample_key(t[(size_t)row * t_stride + col], i);
                if ((key >> shift) == floor_key) atomicAdd(&hist[(int)(key >> next) & ((1 << bits) - 1)], 1);
            }
            floor_key <<= bits;
            shift = next;
        }
        // ---- the entries that reach it go to CTA 0 ----
        for (int row = row0; row < rows; row += kRowsPerPass) {
            const int i = row * kSamplerClasses + cls;
            if (i >= p.vocab) break;
            const uint64_t key = sample_key(t[(size_t)row * t_stride + col], i);
            if ((key >> shift) >= floor_key) take(key);
        }
        sampler_cluster_sync();
    }
    if (cta != 0) return;

    // ---- descending order of the collected keys ----
    const int n = min(n_list, kSamplerCap);
    if (n <= kSamplerRankCap) {  // each key's rank by counting the greater ones, four threads per key: one barrier
        const int i = tid / kRankThreads, part = tid % kRankThreads;
        const uint64_t mine = i < n ? list[i] : 0;
        int rank = 0;
        for (int j = part; j < n; j += kRankThreads) rank += list[j] > mine ? 1 : 0;
#pragma unroll
        for (int m = 1; m < kRankThreads; m <<= 1) rank += __shfl_xor_sync(0xffffffffu, rank, m);
        __syncthreads();
        if (i < n && part == 0) list[rank] = mine;  // keys are unique: so are ranks
        __syncthreads();
    } else {
        int n2 = 512;  // bitonic; the padding sorts last
        while (n2 < n) n2 <<= 1;
        for (int i = n + tid; i < n2; i += kSamplerThreads) list[i] = 0;
        __syncthreads();
        for (int size = 2; size <= n2; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                if (tid < n2 / 2) {
                    const int a = 2 * tid - (tid & (stride - 1)), b = a + stride;
                    const uint64_t ka = list[a], kb = list[b];
                    if ((ka < kb) == ((a & size) == 0)) { list[a] = kb; list[b] = ka; }
                }
                __syncthreads();
            }
    }
    const int have = min(p.want, n);  // n >= want: the threshold bin was chosen so
    if (tid < have) sel_p[tid] = __uint_as_float((uint32_t)(list[tid] >> 32));
    __syncthreads();
    // ---- top_k_sampling: renormalise the first k entries (inference.cu:1088-1096) ----
    const int k = min(p.top_k, have);
    if (tid == 0) {
        float sum_k = 0.0f;
#pragma unroll 8
        for (int i = 0; i < k; ++i) sum_k += sel_p[i];
        sum_s = sum_k;
    }
    __syncthreads();
    if (tid < k) sel_p[tid] = __fdiv_rn(sel_p[tid], sum_s);
    __syncthreads();
    // ---- top_p_sampling: the prefix whose running sum reaches top_p (:1131-1136); entries beyond the first k keep
    // their own probability ----
    if (tid == 0) {
        float cumulative = 0.0f;
        int cutoff = first_reaching(sel_p, have, cumulative, [&](float run) { return run >= p.top_p; });
        if (cutoff < 0 && have == p.vocab) cutoff = p.vocab - 1;  // :1140-1143
        cutoff_s = cutoff;
        sum_s = cumulative;  // :1138
    }
    __syncthreads();
    const int cutoff = cutoff_s;
    if (cutoff < 0) {  // the prefix ran past what this kernel orders: let the host sampler take the step
        if (tid == 0) { p.token_out[0] = -1; p.result[0] = 2; }
        return;
    }
    if (tid <= cutoff) sel_p[tid] = __fdiv_rn(sel_p[tid], sum_s);  // :1146-1148
    __syncthreads();
    if (tid != 0) return;
    float run = 0.0f;  // :1154-1158
    const int drawn = first_reaching(sel_p, cutoff + 1, run, [&](float r) { return p.u < r; });
    const int at = drawn < 0 ? 0 : drawn;  // :1159-1160
    const int token = (int)(0xffffffffu - (uint32_t)list[at]);
    p.token_out[0] = token;
    p.result[0] = 0;
    p.result[1] = n;
    p.result[2] = listed ? 1 : 0;
    if (p.pos && p.history) {
        const int where = p.pos[0];
        if (where >= 0 && where < p.history_len) p.history[where] = token;
    }
}

// The classes' largest entries lead to the wanted ones only where these are fewer than the classes, and it pays where a class has many: us a
// draw at top_k 50 with the radix select / so 8.1 / 8.4 over 8193 entries, 8.5 / 8.7 over 16384, 9.1 / 9.0 over 20000, 9.3 / 8.6 over 32768.
static bool sample_by_class(int vocab, int want) { return want <= kSamplerClasses / 2 && vocab >= 32 * kSamplerClasses; }

}  // namespace llmb

extern "C" size_t llmb_sample_scratch_bytes(int vocab) { return vocab > 0 ? (size_t)vocab * sizeof(float) + 256 : 0; }

extern "C" int llmb_sample_logits(const uint16_t *d_logits, int vocab, float temperature, int top_k, float top_p, uint64_t seed,
                                  uint64_t draw, void *d_scratch, int32_t *d_token_out, int32_t *d_pos, int32_t *d_history,
                                  int history_len, int use_pdl, llmb_stream_t stream_) {
    using namespace llmb;
    if (!d_logits || !d_scratch || !d_token_out || vocab <= 0 || !(temperature > 0.0f) || top_k < 1 || !(top_p > 0.0f) ||
        ((uintptr_t)d_scratch & 255)) {
        set_last_error("llmb_sample_logits: need temperature > 0, top_k >= 1, 0 < top_p, a 256-byte aligned scratch");
        return LLMB_ERR_INVALID;
    }
    if (top_p > 1.0f) top_p = 1.0f;    // inference.cu:1124-1126
    if (top_k > vocab) top_k = vocab;  // :1083-1085
    if (top_k > kSamplerMaxSelect) {
        set_last_error("llmb_sample_logits: top_k above 1024 is not ordered on the device; use llmb_sample_logits_host");
        return LLMB_ERR_UNSUPPORTED;
    }
    SamplerParams p;
    p.logits = reinterpret_cast<const __half *>(d_logits);
    p.result = static_cast<int *>(d_scratch);
    p.probs = reinterpret_cast<float *>(static_cast<unsigned char *>(d_scratch) + 256);
    p.token_out = d_token_out;
    p.pos = d_pos;
    p.history = d_history;
    p.history_len = history_len;
    p.vocab = vocab;
    p.top_k = top_k;
    p.temperature = temperature;
    p.top_p = top_p;
    p.u = llmb_synth_uniform(llmb_stream_key(seed, LLMB_SID_SAMPLER), draw);
    p.want = want_entries(vocab, top_k, top_p);
    const int rows = (vocab + kSamplerClasses - 1) / kSamplerClasses;
    p.in_smem = rows <= kSamplerSmemRows ? 1 : 0;
    const size_t smem = p.in_smem ? (size_t)rows * kClassesPerCta * sizeof(float) : 0;
    static size_t attr_set[2][3][kMaxDevices] = {};  // per instantiation and device
    static const struct { void (*kernel)(const SamplerParams); int most_rows; } kernels[2][3] = {
        {{sample_kernel<false, 1>, kRowsPerPass}, {sample_kernel<false, 4>, 4 * kRowsPerPass}, {sample_kernel<false, 16>, INT_MAX}},
        {{nullptr, 0}, {sample_kernel<true, 4>, 4 * kRowsPerPass}, {sample_kernel<true, 16>, INT_MAX}}};
    const int by_class = sample_by_class(vocab, p.want) ? 1 : 0;
    int loads = 0;
    while (rows > kernels[by_class][loads].most_rows) ++loads;
    void (*kernel)(const SamplerParams) = kernels[by_class][loads].kernel;
    LLMB_CUDA_OK(ensure_dynamic_smem(kernel, attr_set[by_class][loads], smem));
    LLMB_CUDA_OK(launch_pdl_cluster(kernel, dim3(kSamplerCtas), dim3(kSamplerThreads), smem, static_cast<cudaStream_t>(stream_),
                                    use_pdl != 0, dim3(kSamplerCtas, 1, 1), p));
    return LLMB_OK;
}
