// Stable top-k selection and index-gathered sparse attention.
#include <mutex>
#include <thread>
#include <vector>
#include <cooperative_groups.h>
#include "runtime.cuh"
#include "tc_common.cuh"

namespace apus {

// ---- stable top-k --------------------------------------------------------------
//
// Reference c/attn.h:668-687: k passes of strict-greater argmax over unused
// entries, i.e. the k largest scores, equal scores ordered by ascending index,
// emitted in that order.  Restated as a selection on the composite key
// (score, -index): a radix select on the order-preserving integer image of the
// score finds the k-th largest score value, every score above it and the
// lowest-index scores equal to it are collected, and a bitonic sort of the k
// (key, index) pairs gives the output order.
//
// One CTA per row, or a cluster of eight for long rows: there every CTA
// histograms its slice, all of them add their histograms into rank 0's shared
// memory and derive the same digit from the sum, so no result has to be sent
// around; the chosen entries are stored into rank 0's shared memory, where rank 0
// sorts and writes them out.  Nobody touches another CTA's shared memory before a
// first cluster barrier (a CTA of the cluster may not have started yet), and
// nobody leaves before the last reader is done.
//
// The row crosses L2 once: a thread keeps its KPT keys in registers for every
// pass (KPT = 0: rows too long for that are read again by each pass).  Digits of
// 11, 11 and 10 bits; as soon as the bin that holds the k-th score is taken whole
// no further digit is needed, which ends most rows after the second, and only a
// tie at the boundary takes the index-ordered sweep.  The sort exchanges through
// shuffles below a stride of 32.  Bound by the latency of these short phases.
// B200: 262,144 scores, k = 512 83.6 -> 26.6 us; 32 rows of 2,048 14.7 -> 9.1 us.
__device__ __forceinline__ uint32_t order_key(float f) {
    uint32_t u = __float_as_uint(f);
    if ((u << 1) == 0) u = 0;                 // -0.0 and +0.0 compare equal
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

#define TOPK_THREADS 1024
#define TOPK_MAX_K 2048

#define TOPK_CL 8
#define TOPK_BINS 2048
template <int CL, int KPT>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(TOPK_THREADS)
topk_stable_kernel(const float *__restrict__ scores, int n, int k, int32_t *__restrict__ idx_out,
                   const long long *__restrict__ dyn_pos, int ratio, long long chunk_pos0, int rows_per_pos) {
    APUS_PDL_WAIT();
    APUS_PDL_GO();
    namespace cg = cooperative_groups;
    __shared__ unsigned hist[TOPK_BINS];
    __shared__ unsigned ghist[CL > 1 ? 2 : 1][CL > 1 ? TOPK_BINS : 1];   // rank 0's copies: the slices' histograms added up
    __shared__ unsigned s_w[32], s_digit[3];
    __shared__ unsigned s_eq;                           // this slice's keys equal to the boundary
    __shared__ unsigned s_taken;                        // rank 0's copy counts the chosen entries
    __shared__ unsigned long long sel[TOPK_MAX_K];      // rank 0's copy collects the choice
    const int rowi = blockIdx.x / CL, rank = CL > 1 ? (int)(blockIdx.x % CL) : 0;
    const float *row = scores + (size_t)rowi * n;       // n, k as given are the row strides
    int32_t *out = idx_out + (size_t)rowi * k;
    if (dyn_pos || rows_per_pos > 0) {                  // live sizes from the position (of the row, in a chunk)
        const long long nbs = ((dyn_pos ? *dyn_pos : chunk_pos0 + rowi / rows_per_pos) + 1) / ratio;
        n = (int)(nbs < n ? nbs : n);
        k = k < n ? k : n;
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto sync_all = [&]() { if constexpr (CL > 1) cg::this_cluster().sync(); else __syncthreads(); };
    auto at_rank = [&](unsigned *p, int r) -> unsigned * {
        if constexpr (CL > 1) return cg::this_cluster().map_shared_rank(p, r);
        else return p;
    };
    if (tid == 0) { s_taken = 0; s_eq = 0; }
    sync_all();                                         // every CTA of the cluster runs from here on
    if (k <= 0) return;                                 // the same decision in all of them
    const int per = (n + CL - 1) / CL, i0 = min(n, rank * per), i1 = min(n, i0 + per);
    const int steps = (per + TOPK_THREADS - 1) / TOPK_THREADS;       // the same in every CTA
    uint32_t keys[KPT ? KPT : 1];
    if (KPT) {
#pragma unroll
        for (int r = 0; r < KPT; r++) {
            const int i = i0 + r * TOPK_THREADS + tid;
            keys[r] = i < i1 ? order_key(row[i]) : 0u;
        }
    }
    // calls f(i, key) for this thread's scores in ascending order; whole warps stay together (in = a real score)
    auto each = [&](auto &&f) {
        if constexpr (KPT > 0) {
#pragma unroll
            for (int r = 0; r < KPT; r++) {
                if (r >= steps) break;
                const int i = i0 + r * TOPK_THREADS + tid;
                f(i, keys[r], i < i1);
            }
        } else {
            for (int r = 0; r < steps; r++) {
                const int i = i0 + r * TOPK_THREADS + tid;
                f(i, i < i1 ? order_key(row[i]) : 0u, i < i1);
            }
        }
    };
    uint32_t T = 0;                                     // boundary so far: the digits of the k-th key, zeros below
    unsigned need = (unsigned)k, n_greater = 0;         // of the keys that share its digits; keys above them
    bool whole = k >= n;                                // every key >= T is chosen
    if (k > n) k = n;
    for (int pass = 0; pass < 3 && !whole; pass++) {
        const int shift = pass == 0 ? 21 : pass == 1 ? 10 : 0;
        const uint32_t himask = pass == 0 ? 0u : pass == 1 ? 0xffe00000u : 0xfffffc00u, dmask = pass == 2 ? 1023u : 2047u;
        for (int i = tid; i < TOPK_BINS; i += TOPK_THREADS) {
            hist[i] = 0;
            if (CL > 1 && rank == 0) ghist[pass & 1][i] = 0;         // last read two barriers ago
        }
        sync_all();
        each([&](int, uint32_t key, bool in) {
            if (in && (key & himask) == T) atomicAdd(&hist[(key >> shift) & dmask], 1u);
        });
        __syncthreads();
        const unsigned *h = hist;
        if (CL > 1) {
            unsigned *g = at_rank(&ghist[pass & 1][0], 0);
            for (int i = tid; i < TOPK_BINS; i += TOPK_THREADS)
                if (hist[i]) atomicAdd(g + i, hist[i]);
            sync_all();                                 // the sum is complete
            h = g;
        }
        // the bin where the count from the top reaches `need`: thread t holds bins 2047 - 2t and 2046 - 2t
        const unsigned c0 = h[TOPK_BINS - 1 - 2 * tid], c1 = h[TOPK_BINS - 2 - 2 * tid], tot = c0 + c1;
        unsigned inc = tot;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned v = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += v;
        }
        if (lane == 31) s_w[warp] = inc;
        __syncthreads();
        unsigned wv = s_w[lane];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const unsigned v = __shfl_up_sync(0xffffffffu, wv, off);
            if (lane >= off) wv += v;
        }
        const unsigned before = warp ? __shfl_sync(0xffffffffu, wv, (warp + 31) & 31) : 0u;
        const unsigned exc = before + inc - tot;
        if (exc < need && exc + tot >= need) {          // one thread: the counts add up to at least `need`
            const bool first = exc + c0 >= need;
            s_digit[0] = first ? exc : exc + c0;
            s_digit[1] = (unsigned)(first ? TOPK_BINS - 1 - 2 * tid : TOPK_BINS - 2 - 2 * tid);
            s_digit[2] = first ? c0 : c1;
        }
        __syncthreads();
        n_greater += s_digit[0];
        need -= s_digit[0];
        T |= s_digit[1] << shift;
        whole = s_digit[2] == need;
    }
    // keys above the boundary (all those at it too, when they are all chosen) in any order
    unsigned *cnt0 = at_rank(&s_taken, 0);
    unsigned long long *sel0 = sel;
    if constexpr (CL > 1) sel0 = cg::this_cluster().map_shared_rank(sel, 0);
    unsigned eq = 0;
    each([&](int i, uint32_t key, bool in) {
        const bool take = in && (whole ? key >= T : key > T);
        eq += !whole && in && key == T;
        const unsigned m = __ballot_sync(0xffffffffu, take);
        if (!m) return;
        unsigned slot = 0;
        if (lane == 0) slot = atomicAdd(cnt0, (unsigned)__popc(m));
        slot = __shfl_sync(0xffffffffu, slot, 0) + __popc(m & ((1u << lane) - 1u));
        if (take) sel0[slot] = ((unsigned long long)key << 32) | (0xffffffffu - (unsigned)i);
    });
    if (!whole) {
        // more keys at the boundary than places: the lowest indices, counted over the slices before this one
        // and, inside the slice, step by step
        eq = __reduce_add_sync(0xffffffffu, eq);
        if (lane == 0 && eq) atomicAdd(&s_eq, eq);
        sync_all();
        unsigned base = 0;
        for (int q = 0; q < rank; q++) base += *at_rank(&s_eq, q);
        each([&](int i, uint32_t key, bool in) {
            const bool e = in && key == T;
            const unsigned m = __ballot_sync(0xffffffffu, e);
            if (lane == 0) s_w[warp] = __popc(m);
            __syncthreads();
            unsigned wv = s_w[lane], tot = __reduce_add_sync(0xffffffffu, wv);
            const unsigned bef = __reduce_add_sync(0xffffffffu, lane < warp ? wv : 0u);
            const unsigned place = base + bef + __popc(m & ((1u << lane) - 1u));
            if (e && place < need) sel0[n_greater + place] = ((unsigned long long)key << 32) | (0xffffffffu - (unsigned)i);
            base += tot;
            __syncthreads();
        });
    }
    sync_all();                                         // the whole choice sits in rank 0
    if (rank != 0) return;
    // bitonic sort, descending, on the composite (key, -index)
    int kp = 32;
    while (kp < k) kp <<= 1;
    if (kp <= TOPK_THREADS) {
        unsigned long long v = tid < k ? sel[tid] : 0ull;
        int buf = 0;
        __syncthreads();
        for (int size = 2; size <= kp; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                unsigned long long w;
                if (stride >= 32) {                     // the two halves of `sel` in turn: one barrier per exchange
                    if (tid < kp) sel[buf * TOPK_THREADS + tid] = v;
                    __syncthreads();
                    w = tid < kp ? sel[buf * TOPK_THREADS + (tid ^ stride)] : 0ull;
                    buf ^= 1;
                } else {
                    w = __shfl_xor_sync(0xffffffffu, v, stride);
                }
                const bool want_max = ((tid & size) == 0) == ((tid & stride) == 0);
                v = want_max == (v > w) ? v : w;
            }
        if (tid < k) out[tid] = (int32_t)(0xffffffffu - (unsigned)(v & 0xffffffffu));
        return;
    }
    for (int i = k + tid; i < kp; i += TOPK_THREADS) sel[i] = 0ull;
    __syncthreads();
    for (int size = 2; size <= kp; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = tid; i < kp; i += TOPK_THREADS) {
                const int j = i ^ stride;
                if (j > i) {
                    const unsigned long long a = sel[i], b = sel[j];
                    const bool desc = ((i & size) == 0);
                    if (desc ? (a < b) : (a > b)) { sel[i] = b; sel[j] = a; }
                }
            }
            __syncthreads();
        }
    for (int i = tid; i < k; i += TOPK_THREADS)
        out[i] = (int32_t)(0xffffffffu - (unsigned)(sel[i] & 0xffffffffu));
}

int topk_stable(const float *scores, int n, int k, int32_t *idx, int rows,
                cudaStream_t st, const long long *dyn_pos, int ratio, long long chunk_pos0, int rows_per_pos) {
    APUS_REQUIRE(k >= 1 && (k <= n || dyn_pos || rows_per_pos > 0) && k <= TOPK_MAX_K, "topk: n=%d k=%d unsupported", n, k);
    if (rows <= 0) return 0;
    static const int cl_min = [] { const char *e = getenv("APUS_TOPK_CLUSTER_MIN"); return e && e[0] ? atoi(e) : 16384; }();
#define TOPK_LAUNCH(CL, KPT)                                                                                              \
    launch_k(topk_stable_kernel<CL, KPT>, (unsigned)rows * CL, TOPK_THREADS, 0, st, scores, n, k, idx, dyn_pos, ratio,    \
             chunk_pos0, rows_per_pos)
    if (n >= cl_min) {                                  // long rows: a cluster of CTAs per row
        if (n <= TOPK_CL * TOPK_THREADS * 8) TOPK_LAUNCH(TOPK_CL, 8);
        else if (n <= TOPK_CL * TOPK_THREADS * 32) TOPK_LAUNCH(TOPK_CL, 32);
        else TOPK_LAUNCH(TOPK_CL, 0);
    } else {
        if (n <= TOPK_THREADS * 4) TOPK_LAUNCH(1, 4);
        else if (n <= TOPK_THREADS * 16) TOPK_LAUNCH(1, 16);
        else TOPK_LAUNCH(1, 0);
    }
#undef TOPK_LAUNCH
    APUS_LAUNCHED();
    return 0;
}

// ---- sparse attention --------------------------------------------------------------
//
// Reference c/attn.h:1193-1326.  Per (token t, head h): ids < 0 are dropped
// (order kept); s_j = (q . kv_j) * scale; p_j = bf16(exp(s_j - max_j s));
// o = sum_j p_j * kv_j accumulated in j order; o = bf16(o / (sum_j p_j +
// exp(sink_h - max))); no ids -> zeros.  K and V are the same vector; ids
// below `na` index kv_a, the rest kv_b (offset by na).
//
// Kernel 1 (scores): one thread per (head, id) computes the full d-long dot in
// the reference's k order with separate rounded multiply and add, from a
// shared-memory tile of 32 gathered KV rows shared by 16 heads.
// Kernel 2 (softmax + PV): one CTA per (token, head); p_j in shared memory,
// each thread owns two adjacent output channels and walks j in order.
template <bool BF16>
__device__ __forceinline__ float2 kv_pair(const void *base, size_t row, int d, int k2) {
    if (BF16) {
        uint32_t w = __ldg(reinterpret_cast<const uint32_t *>(
            reinterpret_cast<const uint16_t *>(base) + row * d) + k2);
        return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    }
    return __ldg(reinterpret_cast<const float2 *>(reinterpret_cast<const float *>(base) + row * d) + k2);
}

#define SA_IDS 32
#define SA_HEADS 16

template <bool BF16>
__global__ void __launch_bounds__(SA_IDS * SA_HEADS)
sparse_scores_kernel(const float *__restrict__ q, int h, int d, const int32_t *__restrict__ ids,
                     const int *__restrict__ ns, int idxw, float scale, const void *kv_a,
                     int64_t na, const void *kv_b, float *__restrict__ sc, size_t a_stride,
                     size_t b_stride, int seq_mod) {
    APUS_PDL_WAIT();
    APUS_PDL_GO();
    extern __shared__ float sm[];
    const int t = blockIdx.z, hb = blockIdx.y, tile = blockIdx.x;
    const int own = seq_mod > 0 ? t % seq_mod : t;         // whose caches: rows of a chunk are time-major
    kv_a = reinterpret_cast<const char *>(kv_a) + (size_t)own * a_stride;
    kv_b = reinterpret_cast<const char *>(kv_b) + (size_t)own * b_stride;
    const int n = ns[t];
    if (tile * SA_IDS >= n) return;
    const int pitch = d + 1;
    float *s_kv = sm;                          // [SA_IDS][d+1]
    float *s_q = sm + SA_IDS * pitch;          // [SA_HEADS][d]
    const int tid = threadIdx.x;
    const int32_t *idr = ids + (size_t)t * idxw + tile * SA_IDS;
    const int cnt = min(SA_IDS, n - tile * SA_IDS);
    for (int i = tid; i < SA_IDS * (d / 2); i += blockDim.x) {
        int r = i / (d / 2), k2 = i - r * (d / 2);
        float2 v = make_float2(0.f, 0.f);
        if (r < cnt) {
            int32_t id = idr[r];
            v = id < na ? kv_pair<BF16>(kv_a, (size_t)id, d, k2)
                        : kv_pair<BF16>(kv_b, (size_t)(id - na), d, k2);
        }
        s_kv[r * pitch + 2 * k2] = v.x;
        s_kv[r * pitch + 2 * k2 + 1] = v.y;
    }
    for (int i = tid; i < SA_HEADS * d; i += blockDim.x) {
        int hh = i / d, k = i - hh * d;
        int head = hb * SA_HEADS + hh;
        s_q[i] = head < h ? q[((size_t)t * h + head) * d + k] : 0.f;
    }
    __syncthreads();
    const int j = tid & 31, hh = tid >> 5;
    const int head = hb * SA_HEADS + hh;
    if (j >= cnt || head >= h) return;
    const float *kvr = s_kv + j * pitch, *qr = s_q + hh * d;
    float dot = 0.f;
#pragma unroll 8
    for (int k = 0; k < d; k++) dot = __fadd_rn(dot, __fmul_rn(qr[k], kvr[k]));
    sc[((size_t)t * h + head) * idxw + tile * SA_IDS + j] = __fmul_rn(dot, scale);
}

template <bool BF16>
__global__ void __launch_bounds__(256)
sparse_pv_kernel(const float *__restrict__ sc, const float *__restrict__ sink, int h, int d,
                 const int32_t *__restrict__ ids, const int *__restrict__ ns, int idxw,
                 const void *kv_a, int64_t na, const void *kv_b, float *__restrict__ o, size_t a_stride,
                 size_t b_stride, int seq_mod) {
    APUS_PDL_WAIT();
    APUS_PDL_GO();
    extern __shared__ float s_p[];             // [idxw]
    __shared__ float red[32];
    __shared__ float s_mx, s_sum;
    const int t = blockIdx.y, head = blockIdx.x, tid = threadIdx.x;
    const int own = seq_mod > 0 ? t % seq_mod : t;
    kv_a = reinterpret_cast<const char *>(kv_a) + (size_t)own * a_stride;
    kv_b = reinterpret_cast<const char *>(kv_b) + (size_t)own * b_stride;
    const int n = ns[t];
    float *ov = o + ((size_t)t * h + head) * d;
    if (n == 0) {
        for (int k = tid; k < d; k += blockDim.x) ov[k] = 0.f;
        return;
    }
    const float *sr = sc + ((size_t)t * h + head) * idxw;
    float mx = -INFINITY;
    for (int j = tid; j < n; j += blockDim.x) mx = fmaxf(mx, sr[j]);
    mx = warp_max(mx);
    if ((tid & 31) == 0) red[tid >> 5] = mx;
    __syncthreads();
    if (tid < 32) {
        float v = tid < (blockDim.x >> 5) ? red[tid] : -INFINITY;
        v = warp_max(v);
        if (tid == 0) s_mx = v;
    }
    __syncthreads();
    mx = s_mx;
    for (int j = tid; j < n; j += blockDim.x) s_p[j] = bf16_round(exp_rn(__fsub_rn(sr[j], mx)));
    __syncthreads();
    if (tid == 0) {
        float sum = 0.f;
        if (n <= 1024) { for (int j = 0; j < n; j++) sum = __fadd_rn(sum, s_p[j]); s_sum = sum; }
    }
    if (n > 1024) {                            // long HCA rows: tree sum
        float part = 0.f;
        for (int j = tid; j < n; j += blockDim.x) part += s_p[j];
        part = warp_sum(part);
        __syncthreads();
        if ((tid & 31) == 0) red[tid >> 5] = part;
        __syncthreads();
        if (tid == 0) {
            float sum = 0.f;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) sum += red[w];
            s_sum = sum;
        }
    }
    __syncthreads();
    const float den = __fadd_rn(s_sum, exp_rn(__fsub_rn(sink[head], mx)));
    const int32_t *idr = ids + (size_t)t * idxw;
    for (int k2 = tid; k2 < d / 2; k2 += blockDim.x) {
        float a0 = 0.f, a1 = 0.f;
        for (int j = 0; j < n; j++) {
            int32_t id = idr[j];
            float2 v = id < na ? kv_pair<BF16>(kv_a, (size_t)id, d, k2)
                               : kv_pair<BF16>(kv_b, (size_t)(id - na), d, k2);
            float p = s_p[j];
            a0 = __fadd_rn(a0, __fmul_rn(p, v.x));
            a1 = __fadd_rn(a1, __fmul_rn(p, v.y));
        }
        ov[2 * k2] = bf16_round(__fdiv_rn(a0, den));
        ov[2 * k2 + 1] = bf16_round(__fdiv_rn(a1, den));
    }
}

// ---- the same two steps, register-tiled ---------------------------------------------------------
// Same arithmetic, same order, same bits as the two kernels above; what changes is how often a number is
// fetched per flop and how many instructions a flop takes.
//
// Both contractions are chains of (multiply, add) per (head, candidate) or (head, channel), bound by the
// FP32 pipes.  Two things shorten them without touching a bit:
//   - q, the KV rows and the probabilities are BF16 values, so a product is exact and one fused
//     multiply-add returns what the multiply and the add return.  That holds inside an exponent window
//     (fma_ok_f32); every operand is examined, and where one lies outside (or is a true f32 value) the
//     two-instruction walk runs instead.  What the scores kernel and the softmax find about the rows and the
//     probabilities of a token is left in bad[t] for P.V.
//   - two accumulators per instruction (f32x2): two heads in the scores, two channels in P.V.
// One packed instruction does two multiply-adds at the rate of two scalar ones, in half the issue slots; the kernels
// still spend as many on operand moves, and the FP32 pipes are 30-45 % busy.  Times beside the launches below.
//
// Scores: a lane owns HL heads x CL candidates, a warp 4 HL heads x 8 CL candidates, a CTA WH x WC warps.
// The CTA's gathered rows travel 128 bytes of k at a time, three chunks deep, in their natural layout by
// 16-byte cp.async (row pitch 36 words: the eight rows the lanes of a load touch fall into different banks);
// the q chunk sits transposed ([k][head], a 16-byte load gives a lane two head pairs), its 4-head groups
// permuted by k so that the transposing stores do not collide, and passes through registers: loaded before
// the arithmetic of a chunk, stored after it.
// softmax: max, p_j = bf16(exp(s_j - max)) written over the scores, denominator per (row, head).
#define SS_ROWB 128                       // bytes of a KV row staged per chunk: 64 BF16 or 32 f32 values of k
#define SS_PITCHW 36                      // row pitch of the staged tile in 32-bit words (128 B + 16 B pad)
#define SS_NS 3

template <bool BF16, int HL, int CL, int WH, int WC>
struct ScoreCfg {
    static constexpr int THREADS = 32 * WH * WC, HEADS = 4 * HL * WH, CANDS = 8 * CL * WC, KC = BF16 ? 64 : 32;
    static constexpr int Q_WORDS = KC * HEADS, STAGE = (Q_WORDS + CANDS * SS_PITCHW) * 4, SMEM = SS_NS * STAGE;
};

// The operands of four k for a lane: its head pairs and its candidates' words
template <bool BF16, int HL, int CL, int HEADS>
struct ScoreOps {
    ulonglong2 q[4][HL / 4];
    uint32_t kv[CL][BF16 ? 2 : 4];
    __device__ __forceinline__ void load(const float *sq, const uint32_t *skv, int g0, int g) {
        constexpr int SWZ = (HEADS / 4 < 8 ? HEADS / 4 : 8) - 1;
#pragma unroll
        for (int e = 0; e < 4; e++)
#pragma unroll
            for (int i = 0; i < HL / 4; i++)
                q[e][i] = *reinterpret_cast<const ulonglong2 *>(sq + (size_t)(4 * g + e) * HEADS + 4 * ((g0 + i) ^ (g & SWZ)));
#pragma unroll
        for (int b = 0; b < CL; b++) {
            if constexpr (BF16) {
                const uint2 r = *reinterpret_cast<const uint2 *>(skv + (size_t)8 * b * SS_PITCHW + 2 * g);
                kv[b][0] = r.x; kv[b][1] = r.y;
            } else {
                const uint4 r = *reinterpret_cast<const uint4 *>(skv + (size_t)8 * b * SS_PITCHW + 4 * g);
                kv[b][0] = r.x; kv[b][1] = r.y; kv[b][2] = r.z; kv[b][3] = r.w;
            }
        }
    }
    template <bool FUSED>
    __device__ __forceinline__ void walk(f32x2 (&acc)[HL / 2][CL]) const {
#pragma unroll
        for (int e = 0; e < 4; e++)
#pragma unroll
            for (int b = 0; b < CL; b++) {
                const uint32_t u = BF16 ? (e & 1 ? kv[b][e >> 1] & 0xffff0000u : kv[b][e >> 1] << 16) : kv[b][BF16 ? 0 : e];
                const f32x2 y = pack2(__uint_as_float(u), __uint_as_float(u));
#pragma unroll
                for (int a = 0; a < HL / 2; a++) acc[a][b] = mac2<FUSED>(acc[a][b], a & 1 ? q[e][a >> 1].y : q[e][a >> 1].x, y);
            }
    }
};
// One chunk of k for a lane, acc[pair of heads][candidate]; operands are read four k ahead of their use
template <bool BF16, bool FUSED, int HL, int CL, int HEADS>
__device__ __forceinline__ void score_chunk(f32x2 (&acc)[HL / 2][CL], const float *sq, const uint32_t *skv, int g0) {
    constexpr int NG = (BF16 ? 64 : 32) / 4;
    ScoreOps<BF16, HL, CL, HEADS> A, B;
    A.load(sq, skv, g0, 0);
#pragma unroll
    for (int g = 0; g < NG; g += 2) {
        B.load(sq, skv, g0, g + 1);
        A.template walk<FUSED>(acc);
        if (g + 2 < NG) A.load(sq, skv, g0, g + 2);
        B.template walk<FUSED>(acc);
    }
}

template <bool BF16, int HL, int CL, int WH, int WC>
__global__ void __launch_bounds__(32 * WH * WC)
sparse_scores_tile_kernel(const float *__restrict__ q, int h, int d, const int32_t *__restrict__ ids,
                          const int *__restrict__ ns, int idxw, float scale, const void *kv_a, int64_t na,
                          const void *kv_b, float *__restrict__ sc, size_t a_stride, size_t b_stride, int seq_mod,
                          int *__restrict__ bad) {
    APUS_PDL_WAIT();
    APUS_PDL_GO();
    using Cf = ScoreCfg<BF16, HL, CL, WH, WC>;
    constexpr int NT = Cf::THREADS, KC = Cf::KC, HEADS = Cf::HEADS, CANDS = Cf::CANDS;
    constexpr int SWZ = (HEADS / 4 < 8 ? HEADS / 4 : 8) - 1;
    extern __shared__ __align__(16) unsigned char ss_raw[];
    __shared__ int s_bad[SS_NS];                                // chunk in this stage: an operand outside the window
    const int t = blockIdx.z, h0 = (int)blockIdx.y * HEADS, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n = ns[t], j0 = (int)blockIdx.x * CANDS;
    if (j0 >= n) return;                                        // whole CTA past the row
    const int own = seq_mod > 0 ? t % seq_mod : t;
    const size_t esz = BF16 ? 2 : 4;
    const int nchunk = d / KC;
    // copy u of this thread: row (tid + NT u) / 8, 16-byte segment tid % 8; its rows are the same in every chunk
    constexpr int NKV = CANDS * 8 / NT;
    static_assert(CANDS * 8 % NT == 0 && NT % 8 == 0, "row copies must divide among the threads");
    const char *rowp[NKV];
    const char *dummy = reinterpret_cast<const char *>(kv_a ? kv_a : kv_b);
#pragma unroll
    for (int u = 0; u < NKV; u++) {
        const int j = j0 + ((tid + NT * u) >> 3);
        const char *ptr = nullptr;
        if (j < n) {
            const int32_t id = ids[(size_t)t * idxw + j];
            ptr = id < na ? reinterpret_cast<const char *>(kv_a) + (size_t)own * a_stride + (size_t)id * d * esz
                          : reinterpret_cast<const char *>(kv_b) + (size_t)own * b_stride + (size_t)(id - na) * d * esz;
            ptr += (tid & 7) * 16;
        }
        rowp[u] = ptr;
    }
    auto q_of = [&](int st) { return reinterpret_cast<float *>(ss_raw + (size_t)st * Cf::STAGE); };
    auto kv_of = [&](int st) { return reinterpret_cast<uint32_t *>(ss_raw + (size_t)st * Cf::STAGE) + Cf::Q_WORDS; };
    auto kv_stage = [&](int c) {
        if (c < nchunk) {
            uint32_t *dst = kv_of(c % SS_NS);
#pragma unroll
            for (int u = 0; u < NKV; u++)
                cp_async16(dst + (size_t)((tid + NT * u) >> 3) * SS_PITCHW + (tid & 7) * 4,
                           rowp[u] ? rowp[u] + (size_t)c * SS_ROWB : dummy, rowp[u] != nullptr);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    constexpr int QN = HEADS * KC / 4 / NT;
    static_assert(HEADS * (KC / 4) % NT == 0, "the q chunk must divide among the threads");
    const bool q_vec = ((uintptr_t)q & 15) == 0;                // the caller's pointer may have any alignment
    float4 qreg[QN];
    auto q_load = [&](int c) {
#pragma unroll
        for (int u = 0; u < QN; u++) {
            const int i = tid + NT * u, hh = i / (KC / 4), seg = i % (KC / 4);
            const float *src = q + ((size_t)t * h + h0 + hh) * d + c * KC + 4 * seg;
            if (h0 + hh >= h) qreg[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            else if (q_vec) qreg[u] = *reinterpret_cast<const float4 *>(src);
            else qreg[u] = make_float4(src[0], src[1], src[2], src[3]);
        }
    };
    // stores chunk c's q and notes whether one of its values is outside the window
    auto q_store = [&](int c) {
        float *dst = q_of(c % SS_NS);
        bool ok = true;
#pragma unroll
        for (int u = 0; u < QN; u++) {
            const int i = tid + NT * u, hh = i / (KC / 4), seg = i % (KC / 4);
            float *p = dst + (size_t)4 * seg * HEADS + 4 * ((hh >> 2) ^ (seg & SWZ)) + (hh & 3);
            p[0] = qreg[u].x; p[HEADS] = qreg[u].y; p[2 * HEADS] = qreg[u].z; p[3 * HEADS] = qreg[u].w;
            ok = ok && fma_ok_f32(qreg[u].x) && fma_ok_f32(qreg[u].y) && fma_ok_f32(qreg[u].z) && fma_ok_f32(qreg[u].w);
        }
        if (!ok) s_bad[c % SS_NS] = 1;                          // every writer stores the same value
    };
    bool kv_bad = false;
    // this thread's own copies of chunk c have landed: are they all in the window?
    auto kv_check = [&](int c) {
        const uint32_t *src = kv_of(c % SS_NS);
        uint32_t low = 0, mx = 0, mn = 0xffffffffu;             // f32 rows: low halves, largest and smallest non-zero |v|
#pragma unroll
        for (int u = 0; u < NKV; u++) {
            const uint4 v = *reinterpret_cast<const uint4 *>(src + (size_t)((tid + NT * u) >> 3) * SS_PITCHW + (tid & 7) * 4);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                if (BF16) low |= fma_bad_bf16x2(w[e]);
                else { low |= w[e]; mx = max(mx, w[e] << 1); mn = min(mn, (w[e] << 1) - 1u); }
            }
        }
        const bool ok = BF16 ? (low & 0x80008000u) == 0u : (low & 0xffffu) == 0u && mx < (187u << 24) && mn >= (67u << 24) - 1u;
        if (!ok) { s_bad[c % SS_NS] = 1; kv_bad = true; }
    };
    const int wh = warp % WH, wc = warp / WH, hg = lane & 3, jg = lane >> 2;
    const bool live = j0 + wc * 8 * CL < n && h0 + wh * 4 * HL < h;     // other warps only help with the staging
    f32x2 acc[HL / 2][CL];
#pragma unroll
    for (int a = 0; a < HL / 2; a++)
#pragma unroll
        for (int b = 0; b < CL; b++) acc[a][b] = 0ull;
    if (tid < SS_NS) s_bad[tid] = 0;
    kv_stage(0);
    kv_stage(1);
    q_load(0);
    __syncthreads();                                            // the flags are clear
    q_store(0);
    for (int c = 0; c < nchunk; c++) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");    // the newest group is chunk c + 1
        kv_check(c);
        __syncthreads();                                        // chunk c is visible; chunk c - 1 has been consumed
        kv_stage(c + 2);
        if (c + 1 < nchunk) q_load(c + 1);
        const bool fused = s_bad[c % SS_NS] == 0;
        if (tid == 0) s_bad[(c + 2) % SS_NS] = 0;               // read last at chunk c - 1, written next for chunk c + 2
        if (live) {
            const float *sq = q_of(c % SS_NS);
            const uint32_t *skv = kv_of(c % SS_NS) + (size_t)(wc * 8 * CL + jg) * SS_PITCHW;
            const int g0 = (wh * 4 + hg) * (HL / 4);
            if (fused) score_chunk<BF16, true, HL, CL, HEADS>(acc, sq, skv, g0);
            else score_chunk<BF16, false, HL, CL, HEADS>(acc, sq, skv, g0);
        }
        if (c + 1 < nchunk) q_store(c + 1);                     // this stage was consumed at chunk c - 2
    }
    if (kv_bad) bad[t] = 1;
    if (!live) return;
#pragma unroll
    for (int a = 0; a < HL / 2; a++) {
        const int head = h0 + (wh * 4 + hg) * HL + 2 * a;
#pragma unroll
        for (int b = 0; b < CL; b++) {
            const int j = j0 + wc * 8 * CL + jg + 8 * b;
            const float2 v = unpack2(acc[a][b]);
            if (j < n && head < h) sc[((size_t)t * h + head) * idxw + j] = __fmul_rn(v.x, scale);
            if (j < n && head + 1 < h) sc[((size_t)t * h + head + 1) * idxw + j] = __fmul_rn(v.y, scale);
        }
    }
}

// The same for rows of at most 1024 candidates, a warp per (row, head): the denominator is one lane's chain of n adds,
// and eight of them run side by side in a CTA instead of one with seven idle warps beside it.
// B200: 2,048 rows x 64 heads, up to 256 candidates 344 -> 134 us.
__global__ void __launch_bounds__(256)
sparse_softmax_rows_kernel(float *__restrict__ sc, const float *__restrict__ sink, int h, const int *__restrict__ ns, int idxw,
                           float *__restrict__ den, int *__restrict__ bad) {
    APUS_PDL_WAIT();
    APUS_PDL_GO();
    extern __shared__ __align__(16) float s_all[];           // [8][pitch]
    const int t = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, head = (int)blockIdx.x * 8 + warp;
    const int n = ns[t];
    if (n == 0 || head >= h) return;
    float *s_p = s_all + (size_t)warp * ((idxw + 3) & ~3);
    float *sr = sc + ((size_t)t * h + head) * idxw;
    float mx = -INFINITY;
    for (int j = lane; j < n; j += 32) {
        const float v = sr[j];
        s_p[j] = v;
        mx = fmaxf(mx, v);
    }
    mx = warp_max(mx);
    bool ok = true;
    for (int j = lane; j < n; j += 32) {
        const float p = bf16_round(exp_rn(__fsub_rn(s_p[j], mx)));
        s_p[j] = p;
        sr[j] = p;
        ok = ok && fma_ok_f32(p);
    }
    if (!ok) bad[t] = 1;                       // P.V takes the two-instruction walk
    __syncwarp();
    if (lane == 0) den[(size_t)t * h + head] = __fadd_rn(seq_sum_smem(s_p, n, 0.f), exp_rn(__fsub_rn(sink[head], mx)));
}

// max, p over the scores, the denominator sum_j p_j + exp(sink - max): the sums in the order of
// sparse_pv_kernel (one accumulator for n <= 1024, the strided tree above it)
__global__ void __launch_bounds__(256)
sparse_softmax_kernel(float *__restrict__ sc, const float *__restrict__ sink, int h, const int *__restrict__ ns, int idxw,
                      float *__restrict__ den, int *__restrict__ bad) {
    APUS_PDL_WAIT();
    APUS_PDL_GO();
    extern __shared__ __align__(16) float s_p[];             // [idxw]
    __shared__ float red[32];
    __shared__ float s_mx, s_sum;
    const int t = blockIdx.y, head = blockIdx.x, tid = threadIdx.x;
    const int n = ns[t];
    if (n == 0) return;
    float *sr = sc + ((size_t)t * h + head) * idxw;
    float mx = -INFINITY;
    for (int j = tid; j < n; j += blockDim.x) mx = fmaxf(mx, sr[j]);
    mx = warp_max(mx);
    if ((tid & 31) == 0) red[tid >> 5] = mx;
    __syncthreads();
    if (tid < 32) {
        float v = tid < (blockDim.x >> 5) ? red[tid] : -INFINITY;
        v = warp_max(v);
        if (tid == 0) s_mx = v;
    }
    __syncthreads();
    mx = s_mx;
    for (int j = tid; j < n; j += blockDim.x) {
        const float p = bf16_round(exp_rn(__fsub_rn(sr[j], mx)));
        s_p[j] = p;
        sr[j] = p;
        if (!fma_ok_f32(p)) bad[t] = 1;        // P.V takes the two-instruction walk
    }
    __syncthreads();
    if (tid == 0 && n <= 1024) s_sum = seq_sum_smem(s_p, n, 0.f);
    if (n > 1024) {                            // long rows: tree sum
        float part = 0.f;
        for (int j = tid; j < n; j += blockDim.x) part += s_p[j];
        part = warp_sum(part);
        __syncthreads();
        if ((tid & 31) == 0) red[tid >> 5] = part;
        __syncthreads();
        if (tid == 0) {
            float sum = 0.f;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++) sum += red[w];
            s_sum = sum;
        }
    }
    __syncthreads();
    if (tid == 0) den[(size_t)t * h + head] = __fadd_rn(s_sum, exp_rn(__fsub_rn(sink[head], mx)));
}

#define PV_JC 128
template <bool BF16, int HG>
__global__ void __launch_bounds__(256)
sparse_pv_tile_kernel(const float *__restrict__ p, const float *__restrict__ den, int h, int d,
                      const int32_t *__restrict__ ids, const int *__restrict__ ns, int idxw, const void *kv_a, int64_t na,
                      const void *kv_b, float *__restrict__ o, size_t a_stride, size_t b_stride, int seq_mod, const SaRope rope) {
    APUS_PDL_WAIT();
    APUS_PDL_GO();
    __shared__ __align__(16) float s_p[PV_JC][HG];
    __shared__ int32_t s_id[PV_JC];
    const int t = blockIdx.y, h0 = (int)blockIdx.x * HG, tid = threadIdx.x;
    const int own = seq_mod > 0 ? t % seq_mod : t;
    kv_a = reinterpret_cast<const char *>(kv_a) + (size_t)own * a_stride;
    kv_b = reinterpret_cast<const char *>(kv_b) + (size_t)own * b_stride;
    const int n = ns[t];
    const int32_t *idr = ids + (size_t)t * idxw;
    for (int c0 = 0; c0 < d / 2; c0 += 256) {
        const int k2 = c0 + tid;
        const bool on = k2 < d / 2;
        float a0[HG], a1[HG];
#pragma unroll
        for (int a = 0; a < HG; a++) a0[a] = a1[a] = 0.f;
        for (int j0 = 0; j0 < n; j0 += PV_JC) {
            const int cnt = min(PV_JC, n - j0);
            __syncthreads();
            for (int i = tid; i < PV_JC * HG; i += 256) {
                const int a = i / PV_JC, jj = i - a * PV_JC;
                s_p[jj][a] = (jj < cnt && h0 + a < h) ? p[((size_t)t * h + h0 + a) * idxw + j0 + jj] : 0.f;
            }
            for (int i = tid; i < cnt; i += 256) s_id[i] = idr[j0 + i];
            __syncthreads();
            if (on) {
                // LB gathered rows in flight per thread: the rows come from L2 / HBM with nothing else to
                // hide their latency behind (few heads per CTA: little arithmetic per row, so more rows)
                constexpr int LB = HG >= 16 ? 16 : 32;
                for (int jb = 0; jb < cnt; jb += LB) {
                    float2 v[LB];
#pragma unroll
                    for (int u = 0; u < LB; u++) {
                        const int jj = jb + u < cnt ? jb + u : cnt - 1;
                        const int32_t id = s_id[jj];
                        v[u] = id < na ? kv_pair<BF16>(kv_a, (size_t)id, d, k2) : kv_pair<BF16>(kv_b, (size_t)(id - na), d, k2);
                    }
#pragma unroll
                    for (int u = 0; u < LB; u++) {
                        if (jb + u >= cnt) break;
#pragma unroll
                        for (int m = 0; m < HG / 4; m++) {
                            const float4 p4 = *reinterpret_cast<const float4 *>(&s_p[jb + u][4 * m]);
                            const float pa[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                            for (int e = 0; e < 4; e++) {
                                a0[4 * m + e] = __fadd_rn(a0[4 * m + e], __fmul_rn(pa[e], v[u].x));
                                a1[4 * m + e] = __fadd_rn(a1[4 * m + e], __fmul_rn(pa[e], v[u].y));
                            }
                        }
                    }
                }
            }
        }
        if (on) {
            // a thread holds one (even, odd) pair of every head row: the pairs of the rotated tail are
            // turned back here (the operations of the row kernel, c/attn.h:290-299 with -sin)
            const int ri = rope.cs ? k2 - (d - rope.rd) / 2 : -1;
            float co = 1.f, si = 0.f;
            if (ri >= 0) {
                const float *c = rope.cs + (rope.pos ? (size_t)*rope.pos * rope.rd : 0);
                co = c[ri]; si = -c[rope.rd / 2 + ri];
            }
#pragma unroll
            for (int a = 0; a < HG; a++) {
                if (h0 + a >= h) continue;
                float *ov = o + ((size_t)t * h + h0 + a) * d;
                if (n == 0) { ov[2 * k2] = 0.f; ov[2 * k2 + 1] = 0.f; continue; }
                const float dn = den[(size_t)t * h + h0 + a];
                float x1 = bf16_round(__fdiv_rn(a0[a], dn)), x2 = bf16_round(__fdiv_rn(a1[a], dn));
                if (ri >= 0) {
                    const float y1 = bf16_round(__fsub_rn(__fmul_rn(x1, co), __fmul_rn(x2, si)));
                    const float y2 = bf16_round(__fadd_rn(__fmul_rn(x1, si), __fmul_rn(x2, co)));
                    x1 = y1; x2 = y2;
                }
                ov[2 * k2] = x1;
                ov[2 * k2 + 1] = x2;
            }
        }
    }
}

// P.V from staged rows.  A CTA owns HG heads x 2 NPAIR NT channels of a row; a thread owns NPAIR channel pairs
// for all HG heads (one f32x2 accumulator each).  The row segments of T candidates at a time come in two tiles ahead
// of the one that is consumed, by 16-byte cp.async or (BULK) by one bulk copy per segment, issued by the thread that
// holds the candidate's id: a bulk copy costs its SM some 33 cycles whatever its size, so only the widest CTAs, where
// the arithmetic per candidate exceeds that, gain by the instructions it saves; the probabilities of a tile pass through registers into shared memory, each written
// twice side by side ([j][head] pairs, pitch +16 bytes: the stores of 8 candidates x 2 heads fall into different
// banks), so that one 16-byte load gives the factor pairs of two heads.  Per candidate a thread issues HG / 2 + 1
// shared loads for HG * NPAIR packed multiply-adds.
#define PVS_NS 3
template <bool BF16, int HG, int NPAIR, int T, int NT, bool BULK>
struct PvCfg {
    static constexpr int ROWB = NT * NPAIR * (BF16 ? 4 : 8);     // bytes of a row's segment
    static constexpr int PP = HG * 8 + 16;                       // bytes per candidate of the probability tile
    static constexpr int STAGE = T * (ROWB + PP), SMEM = PVS_NS * STAGE + (BULK ? 0 : 4 * T * 4);
};

// The operands of GJ candidates for a thread: its channel pairs and the factor pairs of the heads
template <bool BF16, int HG, int NPAIR, int GJ, int ROWB, int PP>
struct PvOps {
    uint32_t w[GJ][BF16 ? NPAIR : 1];
    ulonglong2 v[GJ][BF16 ? 1 : (NPAIR + 1) / 2], p[GJ][HG / 2];
    __device__ __forceinline__ void load(const unsigned char *rows, const unsigned char *sp, int j0, int tid) {
#pragma unroll
        for (int u = 0; u < GJ; u++) {
            const unsigned char *r = rows + (size_t)(j0 + u) * ROWB + tid * (NPAIR * (BF16 ? 4 : 8));
            if constexpr (BF16 && NPAIR == 2) {
                const uint2 x = *reinterpret_cast<const uint2 *>(r);
                w[u][0] = x.x; w[u][1] = x.y;
            } else if constexpr (BF16) {
                w[u][0] = *reinterpret_cast<const uint32_t *>(r);
            } else if constexpr (NPAIR == 2) {
                v[u][0] = *reinterpret_cast<const ulonglong2 *>(r);
            } else {
                v[u][0].x = *reinterpret_cast<const f32x2 *>(r);
            }
#pragma unroll
            for (int a = 0; a < HG / 2; a++) p[u][a] = *reinterpret_cast<const ulonglong2 *>(sp + (size_t)(j0 + u) * PP + a * 16);
        }
    }
    template <bool FUSED>
    __device__ __forceinline__ void walk(f32x2 (&acc)[HG][NPAIR]) const {
#pragma unroll
        for (int u = 0; u < GJ; u++)
#pragma unroll
            for (int i = 0; i < NPAIR; i++) {
                f32x2 x;
                if constexpr (BF16) x = pack2(__uint_as_float(w[u][i] << 16), __uint_as_float(w[u][i] & 0xffff0000u));
                else x = i ? v[u][0].y : v[u][0].x;
#pragma unroll
                for (int a = 0; a < HG; a++) acc[a][i] = mac2<FUSED>(acc[a][i], a & 1 ? p[u][a >> 1].y : p[u][a >> 1].x, x);
            }
    }
};
// A tile of T candidates (cnt of them in the row); the operands are read GJ candidates ahead of their use
template <bool BF16, bool FUSED, int HG, int NPAIR, int T, int ROWB, int PP>
__device__ __forceinline__ void pv_tile(f32x2 (&acc)[HG][NPAIR], const unsigned char *rows, const unsigned char *sp, int cnt, int tid) {
    constexpr int GJ = HG * NPAIR >= 16 ? 1 : HG * NPAIR >= 8 ? 2 : 4;
    if (cnt == T) {
        PvOps<BF16, HG, NPAIR, GJ, ROWB, PP> A, B;
        A.load(rows, sp, 0, tid);
#pragma unroll 2
        for (int j = 0; j < T; j += 2 * GJ) {
            B.load(rows, sp, j + GJ, tid);
            A.template walk<FUSED>(acc);
            if (j + 2 * GJ < T) A.load(rows, sp, j + 2 * GJ, tid);
            B.template walk<FUSED>(acc);
        }
    } else {
        PvOps<BF16, HG, NPAIR, 1, ROWB, PP> A;
        for (int j = 0; j < cnt; j++) { A.load(rows, sp, j, tid); A.template walk<FUSED>(acc); }
    }
}

template <bool BF16, int HG, int NPAIR, int T, int NT, bool BULK>
__global__ void __launch_bounds__(NT)
sparse_pv_stage_kernel(const float *__restrict__ p, const float *__restrict__ den, int h, int d,
                       const int32_t *__restrict__ ids, const int *__restrict__ ns, int idxw, const void *kv_a, int64_t na,
                       const void *kv_b, float *__restrict__ o, size_t a_stride, size_t b_stride, int seq_mod, const SaRope rope,
                       const int *__restrict__ bad, int *__restrict__ status) {
    APUS_PDL_WAIT();
    APUS_PDL_GO();
    using Cf = PvCfg<BF16, HG, NPAIR, T, NT, BULK>;
    constexpr int ROWB = Cf::ROWB, PP = Cf::PP, STAGE = Cf::STAGE, CPR = ROWB / 16;
    constexpr int NP = T * HG / NT;                         // probabilities of a tile per thread
    static_assert(T * HG % NT == 0 && T <= NT && HG % 2 == 0 && ROWB % 16 == 0 && STAGE % 16 == 0, "tile shape");
    extern __shared__ __align__(16) unsigned char pvs[];
    __shared__ uint64_t s_full[PVS_NS];
    __shared__ volatile int s_abort;
    const int t = blockIdx.y, h0 = (int)blockIdx.x * HG, tid = threadIdx.x;
    const int own = seq_mod > 0 ? t % seq_mod : t;
    const size_t rowsz = (size_t)d * (BF16 ? 2 : 4);
    const char *base_a = reinterpret_cast<const char *>(kv_a) + (size_t)own * a_stride + (size_t)blockIdx.z * ROWB;
    const char *base_b = reinterpret_cast<const char *>(kv_b) + (size_t)own * b_stride + (size_t)blockIdx.z * ROWB - (size_t)na * rowsz;
    const int n = ns[t];
    const bool fused = bad[t] == 0;
    const int32_t *idr = ids + (size_t)t * idxw;
    const int ntile = (n + T - 1) / T;
    auto id_load = [&](int c) { const int j = c * T + tid; return tid < T && j < n ? idr[j] : -1; };
    // tile c's segments.  BULK: thread r copies the one of candidate c T + r (id < 0: past the row's end); otherwise the
    // ids pass through shared memory and every thread copies its 16-byte column of every NT / CPR-th row
    int32_t *s_id = reinterpret_cast<int32_t *>(pvs + (size_t)PVS_NS * STAGE);       // [4][T]
    auto id_store = [&](int c, int32_t v) { if (!BULK && tid < T) s_id[(c & 3) * T + tid] = v; };
    auto stage = [&](int c, int32_t id) {
        if constexpr (!BULK) {
            static_assert(BULK || (NT % CPR == 0 && T * CPR % NT == 0), "copies must divide among the threads");
            if (c < ntile) {
                unsigned char *st = pvs + (size_t)(c % PVS_NS) * STAGE;
                const int cnt = min(T, n - c * T), seg = tid % CPR;
#pragma unroll 8
                for (int i = 0; i < T * CPR / NT; i++) {
                    const int r = tid / CPR + i * (NT / CPR);
                    if (r < cnt) {
                        const int32_t rid = s_id[(c & 3) * T + r];
                        cp_async16(st + (size_t)r * ROWB + seg * 16, (rid < na ? base_a : base_b) + (size_t)rid * rowsz + seg * 16, true);
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            return;
        }
        if (c >= ntile || tid >= T) return;
        uint64_t *bar = &s_full[c % PVS_NS];
        if (id >= 0) {
            mbar_expect_tx(bar, ROWB);
            bulk_load(pvs + (size_t)(c % PVS_NS) * STAGE + (size_t)tid * ROWB, (id < na ? base_a : base_b) + (size_t)id * rowsz, ROWB, bar);
        } else {
            mbar_arrive(bar);
        }
    };
    // probability u of this thread: head 2 (i / 2T) + i % 2, candidate (i / 2) % T with i = tid + NT u
    float preg[NP];
    auto p_load = [&](int c) {
#pragma unroll
        for (int u = 0; u < NP; u++) {
            const int i = tid + NT * u, a = 2 * (i / (2 * T)) + (i & 1), j = c * T + (i >> 1) % T;
            preg[u] = j < n && h0 + a < h ? p[((size_t)t * h + h0 + a) * idxw + j] : 0.f;
        }
    };
    auto p_store = [&](int c) {
        unsigned char *sp = pvs + (size_t)(c % PVS_NS) * STAGE + T * ROWB;
#pragma unroll
        for (int u = 0; u < NP; u++) {
            const int i = tid + NT * u, a = 2 * (i / (2 * T)) + (i & 1), j = (i >> 1) % T;
            *reinterpret_cast<f32x2 *>(sp + (size_t)j * PP + a * 8) = pack2(preg[u], preg[u]);
        }
    };
    f32x2 acc[HG][NPAIR];
#pragma unroll
    for (int a = 0; a < HG; a++)
#pragma unroll
        for (int i = 0; i < NPAIR; i++) acc[a][i] = 0ull;
    if (tid == 0) {
        for (int i = 0; i < PVS_NS; i++) mbar_init(&s_full[i], T);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    int32_t id_next = id_load(2);                              // one tile ahead of the copies that need it
    p_load(0);
    const int32_t id0 = id_load(0), id1 = id_load(1);
    id_store(0, id0);
    id_store(1, id1);
    id_store(2, id_next);
    __syncthreads();
    stage(0, id0);
    stage(1, id1);
    p_store(0);
    int fail = 0;
    for (int c = 0; c < ntile; c++) {
        const int32_t id_after = id_load(c + 3);
        if constexpr (BULK) {
            fail = !mbar_wait(&s_full[c % PVS_NS], (uint32_t)(c / PVS_NS) & 1u, &s_abort);
            if (__syncthreads_or(fail)) { fail = 1; break; }   // tile c has landed for every thread, tile c - 1 is consumed
        } else {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
        }
        stage(c + 2, id_next);
        id_next = id_after;
        if (c + 1 < ntile) p_load(c + 1);
        const unsigned char *st = pvs + (size_t)(c % PVS_NS) * STAGE;
        const int cnt = min(T, n - c * T);
        if (fused) pv_tile<BF16, true, HG, NPAIR, T, ROWB, PP>(acc, st, st + T * ROWB, cnt, tid);
        else pv_tile<BF16, false, HG, NPAIR, T, ROWB, PP>(acc, st, st + T * ROWB, cnt, tid);
        if (c + 1 < ntile) p_store(c + 1);                     // this stage was consumed at tile c - 2
        id_store(c + 3, id_after);                             // slot of tile c - 1, whose copies are all issued
    }
    if (fail) {
        if (tid == 0) atomicCAS(status, 0, 31);               // a row copy did not arrive in time
        for (int i = 0; i < 2000; i++) __nanosleep(1000);      // copies already issued to this CTA's shared memory land
        return;
    }
#pragma unroll
    for (int i = 0; i < NPAIR; i++) {
        const int k2 = ((int)blockIdx.z * NT + tid) * NPAIR + i;       // this channel pair
        const int ri = rope.cs ? k2 - (d - rope.rd) / 2 : -1;
        float co = 1.f, si = 0.f;
        if (ri >= 0) {
            const float *c = rope.cs + (rope.pos ? (size_t)*rope.pos * rope.rd : 0);
            co = c[ri]; si = -c[rope.rd / 2 + ri];
        }
#pragma unroll
        for (int a = 0; a < HG; a++) {
            if (h0 + a >= h) continue;
            float *ov = o + ((size_t)t * h + h0 + a) * d + 2 * k2;
            if (n == 0) { ov[0] = 0.f; ov[1] = 0.f; continue; }
            const float dn = den[(size_t)t * h + h0 + a];
            const float2 s = unpack2(acc[a][i]);
            float x1 = bf16_round(__fdiv_rn(s.x, dn)), x2 = bf16_round(__fdiv_rn(s.y, dn));
            if (ri >= 0) {
                const float y1 = bf16_round(__fsub_rn(__fmul_rn(x1, co), __fmul_rn(x2, si)));
                const float y2 = bf16_round(__fadd_rn(__fmul_rn(x1, si), __fmul_rn(x2, co)));
                x1 = y1; x2 = y2;
            }
            if (((uintptr_t)o & 7) == 0) *reinterpret_cast<float2 *>(ov) = make_float2(x1, x2);
            else { ov[0] = x1; ov[1] = x2; }
        }
    }
}

// Drops negative ids keeping order (reference c/attn.h:1314-1321).
__global__ void compact_ids_kernel(const int32_t *__restrict__ idxs, int idxw,
                                   int32_t *__restrict__ out, int *__restrict__ ns, int *__restrict__ bad) {
    APUS_PDL_WAIT();
    APUS_PDL_GO();
    __shared__ int s_base;
    __shared__ int w_cnt[32];
    const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_base = 0;
    __syncthreads();
    for (int base = 0; base < idxw; base += blockDim.x) {
        int i = base + tid;
        int32_t v = i < idxw ? idxs[(size_t)t * idxw + i] : -1;
        bool keep = v >= 0;
        unsigned m = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) w_cnt[warp] = __popc(m);
        __syncthreads();
        int before = 0, total = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
            if (w < warp) before += w_cnt[w];
            total += w_cnt[w];
        }
        if (keep) out[(size_t)t * idxw + s_base + before + __popc(m & ((1u << lane) - 1u))] = v;
        __syncthreads();
        if (tid == 0) s_base += total;
        __syncthreads();
    }
    if (tid == 0) { ns[t] = s_base; bad[t] = 0; }
}

// Scores / compacted ids between the kernels of a call: the caller's scratch (a model object keeps its own), else a
// buffer of the library that belongs to the call's stream.  Calls on several streams never share one (a shared one
// would let a call read the ids another is writing, or take the walk flags of another's rows); a call holds the lock
// until its last launch, so that those of two threads on one stream do not mix and none loses its buffer to a growing
// one.  A call that is being recorded gets memory that its graph owns.  At most SCR_MAX buffers are kept, the longest
// unused one makes room for a new stream's, apus_cuda_disable frees them all.
#define SCR_MAX 16
struct ScrSlot {
    int dev;
    cudaStream_t st;
    std::thread::id th;                                    // cudaStreamPerThread is another stream in every thread
    DevBuf buf;
    unsigned long long used;
};
static std::mutex g_scr_mu;
static std::vector<ScrSlot> g_scr;
static unsigned long long g_scr_calls = 0;
static void scr_release() {
    std::lock_guard<std::mutex> lock(g_scr_mu);
    for (ScrSlot &s : g_scr) s.buf.release();
    g_scr.clear();
}
struct ScrReg { ScrReg() { on_disable(scr_release, nullptr); } };
static ScrReg g_scr_reg;

struct CallScratch {
    std::unique_lock<std::mutex> lock;
    cudaStream_t st;
    void *p = nullptr;
    bool recorded = false;
    explicit CallScratch(cudaStream_t s) : st(s) {}
    ~CallScratch() { if (recorded && p) cudaFreeAsync(p, st); }
    CallScratch(const CallScratch &) = delete;
    CallScratch &operator=(const CallScratch &) = delete;
    int get(size_t bytes) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        APUS_CUDA_OK(cudaStreamIsCapturing(st, &cs));
        if (cs != cudaStreamCaptureStatusNone) {
            recorded = true;
            APUS_CUDA_OK(cudaMallocAsync(&p, bytes, st));
            return 0;
        }
        int dev = 0;
        APUS_CUDA_OK(cudaGetDevice(&dev));
        const std::thread::id th = st == cudaStreamPerThread ? std::this_thread::get_id() : std::thread::id();
        lock = std::unique_lock<std::mutex>(g_scr_mu);
        ScrSlot *slot = nullptr, *idle = nullptr;
        for (ScrSlot &s : g_scr) {
            if (s.dev == dev && s.st == st && s.th == th) slot = &s;
            if (s.dev == dev && (!idle || s.used < idle->used)) idle = &s;
        }
        if (!slot && (g_scr.size() < SCR_MAX || !idle)) {
            g_scr.push_back(ScrSlot{dev, st, th, DevBuf(), 0});
            slot = &g_scr.back();
        } else if (!slot) {
            APUS_CUDA_OK(cudaDeviceSynchronize());         // another stream may still be using it
            slot = idle;
            slot->st = st; slot->th = th;
        }
        slot->used = ++g_scr_calls;
        return slot->buf.get(bytes, &p);
    }
};
// Layout of that scratch: scores, compacted ids, their counts, denominators, the walk flags of P.V.
struct SaScratch {
    size_t ids, ns, den, bad, bytes;
    SaScratch(int h, int idxw, int s) {
        ids = (size_t)s * h * idxw * sizeof(float);
        ns = (ids + (size_t)s * idxw * sizeof(int32_t) + 255) & ~(size_t)255;
        den = (ns + (size_t)s * sizeof(int) + 255) & ~(size_t)255;
        bad = den + (size_t)s * h * sizeof(float);
        bytes = bad + (size_t)s * sizeof(int);
    }
};
size_t sparse_attn_scratch(int h, int idxw, int s) { return SaScratch(h, idxw, s).bytes; }

// ---- launches of the tiled kernels ----
template <bool BF16, int HL, int CL, int WH, int WC>
static int scores_launch(const float *q, int h, int d, const int32_t *ids, const int *ns, int idxw, int s, float scale,
                         const void *kv_a, int64_t na, const void *kv_b, float *sc, int *bad, cudaStream_t st, size_t sa,
                         size_t sb, int seq_mod) {
    using Cf = ScoreCfg<BF16, HL, CL, WH, WC>;
    auto kern = sparse_scores_tile_kernel<BF16, HL, CL, WH, WC>;
    if (ensure_dyn_smem((const void *)kern, Cf::SMEM + 64)) return 1;
    launch_k(kern, dim3((unsigned)ceil_div(idxw, Cf::CANDS), (unsigned)ceil_div(h, Cf::HEADS), (unsigned)s), Cf::THREADS, Cf::SMEM,
             st, q, h, d, ids, ns, idxw, scale, kv_a, na, kv_b, sc, sa, sb, seq_mod, bad);
    APUS_LAUNCHED();
    return 0;
}
template <bool BF16, int HG, int NPAIR, int T, int NT, bool BULK>
static int pv_launch(const float *sc, const float *den, int h, int d, const int32_t *ids, const int *ns, int idxw, int s,
                     const void *kv_a, int64_t na, const void *kv_b, float *o, const int *bad, cudaStream_t st, size_t sa,
                     size_t sb, int seq_mod, const SaRope &rope) {
    using Cf = PvCfg<BF16, HG, NPAIR, T, NT, BULK>;
    auto kern = sparse_pv_stage_kernel<BF16, HG, NPAIR, T, NT, BULK>;
    int *status = wait_word();
    if (!status || ensure_dyn_smem((const void *)kern, Cf::SMEM + 64)) return 1;
    launch_k(kern, dim3((unsigned)ceil_div(h, HG), (unsigned)s, (unsigned)(d / (2 * NPAIR * NT))), NT, Cf::SMEM, st,
             sc, den, h, d, ids, ns, idxw, kv_a, na, kv_b, o, sa, sb, seq_mod, rope, bad, status);
    APUS_LAUNCHED();
    return 0;
}
template <bool BF16>
static int attn_tiled(const float *q, const float *sink, int h, int d, const int32_t *ids, const int *ns, int idxw, int s,
                      float scale, const void *kv_a, int64_t na, const void *kv_b, float *sc, float *den, int *bad, float *o,
                      cudaStream_t st, size_t sa, size_t sb, int seq_mod, const SaRope &rope) {
#define SA_ARGS q, h, d, ids, ns, idxw, s, scale, kv_a, na, kv_b, sc, bad, st, sa, sb, seq_mod
    // The larger a lane's tile, the fewer shared loads per multiply-add; the smaller, the more warps share the work of a
    // small step.  Three sizes of work, counted in 16-head tiles so that a head count below 64 is not taken for more than
    // it is (us, BF16 rows, d = 512, with 16 heads x 32 candidates of 4 x 1 per lane / 16 x 32 of 4 x 2 / the large tile):
    // the smallest tile while its CTAs have an SM each (64 heads: 1 row of 909 11.8 / 15.2 / 25, 2 rows of 640, 160 CTAs,
    // 16.3 / 15.4 / 25; 32 rows of 16 10.7 / 14.9 / 19), the large one when it has 80 tiles of 64 x 64 (8 rows of 640 32 /
    // 24.4 / 25.5, 32 rows 107 / 76 / 61).  The large one is as tall as the heads: 4 x 4 per lane, 64 heads x 64
    // candidates, 32 x 64 or 16 x 128 (8 heads: 256 rows of 640 129 / 96 as 16 x 128, 224 as 64 x 64; 32 heads: 253 / 178
    // as 32 x 64, 320), unless the rows are shorter than a tile is wide (8 heads, 1,024 rows of 16: 29 / 53).
    const long long ctas0 = (long long)ceil_div(idxw, 32) * ceil_div(h, 16) * s, c16 = (long long)ceil_div(idxw, 64) * ceil_div(h, 16) * s;
    if (ctas0 <= 148) { if (scores_launch<BF16, 4, 1, 1, 4>(SA_ARGS)) return 1; }
    else if (c16 < 320 || (h <= 32 && idxw <= 32)) { if (scores_launch<BF16, 4, 2, 1, 2>(SA_ARGS)) return 1; }
    else if (h <= 16) { if (scores_launch<BF16, 4, 4, 1, 4>(SA_ARGS)) return 1; }
    else if (h <= 32) { if (scores_launch<BF16, 4, 4, 2, 2>(SA_ARGS)) return 1; }
    else if (scores_launch<BF16, 4, 4, 4, 2>(SA_ARGS)) return 1;
#undef SA_ARGS
    // a warp per row once that is a warp and more for every scheduler; with fewer rows the exponentials want a CTA per
    // row (64 rows of 640: 5.1 us against 7.9, 448 of 909: 7.8 / 11, 2,048 of 640: 12.2 / 10.6)
    if (idxw <= 1024 && (long long)s * h >= 1024) {
        const size_t sm = (size_t)8 * ((idxw + 3) & ~3) * sizeof(float);
        launch_k(sparse_softmax_rows_kernel, dim3((unsigned)ceil_div(h, 8), (unsigned)s), 256, sm, st, sc, sink, h, ns, idxw, den, bad);
    } else {
        const size_t sm2 = (size_t)idxw * sizeof(float);
        if (ensure_dyn_smem((const void *)sparse_softmax_kernel, sm2 + 256)) return 1;
        launch_k(sparse_softmax_kernel, dim3((unsigned)h, (unsigned)s), 256, sm2, st, sc, sink, h, ns, idxw, den, bad);
    }
    APUS_LAUNCHED();
    if (d % 256 == 0) {
        // Few rows: few heads per CTA and short chains of instructions per candidate; many rows: many heads per
        // gathered row.  Lines drawn where the measured times cross (64 heads, d = 512, BF16 rows of 640; us with 2 / 4 /
        // 4 / 8 / 8 heads per CTA as listed): 1 row 15.8 / 18.0 / 22.0 / 29.1 / 52.0 (42.6 before), 4 rows 20.4 / 19.3 /
        // 23.3 / 29.5 / 52.1, 12 rows 57 / 44 / 36 / 41 / 53, 16 rows 74 / 59 / 44 / 41 / 53, 32 rows 131 / 99 / 81 / 76 /
        // 63 (94 before).  The last takes rows of 512 channels, with 256 its CTA is half as wide.
        const long long w16 = (long long)s * ceil_div(h, 16) * (d / 128);
#define PV_ARGS sc, den, h, d, ids, ns, idxw, s, kv_a, na, kv_b, o, bad, st, sa, sb, seq_mod, rope
        if (w16 <= 32) return pv_launch<BF16, 2, 1, 64, 64, false>(PV_ARGS);
        if (w16 <= 64) return pv_launch<BF16, 4, 1, 64, 64, false>(PV_ARGS);
        if (w16 <= 224) return pv_launch<BF16, 4, 1, 32, 64, false>(PV_ARGS);
        if (w16 <= 352) return pv_launch<BF16, 8, 1, 32, 128, false>(PV_ARGS);
        if (d % 512 == 0) return pv_launch<BF16, 8, 2, 16, 128, true>(PV_ARGS);
        return pv_launch<BF16, 8, 2, (BF16 ? 32 : 16), 64, true>(PV_ARGS);
#undef PV_ARGS
    }
    if (h >= 16 && (long long)s * ceil_div(h, 16) >= 96)
        launch_k(sparse_pv_tile_kernel<BF16, 16>, dim3((unsigned)ceil_div(h, 16), (unsigned)s), 256, 0, st, sc, den, h, d, ids, ns,
                 idxw, kv_a, na, kv_b, o, sa, sb, seq_mod, rope);
    else
        launch_k(sparse_pv_tile_kernel<BF16, 4>, dim3((unsigned)ceil_div(h, 4), (unsigned)s), 256, 0, st, sc, den, h, d, ids, ns,
                 idxw, kv_a, na, kv_b, o, sa, sb, seq_mod, rope);
    APUS_LAUNCHED();
    return 0;
}

int sparse_attn(const float *q, const float *sink, int h, int d,
                const int32_t *idxs, int idxw, int s, float scale,
                const void *kv_a, int64_t na, const void *kv_b, int64_t nb,
                int kv_bf16, float *o, cudaStream_t st, long long kv_a_stride, long long kv_b_stride,
                void *callers, size_t callers_cap, int seq_mod, bool ids_ready, const SaRope *rope) {
    (void)nb;
    const size_t esz = kv_bf16 ? 2 : 4;
    const size_t sa = (size_t)kv_a_stride * esz, sb = (size_t)kv_b_stride * esz;
    APUS_REQUIRE(d % 2 == 0 && d <= 1024, "sparse_attn: d=%d unsupported", d);
    APUS_REQUIRE((size_t)idxw * sizeof(float) <= 160 * 1024, "sparse_attn: idxw=%d too wide", idxw);
    if (s <= 0 || idxw <= 0) return 0;
    const SaScratch lay(h, idxw, s);
    APUS_REQUIRE(!callers || lay.bytes <= callers_cap, "sparse_attn: scratch of %zu bytes given, %zu needed", callers_cap, lay.bytes);
    CallScratch own(st);
    if (!callers && own.get(lay.bytes)) return 1;
    char *scratch = (char *)(callers ? callers : own.p);
    float *sc = (float *)scratch;
    int32_t *ids = (int32_t *)(scratch + lay.ids);
    int *ns = (int *)(scratch + lay.ns);
    float *den = (float *)(scratch + lay.den);
    int *bad = (int *)(scratch + lay.bad);
    APUS_REQUIRE(!ids_ready || callers, "sparse_attn: compacted ids need the caller's scratch");
    if (!ids_ready) {
        launch_k(compact_ids_kernel, s, 256, 0, st, idxs, idxw, ids, ns, bad);
        APUS_LAUNCHED();
    }
    const SaRope no_rope = {nullptr, nullptr, 0};
    static const int tiled = [] { const char *e = getenv("APUS_ATTN_TILED"); return !(e && e[0] == '0'); }();
    if (tiled && d % 64 == 0) {
        const SaRope rp = rope ? *rope : no_rope;
        return kv_bf16 ? attn_tiled<true>(q, sink, h, d, ids, ns, idxw, s, scale, kv_a, na, kv_b, sc, den, bad, o, st, sa, sb, seq_mod, rp)
                       : attn_tiled<false>(q, sink, h, d, ids, ns, idxw, s, scale, kv_a, na, kv_b, sc, den, bad, o, st, sa, sb, seq_mod, rp);
    }
    size_t sm1 = ((size_t)SA_IDS * (d + 1) + (size_t)SA_HEADS * d) * sizeof(float);
    dim3 g1((unsigned)ceil_div(idxw, SA_IDS), (unsigned)ceil_div(h, SA_HEADS), (unsigned)s);
    size_t sm2 = (size_t)idxw * sizeof(float);
    dim3 g2((unsigned)h, (unsigned)s);
    // each kernel's limit only ever grows (per device): a later call with a smaller size keeps the larger one
    if (ensure_dyn_smem(kv_bf16 ? (const void *)sparse_scores_kernel<true> : (const void *)sparse_scores_kernel<false>, sm1) ||
        ensure_dyn_smem(kv_bf16 ? (const void *)sparse_pv_kernel<true> : (const void *)sparse_pv_kernel<false>, sm2))
        return 1;
    if (kv_bf16) {
        launch_k(sparse_scores_kernel<true>, g1, SA_IDS * SA_HEADS, sm1, st, q, h, d, ids, ns, idxw, scale,
                                                                       kv_a, na, kv_b, sc, sa, sb, seq_mod);
        APUS_LAUNCHED();
        launch_k(sparse_pv_kernel<true>, g2, 256, sm2, st, sc, sink, h, d, ids, ns, idxw, kv_a, na, kv_b, o, sa, sb, seq_mod);
        APUS_LAUNCHED();
    } else {
        launch_k(sparse_scores_kernel<false>, g1, SA_IDS * SA_HEADS, sm1, st, q, h, d, ids, ns, idxw, scale,
                                                                        kv_a, na, kv_b, sc, sa, sb, seq_mod);
        APUS_LAUNCHED();
        launch_k(sparse_pv_kernel<false>, g2, 256, sm2, st, sc, sink, h, d, ids, ns, idxw, kv_a, na, kv_b, o, sa, sb, seq_mod);
        APUS_LAUNCHED();
    }
    if (rope && rope->cs) {                           // these kernels do not rotate: the row kernel does
        const RowDyn dyn = {rope->pos, 0, 0, 0};
        return row_ops(o, d, o, d, s * h, d, ROW_ROPE_INV, nullptr, 0.f, rope->rd, rope->cs, s * h, 0, st, rope->pos ? &dyn : nullptr);
    }
    return 0;
}

int sparse_attn_compact(const int32_t *idxs, int h, int idxw, int s, void *scratch, size_t scratch_cap, cudaStream_t st) {
    if (s <= 0 || idxw <= 0) return 0;
    const SaScratch lay(h, idxw, s);
    APUS_REQUIRE(scratch && lay.bytes <= scratch_cap, "sparse_attn_compact: scratch of %zu bytes given, %zu needed", scratch_cap,
                 lay.bytes);
    char *p = (char *)scratch;
    launch_k(compact_ids_kernel, s, 256, 0, st, idxs, idxw, (int32_t *)(p + lay.ids), (int *)(p + lay.ns), (int *)(p + lay.bad));
    APUS_LAUNCHED();
    return 0;
}

}  // namespace apus
