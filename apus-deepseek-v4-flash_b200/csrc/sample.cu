// Temperature + nucleus (top-p) sampling and the splitmix64 stream on the device
// (reference c/sample.h:91-180): per row
//   p_i = (float)(expf((l_i - max) / temp) / sum)            (sum in double)
//   order the tokens by (p descending, index ascending)
//   keep token i of that order iff the mass before it is <= top_p
//   draw: first kept token whose renormalised inclusive mass exceeds u.
//
// The reference sorts all n probabilities.  Both walks over the sorted list
// ask the same question -- "which is the first token, in (p desc, index asc)
// order, whose inclusive prefix mass exceeds M?" -- and that is a WEIGHTED
// SELECTION, answered here without sorting: four radix passes over the
// order-preserving integer image of p, each building a 256-bin histogram of
// probability MASS under the prefix found so far, locate the value p* at which
// the running mass crosses M; the ties at p* are then counted in index order.
// Mass is accumulated as 2^-60 fixed point in integers, so the sums are
// exact, associative and therefore deterministic whatever the order of the
// atomic adds (the reference's double sums differ from exact sums by ~1e-16,
// which can only matter for a u within that distance of a boundary).
//
// A row of more than 2,048 entries is spread over a cluster of eight CTAs whose
// slices of the probabilities stay in their shared memory for all sweeps (max,
// exponentials, eight histogram passes).  What bounds it is latency: twelve
// cluster barriers (one more when the uniform comes from the generator) and
// the sweeps between them; the row itself is read once.  Vocabulary 129,280,
// five rows: about 4,000 us with one CTA per row sweeping L2 and adding 64-bit
// masses to shared memory (a compare-and-swap loop per add, all lanes on the
// few bins the leading digit has), 85 us like this; 32 rows 240 us.
#include <cooperative_groups.h>
#include "common.cuh"
#include "kernels.cuh"

namespace apus {

namespace {

namespace cg = cooperative_groups;

constexpr int SMP_THREADS = 1024;
constexpr int SMP_BATCH = 1 << 17;                        // elements of a slice between flushes of the 32-bit counters
constexpr double SMP_ONE = 1152921504606846976.0;        // 2^60

__device__ __forceinline__ unsigned long long mass_of(float p) {
    return (unsigned long long)((double)p * SMP_ONE);     // exact: p has 24 significant bits, p <= 1
}

struct SmpShared {
    unsigned lo[256], mid[256], hi[256];      // this slice's histogram: bits 0..14, 15..29 and 30.. of the masses
    unsigned long long mass[2][256];          // ... as one number each, read by the other CTAs (two, alternating)
    unsigned long long tot[256];              // the row's histogram
    unsigned long long above;
    unsigned digit;
    int cnt[32];
    double sum[32], part;                     // part: read by the other CTAs
    float mx[32], mxpart;
};

struct Sel {                 // answer of first_exceed
    int found;               // 0: the total mass does not exceed M
    unsigned key;            // integer image of p*
    unsigned long long above;// mass of the tokens with p > p*
    unsigned long long k;    // the k-th tie at p* (1-based, index order) is the token
    unsigned long long before;// ties in the slices of lower rank
    unsigned long long here; // ties in this slice
};

// First token, in (p desc, index asc) order, whose inclusive prefix mass exceeds M: every thread of the
// cluster (CL CTAs) gets the same found / key / above / k.  p: this slice's np probabilities.  row_mass (may be null): the row's mass.
template <int CL>
__device__ __forceinline__ Sel first_exceed(cg::cluster_group &cluster, SmpShared &S, const float *p, int np,
                                            unsigned long long M, unsigned long long *row_mass) {
    const int tid = threadIdx.x, lane = tid & 31;
    unsigned prefix = 0;
    unsigned long long above = 0;
    Sel r = {1, 0, 0, 0, 0, 0};
    for (int pass = 0; pass < 4; pass++) {
        const int shift = 24 - 8 * pass, buf = pass & 1;
        const unsigned himask = pass ? (0xffffffffu << (shift + 8)) : 0u;
        unsigned long long mine = 0;
        for (int b0 = 0; b0 < np || b0 == 0; b0 += SMP_BATCH) {
            const int b1 = min(np, b0 + SMP_BATCH);
            if (tid < 256) S.lo[tid] = S.mid[tid] = S.hi[tid] = 0;
            __syncthreads();
            for (int i = b0 + tid; __any_sync(0xffffffffu, i < b1); i += SMP_THREADS) {
                const float v = i < b1 ? p[i] : 0.f;
                const unsigned key = __float_as_uint(v);  // p >= 0: the bit pattern orders like the value
                const unsigned long long m = mass_of(v);
                const bool in = m != 0 && (key & himask) == prefix;   // massless tokens cannot cross anything
                const unsigned act = __ballot_sync(0xffffffffu, in);
                if (!act) continue;
                const unsigned b = (key >> shift) & 0xffu;
                unsigned lo = (unsigned)m & 0x7fffu, mid = (unsigned)(m >> 15) & 0x7fffu, hi = (unsigned)(m >> 30);
                int same = 0;
                if (in) __match_all_sync(act, b, &same);
                if (in && same) {                         // a warp on one bin (the leading digit of a flat row): one add
                    lo = __reduce_add_sync(act, lo); mid = __reduce_add_sync(act, mid); hi = __reduce_add_sync(act, hi);
                }
                if (in && (!same || lane == __ffs(act) - 1)) {
                    atomicAdd(&S.lo[b], lo); atomicAdd(&S.mid[b], mid); atomicAdd(&S.hi[b], hi);
                }
            }
            __syncthreads();
            if (tid < 256)
                mine += (unsigned long long)S.lo[tid] + ((unsigned long long)S.mid[tid] << 15) + ((unsigned long long)S.hi[tid] << 30);
        }
        if (tid < 256) S.mass[buf][tid] = mine;
        cluster.sync();                                   // the eight slices' histograms stand
        if (tid < 256) {
            unsigned long long t = 0;
#pragma unroll
            for (int q = 0; q < CL; q++) t += *cluster.map_shared_rank(&S.mass[buf][tid], q);
            S.tot[tid] = t;
        }
        __syncthreads();
        if (tid < 32) {
            // lane L holds bins 255 - 8L .. 248 - 8L; a warp scan finds the lane where the running mass passes M
            unsigned long long c[8], tot = 0;
#pragma unroll
            for (int j = 0; j < 8; j++) { c[j] = S.tot[255 - 8 * lane - j]; tot += c[j]; }
            unsigned long long inc = tot;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const unsigned long long v = __shfl_up_sync(0xffffffffu, inc, off);
                if (lane >= off) inc += v;
            }
            const unsigned hit = __ballot_sync(0xffffffffu, above + inc > M);
            if (!hit && lane == 31) { S.digit = 0xffffffffu; S.above = inc; }
            if (hit && lane == __ffs(hit) - 1) {
                unsigned long long acc = above + inc - tot;
                int b = 0;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    if (acc + c[j] > M) { b = 255 - 8 * lane - j; break; }
                    acc += c[j];
                }
                S.digit = (unsigned)b; S.above = acc;
            }
            if (pass == 0 && row_mass) {
                const unsigned long long whole = __shfl_sync(0xffffffffu, inc, 31);
                if (lane == 0) S.tot[0] = whole;          // bin 0 was read above
            }
        }
        __syncthreads();
        if (pass == 0 && row_mass) *row_mass = S.tot[0];
        const unsigned b = S.digit;
        if (b == 0xffffffffu) { r.found = 0; cluster.sync(); return r; }
        above = S.above;
        prefix |= b << shift;
        if (pass == 3) {
            // a slice's mass under the whole key is its number of ties at p* times their mass
            const unsigned long long pm = mass_of(__uint_as_float(prefix));
            unsigned long long ties = 0;
            const int rank = (int)cluster.block_rank();
            for (int q = 0; q < CL; q++) {
                const unsigned long long n = *cluster.map_shared_rank(&S.mass[buf][b], q) / pm;
                if (q == rank) { r.before = ties; r.here = n; }
                ties += n;
            }
            r.k = (M - above) / pm + 1;
            if (r.k > ties) r.k = ties;                   // cannot happen for an exact crossing
            r.key = prefix; r.above = above;
            cluster.sync();                               // the histograms are free again
        }
        __syncthreads();
    }
    return r;
}

// u == NULL: the row's uniform comes from its splitmix64 state (advanced here).
template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(SMP_THREADS)
sample_rows_kernel(const float *__restrict__ logits, int n, float temp, float top_p,
                   const double *__restrict__ u_in, unsigned long long *__restrict__ rng,
                   float *probs, int in_smem, int32_t *__restrict__ out) {
    APUS_PDL_WAIT();
    APUS_PDL_GO();
    extern __shared__ float s_slice[];
    __shared__ SmpShared S;
    cg::cluster_group cluster = cg::this_cluster();
    const int row = blockIdx.x / CL, rank = (int)cluster.block_rank(), tid = threadIdx.x, lane = tid & 31;
    const int per = (n + CL - 1) / CL, i0 = min(n, rank * per), np = min(n, i0 + per) - i0;
    const float *l = logits + (size_t)row * n + i0;
    float *p = in_smem ? s_slice : probs + (size_t)row * n + i0;
    // max
    float mx = -INFINITY;
    for (int i = tid; i < np; i += SMP_THREADS) {
        const float v = l[i];
        if (in_smem) p[i] = v;
        mx = fmaxf(mx, v);
    }
    mx = warp_max(mx);
    if (lane == 0) S.mx[tid >> 5] = mx;
    __syncthreads();
    if (tid < 32) {
        mx = warp_max(S.mx[lane]);
        if (lane == 0) S.mxpart = mx;
    }
    cluster.sync();
#pragma unroll
    for (int q = 0; q < CL; q++) { const float v = *cluster.map_shared_rank(&S.mxpart, q); mx = q ? fmaxf(mx, v) : v; }
    // softmax: f32 exponent argument, double sum (a tree here), one rounding back to f32
    double part = 0.0;
    for (int i = tid; i < np; i += SMP_THREADS) {
        const float e = exp_rn(__fdiv_rn(__fsub_rn(in_smem ? p[i] : l[i], mx), temp));
        p[i] = e;
        part += (double)e;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) S.sum[tid >> 5] = part;
    __syncthreads();
    if (tid < 32) {
        part = S.sum[lane];
#pragma unroll
        for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        if (lane == 0) S.part = part;
    }
    cluster.sync();
    double sum = 0.0;
#pragma unroll
    for (int q = 0; q < CL; q++) sum += *cluster.map_shared_rank(&S.part, q);
    for (int i = tid; i < np; i += SMP_THREADS) p[i] = (float)((double)p[i] / sum);
    // the row's uniform
    double u;
    if (u_in) u = u_in[row];
    else {
        unsigned long long s = rng[row] + 0x9E3779B97F4A7C15ull, z = s;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        u = (double)(z >> 11) * 0x1.0p-53;
        cluster.sync();                                      // every CTA has read the state
        if (rank == 0 && tid == 0) rng[row] = s;
    }
    // nucleus: tokens are kept up to and including the first whose inclusive mass exceeds top_p
    // (top_p >= 1.5 can never be exceeded by probabilities: then this call only adds up the row's mass)
    const double tp = (double)top_p;
    unsigned long long total = 0;
    const Sel cut = first_exceed<CL>(cluster, S, p, np, tp >= 1.5 ? ~0ull : tp <= 0.0 ? 0ull : (unsigned long long)(tp * SMP_ONE), &total);
    const unsigned long long kept = cut.found ? cut.above + cut.k * mass_of(__uint_as_float(cut.key)) : total;
    // draw inside the kept mass
    const unsigned long long Mu = (unsigned long long)(u * (double)kept);
    const Sel d = first_exceed<CL>(cluster, S, p, np, Mu < kept ? Mu : kept - 1, nullptr);
    if (!d.found) {                                          // no mass at all (logits without a finite maximum)
        if (rank == 0 && tid == 0) out[row] = 0;
        return;
    }
    // the slice that holds the k-th tie finds it: thread t counts the contiguous range [t * chunk, (t + 1) * chunk)
    if (d.before < d.k && d.k <= d.before + d.here) {        // one CTA of the cluster
        const int chunk = (np + SMP_THREADS - 1) / SMP_THREADS, lo = min(np, tid * chunk), hi = min(np, lo + chunk);
        int cnt = 0;
        for (int i = lo; i < hi; i++) cnt += __float_as_uint(p[i]) == d.key;
        int inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) S.cnt[tid >> 5] = inc;
        __syncthreads();
        int before = inc - cnt;
        for (int w = 0; w < (tid >> 5); w++) before += S.cnt[w];
        const int want = (int)(d.k - d.before);
        if (before < want && want <= before + cnt)
            for (int i = lo; i < hi; i++)
                if (__float_as_uint(p[i]) == d.key && ++before == want) { out[row] = i0 + i; break; }
    }
}

}  // namespace

// logits [rows, n] -> tokens [rows]; temp <= 0: greedy.  probs: scratch [rows, n] floats.
// u (device, [rows], nullable) are explicit uniforms in [0, 1); otherwise rng [rows]
// holds the rows' splitmix64 states and is advanced by one draw.
template <int CL>
static int sample_launch(const float *logits, int n, int rows, float temp, float top_p, const double *u, unsigned long long *rng,
                         float *probs, int32_t *out, cudaStream_t st) {
    // slices up to 160 KB stay in shared memory (clusters of eight: vocabularies up to 327,680), longer ones in `probs`
    const size_t slice = (size_t)ceil_div(n, CL) * sizeof(float);
    const int in_smem = slice <= 160 * 1024;
    if (in_smem && ensure_dyn_smem((const void *)sample_rows_kernel<CL>, slice)) return 1;
    launch_k(sample_rows_kernel<CL>, rows * CL, SMP_THREADS, in_smem ? slice : 0, st, logits, n, temp, top_p, u, rng, probs,
             in_smem, out);
    APUS_LAUNCHED();
    return 0;
}

int sample_rows(const float *logits, int n, int rows, float temp, float top_p, const double *u,
                unsigned long long *rng, float *probs, int32_t *out, cudaStream_t st) {
    if (rows <= 0) return 0;
    if (temp <= 0.f) return argmax_rows(logits, n, rows, out, st);
    APUS_REQUIRE(u || rng, "sample: neither uniforms nor generator states given");
    // Short rows leave a cluster nothing to share out but its barriers, and fewer clusters than CTAs fit the GPU: one CTA
    // per row up to 2,048 entries (B200, 256 entries: 1 row 17.6 us with one CTA, 31.0 with eight, 64 rows 18.5 / 154;
    // 2,000 entries, 1 row 22.4 / 32.2; 8,192 entries 37.8 / 34.0).
    return n <= 2048 ? sample_launch<1>(logits, n, rows, temp, top_p, u, rng, probs, out, st)
                     : sample_launch<8>(logits, n, rows, temp, top_p, u, rng, probs, out, st);
}

}  // namespace apus
