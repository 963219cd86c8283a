// Host-side planning and the small kernels around the fused pass: the
// launch dispatch of the track kernels (instantiated per precision in
// phk_track_f32.cu / phk_track_f64.cu), the fixed-order merge of the
// per-CTA partials, the wake convolution and the batched merge / wake
// kernels.
#include "phk_track64.cuh"

namespace phk {

size_t track_smem_bytes(int32_t dtype, int32_t Sa, int32_t Sp) {
    // a turn's pending kicks: four dipolar kicks (resonator and resistive
    // wall, both planes), staged as one summed table per plane (the launched
    // grid is the caller's column count either way)
    if (dtype == PHK_F64) {
        const size_t tables = (size_t)2 * Sp * sizeof(double) <= 48 * 1024 ? 2 : 0;
        return track64_smem(Sa, Sp, (int)tables, true, true).bytes;
    }
    int ks, st;
    return smem_for(Sa, Sp, 2, true, &ks, &st);
}

// Compile-time shape of a program (see TrackShape), from its op kinds.
int program_shape(const phk_program* prog) {
    const int n = prog->n_ops;
    int k[4] = {0, 0, 0, 0};
    for (int i = 0; i < n && i < 4; ++i) k[i] = prog->op[i].kind;
    if (n == 0) return SHAPE_NONE;
    // the shapes read op[0]'s detuners from det[0] on
    if (k[0] == PHK_OP_TRANSVERSE && prog->op[0].det_begin != 0)
        return SHAPE_GENERIC;
    if (n == 1 && k[0] == PHK_OP_TRANSVERSE) return SHAPE_T;
    if (n == 2 && k[0] == PHK_OP_TRANSVERSE && k[1] == PHK_OP_LINEAR_LONG)
        return SHAPE_T_LIN;
    if (n == 4 && k[0] == PHK_OP_TRANSVERSE && k[1] == PHK_OP_DRIFT &&
        k[2] == PHK_OP_RF_KICK && k[3] == PHK_OP_DRIFT)
        return SHAPE_T_RF;
    return SHAPE_GENERIC;
}

// partial columns (= clusters) of an accumulating launch over n particles
int track_grid(int64_t n, int32_t dtype, int32_t n_slices) {
    // size for an accumulation with a pending kick on the same slicing (the
    // largest shared-memory layout of a turn)
    const size_t smem = track_smem_bytes(dtype, n_slices, n_slices);
    const int vec = dtype == PHK_F64 ? 1 : kF32Vec;
    // FP64: a column per CTA; FP32: a column per cluster
    const int cluster = dtype == PHK_F64 ? 1 : kCluster;
    const int nc = dtype == PHK_F64 ? track_ctas_f64(smem)
                                    : track_clusters_f32(smem);
    const int64_t tiles = (n + (int64_t)kTrackThreads * vec - 1) /
                          ((int64_t)kTrackThreads * vec);
    int64_t g = nc;
    const int64_t need = (tiles + cluster - 1) / cluster;
    if (need < g) g = need;
    if (g < 1) g = 1;
    return (int)g;
}

int launch_track(const phk_program* prog, const phk_coords* c,
                 const phk_kick_set* pk, const phk_accum* acc,
                 cudaStream_t st) {
    int ld, stm;
    track_masks(prog, pk, acc, &ld, &stm);
    uintptr_t align = 0;
    void* ptrs[6] = {c->x, c->xp, c->y, c->yp, c->z, c->dp};
    for (int q = 0; q < 6; ++q)
        if ((ld >> q) & 1) align |= reinterpret_cast<uintptr_t>(ptrs[q]);
    const bool vec_ok = (align & 15) == 0;
    if (c->dtype == PHK_F64)
        return launch_track_f64(prog, c, pk, acc, ld, stm, vec_ok, st);
    return launch_track_f32(prog, c, pk, acc, ld, stm, vec_ok, st);
}

// ===================================================================
// fixed-order merge of the per-CTA partials (one warp per slice)
// ===================================================================

// Fixed-order sum of the partial columns [g0, g1) of slice s (P laid out
// [3][S][G]) and the finalised outputs, by LANES adjacent lanes (`lane` of
// them); all 32 lanes of the warp call it.
template <int LANES>
__device__ __forceinline__ void merge_slice(const double* __restrict__ P,
                                            int S, int G, int s, int g0,
                                            int g1, int32_t* counts,
                                            double* mean_x, double* mean_y,
                                            double* moments, int lane) {
    const double* pc = P + (int64_t)s * G;
    const double* px = P + (int64_t)(S + s) * G;
    const double* py = P + (int64_t)(2 * S + s) * G;
    // four independent strided partial sums per lane (loads in flight),
    // combined in a fixed order: the result does not depend on timing
    double c[4] = {0, 0, 0, 0}, sx[4] = {0, 0, 0, 0}, sy[4] = {0, 0, 0, 0};
    int g = g0 + lane;
    for (; g + 3 * LANES < g1; g += 4 * LANES) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            c[u] += pc[g + LANES * u];
            sx[u] += px[g + LANES * u];
            sy[u] += py[g + LANES * u];
        }
    }
    for (; g < g1; g += LANES) {
        c[0] += pc[g];
        sx[0] += px[g];
        sy[0] += py[g];
    }
    double tc = (c[0] + c[1]) + (c[2] + c[3]);
    double tx = (sx[0] + sx[1]) + (sx[2] + sx[3]);
    double ty = (sy[0] + sy[1]) + (sy[2] + sy[3]);
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
        tc += __shfl_xor_sync(0xffffffffu, tc, o);
        tx += __shfl_xor_sync(0xffffffffu, tx, o);
        ty += __shfl_xor_sync(0xffffffffu, ty, o);
    }
    if (lane != 0) return;
    const int32_t n = (int32_t)tc;
    // stats.pyx:251-253: divide non-empty slices by their count
    const double mx = n ? dvd(tx, (double)n) : 0.0;
    const double my = n ? dvd(ty, (double)n) : 0.0;
    if (counts) counts[s] = n;
    if (mean_x) mean_x[s] = mx;
    if (mean_y) mean_y[s] = my;
    if (moments) {
        // wake_kicks.py:217-218: n_macroparticles_per_slice * mean
        moments[s] = (double)n;
        moments[S + s] = mul((double)n, mx);
        moments[2 * S + s] = mul((double)n, my);
    }
}

// One warp, one CTA per slice.  Bound by FP64, 64 instructions of 19 cycles
// for a slice, so the slices are spread over the SMs: eight to a CTA kept 7 of
// them busy at 50 slices and 63 at 500 (50 slices: 9.4 us, now 6.9 from cold
// caches; 16 or 8 lanes per slice have fewer instructions but longer chains: 200
// slices, the whole turn 42.2 and 43.5 us against 41.3).
__global__ void finalize_kernel(const double* __restrict__ P, int S, int G,
                                int32_t* counts, double* mean_x,
                                double* mean_y, double* moments) {
    merge_slice<32>(P, S, G, blockIdx.x, 0, G, counts, mean_x, mean_y, moments,
                    threadIdx.x);
}

int launch_finalize(const phk_accum* acc, int32_t* counts, double* mean_x,
                    double* mean_y, double* moments, cudaStream_t st) {
    const int S = acc->slicer.n_slices;
    finalize_kernel<<<S, 32, 0, st>>>(acc->partials, S, acc->grid,
                                                counts, mean_x, mean_y,
                                                moments);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return set_error(PHK_ECUDA, "phk_slice_finalize launch: %s",
                         cudaGetErrorString(e));
    count_launches(1);
    return PHK_OK;
}

// ===================================================================
// compensated column sums of a particle shard (one warp per slice)
// ===================================================================

// Error-free sum: s + e == a + b exactly (Knuth's TwoSum, six operations,
// no branch); symmetric in a and b.
__device__ __forceinline__ void two_sum(double a, double b, double* s,
                                        double* e) {
    const double t = add(a, b);
    const double bb = sub(t, a);
    *e = add(sub(a, sub(t, bb)), sub(b, bb));
    *s = t;
}

// (hi, lo) pairs: hi the running sum, lo the running sum of the exact
// rounding errors; combining two pairs adds their lows and the error of
// the high sum.
__device__ __forceinline__ void dd_combine(double& hi, double& lo, double bh,
                                           double bl) {
    double s, e;
    two_sum(hi, bh, &s, &e);
    lo = add(add(lo, bl), e);
    hi = s;
}

// Per slice s and quantity q (count, sum x, sum y): lane l adds columns
// l, l + 32, ... in order into its (hi, lo) pair, then the lanes combine
// in a fixed butterfly (partner l ^ 16, ^ 8, ^ 4, ^ 2, ^ 1); lane 0 writes
// out[(0 * 3 + q) * S + s] = hi, out[(1 * 3 + q) * S + s] = lo.  hi + lo
// is the sum of the columns to about 2^-106 of the largest partial sum,
// so sums of disjoint column sets merged the same way (phk_slice_merge on
// the pairs of every shard) round to the same double as one fold over
// all columns.
__global__ void slice_sums_kernel(const double* __restrict__ P, int S, int G,
                                  double* __restrict__ out) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= S) return;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double* pc = P + ((int64_t)q * S + warp) * G;
        double hi = 0.0, lo = 0.0;
        for (int g = lane; g < G; g += 32) {
            double s, e;
            two_sum(hi, pc[g], &s, &e);
            hi = s;
            lo = add(lo, e);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double bh = __shfl_xor_sync(0xffffffffu, hi, o);
            const double bl = __shfl_xor_sync(0xffffffffu, lo, o);
            dd_combine(hi, lo, bh, bl);
        }
        if (lane == 0) {
            out[(int64_t)q * S + warp] = hi;
            out[(int64_t)(3 + q) * S + warp] = lo;
        }
    }
}

int launch_slice_sums(const phk_accum* acc, double* out, cudaStream_t st) {
    const int S = acc->slicer.n_slices;
    const int threads = 256;
    const int blocks = (S * 32 + threads - 1) / threads;
    slice_sums_kernel<<<blocks, threads, 0, st>>>(acc->partials, S, acc->grid,
                                                  out);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return set_error(PHK_ECUDA, "phk_slice_sums launch: %s",
                         cudaGetErrorString(e));
    count_launches(1);
    return PHK_OK;
}

// Rank-ordered merge of the (hi, lo) pairs of n_shards shards, laid out
// [n_shards][2][3][S]: shard 0's pair, combined with shard 1's, then 2's,
// ...; then the finalised outputs of phk_slice_finalize from the totals
// hi + lo.  One thread per slice.
__global__ void slice_merge_kernel(const double* __restrict__ sums,
                                   int n_shards, int S, int32_t* counts,
                                   double* mean_x, double* mean_y,
                                   double* moments) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    double t[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        double hi = sums[(int64_t)q * S + s];
        double lo = sums[(int64_t)(3 + q) * S + s];
        for (int r = 1; r < n_shards; ++r) {
            const double* b = sums + (int64_t)r * 6 * S;
            dd_combine(hi, lo, b[(int64_t)q * S + s], b[(int64_t)(3 + q) * S + s]);
        }
        t[q] = add(hi, lo);
    }
    const int32_t n = (int32_t)t[0];
    const double mx = n ? dvd(t[1], (double)n) : 0.0;
    const double my = n ? dvd(t[2], (double)n) : 0.0;
    if (counts) counts[s] = n;
    if (mean_x) mean_x[s] = mx;
    if (mean_y) mean_y[s] = my;
    if (moments) {
        moments[s] = (double)n;
        moments[S + s] = mul((double)n, mx);
        moments[2 * S + s] = mul((double)n, my);
    }
}

int launch_slice_merge(const double* sums, int n_shards, int S,
                       int32_t* counts, double* mean_x, double* mean_y,
                       double* moments, cudaStream_t st) {
    const int threads = 128;
    const int blocks = (S + threads - 1) / threads;
    slice_merge_kernel<<<blocks, threads, 0, st>>>(sums, n_shards, S, counts,
                                                   mean_x, mean_y, moments);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return set_error(PHK_ECUDA, "phk_slice_merge launch: %s",
                         cudaGetErrorString(e));
    count_launches(1);
    return PHK_OK;
}

// ===================================================================
// wake convolution
// ===================================================================

// numpy path: one warp for target slice i of kick k; lanes split the sources.
// Each lane keeps its partial sums over every stored turn and the warp reduces
// once at the end (the reference sums each turn's convolution, then the turns:
// the same terms, regrouped; GB300's FP64 pipe makes the per-turn reductions the
// larger part of the cost otherwise).
__device__ __forceinline__ void wake_conv_one(const phk_wake_set& w, int k, int i,
                                              int lane) {
    const int S = w.n_slices;
    const phk_wake_kick& kk = w.kick[k];
    const int L2 = 2 * S - 1;
    double p0 = 0.0, p1 = 0.0, p2 = 0.0, p3 = 0.0;
    int slot = (w.head % w.ring_len + w.ring_len) % w.ring_len;
    for (int a = 0; a < kk.n_lags; ++a) {
        const double* m = w.moments + ((int64_t)slot * 3 + kk.source) * S;
        const double* v = kk.table + (int64_t)a * L2 + i + S - 1;
        int j = lane;
        for (; j + 96 < S; j += 128) {
            p0 = fma(__ldg(m + j), __ldg(v - j), p0);
            p1 = fma(__ldg(m + j + 32), __ldg(v - j - 32), p1);
            p2 = fma(__ldg(m + j + 64), __ldg(v - j - 64), p2);
            p3 = fma(__ldg(m + j + 96), __ldg(v - j - 96), p3);
        }
        for (; j < S; j += 32) p0 = fma(__ldg(m + j), __ldg(v - j), p0);
        slot = slot == 0 ? w.ring_len - 1 : slot - 1;
    }
    double part = (p0 + p1) + (p2 + p3);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) {
        const double r = mul(kk.factor, part);
        if (w.out_dtype == PHK_F64)
            reinterpret_cast<double*>(kk.out)[i] = r;
        else
            reinterpret_cast<float*>(kk.out)[i] = (float)r;
    }
}

// Single-bunch numpy path, little work: one CTA of kDirectWarps warps per (kick, target
// slice); warp w takes the stored turns w, w + kDirectWarps, ...; the warps'
// partial sums are added in a fixed order.  (One warp per output leaves
// too few warps on GB300 to cover the load latency of a 50-turn history.)
constexpr int kDirectWarps = 8;
__global__ void __launch_bounds__(kDirectWarps * 32)
wake_direct_kernel(const __grid_constant__ phk_wake_set w) {
    __shared__ double part_w[kDirectWarps];
    const int S = w.n_slices;
    const int k = blockIdx.x / S;
    const int i = blockIdx.x - k * S;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (k >= w.n_kicks) return;
    const phk_wake_kick& kk = w.kick[k];
    if (kk.dense) return;
    const int L2 = 2 * S - 1;
    double p0 = 0.0, p1 = 0.0, p2 = 0.0, p3 = 0.0;
    for (int a = warp; a < kk.n_lags; a += kDirectWarps) {
        const int slot = ((w.head - a) % w.ring_len + w.ring_len) % w.ring_len;
        const double* m = w.moments + ((int64_t)slot * 3 + kk.source) * S;
        const double* v = kk.table + (int64_t)a * L2 + i + S - 1;
        int j = lane;
        for (; j + 96 < S; j += 128) {
            p0 = fma(__ldg(m + j), __ldg(v - j), p0);
            p1 = fma(__ldg(m + j + 32), __ldg(v - j - 32), p1);
            p2 = fma(__ldg(m + j + 64), __ldg(v - j - 64), p2);
            p3 = fma(__ldg(m + j + 96), __ldg(v - j - 96), p3);
        }
        for (; j < S; j += 32) p0 = fma(__ldg(m + j), __ldg(v - j), p0);
    }
    if (warp < kk.n_lags) {             // warps without a turn add nothing up
        double part = (p0 + p1) + (p2 + p3);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            part += __shfl_xor_sync(0xffffffffu, part, o);
        if (lane == 0) part_w[warp] = part;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const int turns = kk.n_lags < kDirectWarps ? kk.n_lags : kDirectWarps;
        double acc = 0.0;
        if (turns > 0) acc = part_w[0];
        for (int q = 1; q < turns; ++q) acc += part_w[q];
        const double r = mul(kk.factor, acc);
        if (w.out_dtype == PHK_F64)
            reinterpret_cast<double*>(kk.out)[i] = r;
        else
            reinterpret_cast<float*>(kk.out)[i] = (float)r;
    }
}

// Single-bunch numpy path, more work.  S^2 multiply-adds per stored turn
// and kick, 25 million a turn with a 50-turn wake at 500 slices: 49 us of the
// FP64 pipe alone.  As integers they are cheaper: the factors become 54-bit
// fixed-point numbers in two 27-bit limbs, a product is four 32 x 32 + 64 bit
// multiply-adds into 64-bit sums (high, two middle, low), exact over a unit of
// up to 96 source slices, and one conversion and FP64 multiply-add takes a
// unit's sum to the output.  Two 50-turn kicks at 500 slices: 95 -> 28 us
// (the direct kernel below a million multiply-adds), bound by the wide
// multiply-adds; errors against extended precision 2.3e-16 (2.5e-16 before).
// Clusters of 8 would be packed two CTAs to an SM and leave half the SMs idle
// (45 us).
//
// One cluster of kConvCluster CTAs per (kick, block of 32 target slices); its
// warps share the (stored turn, chunk of source slices) units.  A warp loads
// a unit's sources and its window of the table, finds the largest magnitude
// of each (the unit's own scales: each factor is off by at most 2^-54 of the
// largest in the window), converts them into its part of shared memory and
// accumulates one target per lane.  Warps, then CTAs, are added in a fixed
// order.  A unit with a non-finite, subnormal or extreme factor runs in FP64
// (conv_unit_fp64), one whose moments or samples are all zero adds nothing.
//
// A target whose terms are all far below its windows' largest (the head of a
// bunch in a causal wake) would lose relative accuracy.  So every unit also notes
// its error (rms, sqrt(sources) / 2 of the unit that its sum is rounded to) and
// the magnitudes of every eighth source's terms.  An FP64 sum of n terms is off
// by n 2^-53 of their magnitudes at most; a target whose noted errors exceed a
// sixteenth of that is summed again in FP64.  The notes cost 2.5 us of 27.
constexpr int kConvWarps = 16;
constexpr int kConvCluster = 4;
constexpr int kConvTargets = 32;    // per cluster, one per lane
constexpr int kConvSources = 96;    // per unit, at most (27 + 27 + 1 + 7 < 63 bits)
constexpr int kConvWindow = kConvSources + kConvTargets - 1;

// v as two 27-bit limbs of a 54-bit integer, r: mant64 shift
__device__ __forceinline__ int2 conv_limbs(double v, int e_max) {
    const int hi = __double2hiint(v), lo = __double2loint(v);
    const int r = e_max + 10 - biased_exp(hi);       // 10 for the largest
    long long q = (long long)((shr_clamp(mant64(hi, lo), r - 1) + 1) >> 1);
    if (hi < 0) q = -q;
    return make_int2((int)(q & 0x7ffffff), (int)(q >> 27));
}

__device__ __forceinline__ void conv_unit_fp64(const double* m, const double* tab,
                                               int len, int i, int S, double& acc) {
    if (i >= S) return;
    for (int j = 0; j < len; ++j) acc = fma(m[j], tab[i - j], acc);
}

// Errors (squared, they are independent) and terms of integer units, in units of
// 2^e
struct ConvBound {
    int e;
    float error;
    float terms[kConvTargets];
};
__device__ __forceinline__ float exp2_int(int d) {       // 2^d, d <= 0; 0 below 2^-126
    return d < -126 ? 0.0f : __int_as_float((d + 127) << 23);
}

// The sum of n bounds for target t (32 threads of a warp)
__device__ __forceinline__ void add_bounds(const ConvBound* b, int n, int t, ConvBound* sum) {
    int e = b[0].e;
    for (int q = 1; q < n; ++q) e = max(e, b[q].e);
    float error = 0.0f, terms = 0.0f;
    for (int q = 0; q < n; ++q) {
        const float down = exp2_int(max(b[q].e - e, -1000));
        error += b[q].error * down * down;
        terms += b[q].terms[t] * down;
    }
    sum->terms[t] = terms;
    if (t == 0) {
        sum->e = e;
        sum->error = error;
    }
}

__global__ void __cluster_dims__(kConvCluster, 1, 1) __launch_bounds__(kConvWarps * 32)
wake_conv_kernel(const __grid_constant__ phk_wake_set w) {
    namespace cg = cooperative_groups;
    __shared__ int2 s_tab[kConvWarps][kConvWindow + 1];
    __shared__ int2 s_mom[kConvWarps][kConvSources];
    __shared__ double s_acc[kConvWarps][kConvTargets];
    __shared__ double s_sum[kConvTargets];
    __shared__ ConvBound s_bound[kConvWarps];
    __shared__ ConvBound s_all;
    __shared__ unsigned s_again;        // targets to sum in FP64
    cg::cluster_group cl = cg::this_cluster();
    const unsigned rank = cl.block_rank();
    const int S = w.n_slices;
    const int blocks = (S + kConvTargets - 1) / kConvTargets;
    const int job = blockIdx.x / kConvCluster;
    const int k = job / blocks, i0 = (job - k * blocks) * kConvTargets;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const phk_wake_kick& kk = w.kick[k];
    const bool work = k < w.n_kicks && !kk.dense;
    const int L2 = 2 * S - 1;
    // as many sources a unit as leave every warp of the cluster one
    const int most = kk.n_lags * S / (kConvWarps * kConvCluster);
    const int per = most < 16 ? 16 : (most > kConvSources ? kConvSources : most);
    const int chunks = (S + per - 1) / per;
    const int units = work ? kk.n_lags * chunks : 0;
    double acc = 0.0;
    int be = -(1 << 20);                 // this warp's ConvBound
    float error = 0.0f, terms = 0.0f;
    for (int u = warp * kConvCluster + rank; u < units; u += kConvWarps * kConvCluster) {
        const int a = u / chunks, j0 = (u - a * chunks) * per;
        const int len = min(per, S - j0);
        if (len <= 0) continue;
        const int slot = ((w.head - a) % w.ring_len + w.ring_len) % w.ring_len;
        const double* m = w.moments + ((int64_t)slot * 3 + kk.source) * S + j0;
        // target i, source j0 + j: table entry i + S - 1 - j0 - j; window
        // entry t holds table entry base + t
        const double* row = kk.table + (int64_t)a * L2;
        const int base = i0 + S - j0 - len;
        const int n_tab = min(len + kConvTargets - 1, L2 - base);
        constexpr int NT = (kConvWindow + 31) / 32, NM = kConvSources / 32;
        double tv[NT], mv[NM];
#pragma unroll
        for (int q = 0; q < NT; ++q) {
            const int t = lane + 32 * q;
            tv[q] = t < n_tab ? __ldg(row + base + t) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < NM; ++q) {
            const int j = lane + 32 * q;
            mv[q] = j < len ? __ldg(m + j) : 0.0;
        }
        // the low word counts for subnormals alone
        unsigned bt = 0u, bm = 0u;
#pragma unroll
        for (int q = 0; q < NT; ++q)
            bt = max(bt, ((unsigned)__double2hiint(tv[q]) & 0x7fffffffu) |
                             (__double2loint(tv[q]) != 0 ? 1u : 0u));
#pragma unroll
        for (int q = 0; q < NM; ++q)
            bm = max(bm, ((unsigned)__double2hiint(mv[q]) & 0x7fffffffu) |
                             (__double2loint(mv[q]) != 0 ? 1u : 0u));
        bt = __reduce_max_sync(0xffffffffu, bt);
        bm = __reduce_max_sync(0xffffffffu, bm);
        if ((bt == 0u || bm == 0u) && max(bt, bm) < 0x7ff00000u) continue;   // zeros
        const int et = (int)(bt >> 20), em = (int)(bm >> 20);
        const bool normal = et >= 100 && et < 2000 && em >= 100 && em < 2000 &&
                            et + em > 1100 && et + em < 3100;
        if (!normal) {
            conv_unit_fp64(m, row + S - 1 - j0, len, i0 + lane, S, acc);
            continue;
        }
        __syncwarp();                  // the previous unit's limbs are read
#pragma unroll
        for (int q = 0; q < NT; ++q)
            if (lane + 32 * q < kConvWindow)
                s_tab[warp][lane + 32 * q] = conv_limbs(tv[q], et);
#pragma unroll
        for (int q = 0; q < NM; ++q) s_mom[warp][lane + 32 * q] = conv_limbs(mv[q], em);
        __syncwarp();
        long long hh = 0, mid = 0, mil = 0, ll = 0, mag = 0;
        const int2* tp = &s_tab[warp][lane + len - 1];
        const int2* mp = s_mom[warp];
#pragma unroll 8
        for (int j = 0; j < len; ++j) {
            const int2 f = mp[j], t = tp[-j];
            hh += (long long)f.y * t.y;
            mid += (long long)f.y * t.x;
            mil += (long long)f.x * t.y;
            ll += (long long)f.x * t.x;
            if (j % 8 == 0) mag += (long long)abs(f.y) * abs(t.y);
        }
        // unit: 2^(et + em - 2099), a product of high limbs is twice that
        if (et + em > be) {
            const float down = exp2_int(be - (et + em));
            error *= down * down;
            terms *= down;
            be = et + em;
        }
        const float here = exp2_int(et + em - be);
        error += here * here * 0.25f * (float)len;
        terms += here * 2.0f * (float)mag;
        // sum = hh 2^54 + mid 2^27 + ll in units of 2^(et + em - 2152); in
        // units of 2^53 of these it fits 63 bits: one rounding
        const double unit = __hiloint2double((et + em - 1076) << 20, 0);
        acc = fma((double)((hh << 1) + ((mid + mil + (ll >> 27)) >> 26)), unit, acc);
    }
    s_acc[warp][lane] = acc;
    s_bound[warp].terms[lane] = terms;
    if (lane == 0) {
        s_bound[warp].e = be;
        s_bound[warp].error = error;
    }
    __syncthreads();
    if (threadIdx.x < kConvTargets) {
        double sum = s_acc[0][threadIdx.x];
        for (int q = 1; q < kConvWarps; ++q) sum += s_acc[q][threadIdx.x];
        s_sum[threadIdx.x] = sum;
        add_bounds(s_bound, kConvWarps, threadIdx.x, &s_all);
    }
    cl.sync();
    // ---- every CTA finds the targets to sum again, rank 0 stores the others
    if (work && threadIdx.x < kConvTargets) {
        __shared__ ConvBound s_each[kConvCluster], s_total;
        for (int r = 0; r < kConvCluster; ++r) {
            const ConvBound* o = cl.map_shared_rank(&s_all, r);
            s_each[r].terms[lane] = o->terms[lane];
            if (lane == 0) {
                s_each[r].e = o->e;
                s_each[r].error = o->error;
            }
        }
        __syncwarp();
        add_bounds(s_each, kConvCluster, lane, &s_total);
        __syncwarp();
        const int i = i0 + lane;
        const bool again = sqrtf(s_total.error) >
                               s_total.terms[lane] * 0x1p-57f * (float)(kk.n_lags * S) &&
                           i < S;
        const unsigned mask = __ballot_sync(0xffffffffu, again);
        if (lane == 0) s_again = mask;
        if (rank == 0 && i < S && !again) {
            double sum = s_sum[lane];
            for (int r = 1; r < kConvCluster; ++r) sum += cl.map_shared_rank(s_sum, r)[lane];
            const double r = mul(kk.factor, sum);
            if (w.out_dtype == PHK_F64)
                reinterpret_cast<double*>(kk.out)[i] = r;
            else
                reinterpret_cast<float*>(kk.out)[i] = (float)r;
        }
    }
    __syncthreads();
    // ---- in FP64: this CTA's share of these targets, side by side, the warps
    // divided among them
    unsigned mine = work ? s_again & (0x11111111u << rank) : 0u;
    if (mine) {
        const int count = __popc(mine);
        const int per_target = kConvWarps >> (count > 4 ? 3 : count > 2 ? 2 : count - 1);
        const int which = warp / per_target, part = warp % per_target;
        for (int n = 0; n < which; ++n) mine &= mine - 1u;
        const int i = i0 + __ffs(mine) - 1;
        double p[4] = {0.0, 0.0, 0.0, 0.0};
        // terms (turn a, source j) in the order of the tables, four loads in flight
        int a = 0, j = 32 * part + lane, slot = w.head % w.ring_len;
        const int turns = which < count ? kk.n_lags : 0, step = 32 * per_target;
        while (a < turns)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                for (; j >= S && a < turns; j -= S, ++a)
                    slot = slot == 0 ? w.ring_len - 1 : slot - 1;
                if (a < turns)
                    p[u] = fma(__ldg(w.moments + ((int64_t)slot * 3 + kk.source) * S + j),
                               __ldg(kk.table + (int64_t)a * L2 + i + S - 1 - j), p[u]);
                j += step;
            }
        double t = (p[0] + p[1]) + (p[2] + p[3]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) s_acc[warp][0] = t;
        __syncthreads();
        if (lane == 0 && part == 0 && which < count) {
            for (int q = 1; q < per_target; ++q) t += s_acc[warp + q][0];
            const double r = mul(kk.factor, t);
            if (w.out_dtype == PHK_F64)
                reinterpret_cast<double*>(kk.out)[i] = r;
            else
                reinterpret_cast<float*>(kk.out)[i] = (float)r;
        }
    }
    cl.sync();                         // sums stay until rank 0 has read them
}

int launch_wake(const phk_wake_set* w, cudaStream_t st) {
    bool any_dense = false, any_conv = false;
    for (int k = 0; k < w->n_kicks; ++k) {
        if (w->kick[k].dense) any_dense = true; else any_conv = true;
    }
    const int S = w->n_slices;
    if (any_conv)
    {
        // multiply-adds of the launch: below a million, the direct kernel's
        // short chains win (50 slices, one turn: 4.4 against 6.4 us; 200
        // slices: 5.6 / 6.4), above, the FP64 work does (1000 slices, 10
        // turns: 66 / 21 us)
        int64_t macs = 0;
        for (int k = 0; k < w->n_kicks; ++k)
            if (!w->kick[k].dense) macs += (int64_t)w->kick[k].n_lags * S * S;
        if (macs < (1 << 20))
            wake_direct_kernel<<<w->n_kicks * S, kDirectWarps * 32, 0, st>>>(*w);
        else
            wake_conv_kernel<<<w->n_kicks * ((S + kConvTargets - 1) / kConvTargets) *
                                   kConvCluster, kConvWarps * 32, 0, st>>>(*w);
    }
    if (any_dense) launch_wake_dense(w, st);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return set_error(PHK_ECUDA, "phk_wake launch: %s", cudaGetErrorString(e));
    count_launches((int)any_conv + (int)any_dense);
    return PHK_OK;
}

// ===================================================================
// batched form: dispatch, merge and wake
// ===================================================================

int launch_track_batch(const phk_batch* bt, const phk_coords* c,
                       const phk_kick_set* pk, const phk_accum* acc,
                       cudaStream_t st) {
    int ld = 0, stm = 0;
    for (int i = 0; i < bt->n_bunches; ++i) {
        int l, s;
        track_masks(bt->programs_host + i, pk, acc, &l, &s);
        ld |= l;
        stm |= s;
    }
    if (c->dtype == PHK_F64) return launch_batch_f64(bt, c, pk, acc, ld, stm, st);
    return launch_batch_f32(bt, c, pk, acc, ld, stm, st);
}

int batch_max_grid(int32_t dtype, int32_t threads, int32_t S, int32_t nk) {
    // phk_track_batch refuses kick tables beyond 48 KB: they do not narrow the
    // grid of the turns without kicks
    const int most = 48 * 1024 / (S * (dtype == PHK_F64 ? 8 : 4));
    if (nk > most) nk = most;
    int nh = 0;
    int per_sm = 0;
    if (dtype == PHK_F64)
        per_sm = batch_per_sm_f64(
            threads, batch_smem<double>(S, nk > 0 ? S : 0, nk, threads, &nh));
    else
        per_sm = batch_per_sm_f32(
            threads, batch_smem<float>(S, nk > 0 ? S : 0, nk, threads, &nh));
    return per_sm * device_info().sm_count;
}

// LANES lanes per (bunch, slice).  Bound by FP64 (about 19 cycles per warp
// instruction and SM): with a warp per slice, its 15 shuffled additions, two
// divisions and conversions were 256000 warp instructions at 64 bunches of
// 100 slices; four lanes share them among eight slices (25 to 9.4 us).
template <int LANES>
__global__ void batch_finalize_kernel(const double* __restrict__ P, int S,
                                      int G, int nb,
                                      const int32_t* __restrict__ bcols,
                                      int32_t* counts, double* mean_x,
                                      double* mean_y, double* moments,
                                      int64_t mstride, int32_t* status) {
    const int64_t group = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / LANES;
    const int lane = threadIdx.x & (LANES - 1);
    const bool on = group < (int64_t)nb * S;     // the warp's shuffles need all
    const int bunch = on ? (int)(group / S) : 0;
    const int s = on ? (int)(group - (int64_t)bunch * S) : 0;
    int g0 = bcols[bunch], g1 = bcols[bunch + 1];
    if (g0 < 0 || g1 > G || g0 > g1) {
        if (lane == 0 && status) atomicMax(status, PHK_DEV_BAD_TABLE);
        g0 = g1 = 0;
    }
    const int64_t o = (int64_t)bunch * S;
    merge_slice<LANES>(P, S, G, s, g0, g1, counts && on ? counts + o : nullptr,
                       mean_x && on ? mean_x + o : nullptr,
                       mean_y && on ? mean_y + o : nullptr,
                       moments && on ? moments + bunch * mstride : nullptr, lane);
}

int launch_batch_finalize(const phk_accum* acc, int nb, const int32_t* bcols,
                          int32_t* counts, double* mean_x, double* mean_y,
                          double* moments, int64_t mstride, int32_t* status,
                          cudaStream_t st) {
    const int S = acc->slicer.n_slices;
    // four lanes while a bunch has at most 64 columns on average (up to 16
    // terms a lane); a warp where bunches span more of the grid
    const int lanes = acc->grid <= 64 * (int64_t)nb ? 4 : 32;
    const int threads = 128;
    const int64_t blocks = ((int64_t)nb * S * lanes + threads - 1) / threads;
    auto kern = lanes == 4 ? batch_finalize_kernel<4> : batch_finalize_kernel<32>;
    kern<<<(unsigned)blocks, threads, 0, st>>>(acc->partials, S, acc->grid, nb, bcols,
                                               counts, mean_x, mean_y, moments,
                                               mstride, status);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return set_error(PHK_ECUDA, "phk_batch_finalize launch: %s",
                         cudaGetErrorString(e));
    count_launches(1);
    return PHK_OK;
}

// The sum of one lane's target over the sources [j0, j1) of every stored turn, in
// SETS x 4 chains.  The sample of source j: v[j dj], of the next turn `row` on.
template <int SETS>
__device__ __forceinline__ double target_sum(const phk_wake_set& w, const phk_wake_kick& kk,
                                             const double* v, int64_t row, int64_t dj,
                                             int j0, int j1) {
    double p[SETS][4] = {};
    int slot = (w.head % w.ring_len + w.ring_len) % w.ring_len;
    for (int a = 0; a < kk.n_lags; ++a, v += row) {
        const double* m = w.moments + ((int64_t)slot * 3 + kk.source) * w.n_slices;
        int j = j0;
        auto four = [&](double (&q)[4]) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                q[u] = fma(__ldg(m + j + u), __ldg(v + (j + u) * dj), q[u]);
            j += 4;
        };
        while (j + 4 * SETS - 1 < j1)
#pragma unroll
            for (int t = 0; t < SETS; ++t) four(p[t]);
#pragma unroll
        for (int t = 1; t < SETS; ++t)
            if (j + 3 < j1) four(p[t]);
        for (; j < j1; ++j) p[0][0] = fma(__ldg(m + j), __ldg(v + j * dj), p[0][0]);
        slot = slot == 0 ? w.ring_len - 1 : slot - 1;
    }
    double sum = 0.0;
#pragma unroll
    for (int t = 0; t < SETS; ++t) {
        const double q = (p[t][0] + p[t][1]) + (p[t][2] + p[t][3]);
        sum = t ? sum + q : q;
    }
    return sum;
}

// One CTA per (bunch, kick, 32 target slices): lanes are targets, the warps
// split the sources of every stored turn, four sums in flight each (16 above 512
// terms per target, so that the chains stay short); fixed order.  Bound by FP64:
// a warp per target spent 9 of its 13 additions on adding its lanes up (64
// bunches, 2 kicks, 100 slices: 15.5 us, now 7.1; 500 slices 145 / 63; 100 slices
// of six turns 40 / 27).
constexpr int kBatchWarps = 8;
constexpr int kFewTerms = 128;

__global__ void __launch_bounds__(kBatchWarps * 32)
batch_wake_kernel(const phk_wake_set* __restrict__ sets, int nb, int S, int nk) {
    __shared__ double part[kBatchWarps][32];
    const int blocks = (S + 31) / 32;
    const int bunch = blockIdx.x / (nk * blocks);
    const int r = blockIdx.x - bunch * nk * blocks;
    const int k = r / blocks, i0 = (r - k * blocks) * 32;
    const phk_wake_set& w = sets[bunch];
    if (w.n_slices != S || w.n_kicks > nk || w.n_kicks < 0 ||
        w.ring_len < 1 || w.head < 0 || w.head >= w.ring_len)
        return;
    if (k >= w.n_kicks) return;
    const phk_wake_kick& kk = w.kick[k];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t n_terms = (int64_t)kk.n_lags * S;
    if (gridDim.y > 1) {        // few bunches, see launch_wake_batch
        if (!kk.dense && n_terms > kFewTerms) {
            const int i = i0 + blockIdx.y * kBatchWarps + warp;
            if (i < S) wake_conv_one(w, k, i, lane);
            return;
        }
        if (blockIdx.y) return;
    }
    const int i = i0 + lane < S ? i0 + lane : S - 1;
    const int j0 = S * warp / kBatchWarps, j1 = S * (warp + 1) / kBatchWarps;
    // numpy path: table[i + S - 1 - j], dot path [j][i]
    const int64_t row = kk.dense ? (int64_t)S * S : 2 * S - 1;
    const int64_t dj = kk.dense ? S : -1;
    const double* v = kk.table + i + (kk.dense ? 0 : S - 1);
    part[warp][lane] = n_terms <= 512 ? target_sum<1>(w, kk, v, row, dj, j0, j1)
                                      : target_sum<4>(w, kk, v, row, dj, j0, j1);
    __syncthreads();
    if (warp != 0 || i0 + lane >= S) return;
    double t[kBatchWarps];
#pragma unroll
    for (int q = 0; q < kBatchWarps; ++q) t[q] = part[q][lane];
#pragma unroll
    for (int d = kBatchWarps / 2; d > 0; d >>= 1)
#pragma unroll
        for (int q = 0; q < d; ++q) t[q] = add(t[q], t[q + d]);
    const double res = mul(kk.factor, t[0]);
    if (w.out_dtype == PHK_F64)
        reinterpret_cast<double*>(kk.out)[i] = res;
    else
        reinterpret_cast<float*>(kk.out)[i] = (float)res;
}

int launch_wake_batch(const phk_wake_set* sets, int nb, int S, int nk,
                      cudaStream_t st) {
    const int64_t blocks = (int64_t)nb * nk * ((S + 31) / 32);
    // Where the blocks leave half of the SMs idle, four CTAs share a block's
    // targets, one to a warp, from kFewTerms terms on (2 bunches, 200 slices of 50 turns:
    // 147 us on one CTA, now 47; 1 bunch, 500 slices of one turn 7.3 / 4.9; 100
    // slices are better left together, 3.3 / 3.5).
    const bool few = 2 * blocks <= device_info().sm_count;
    batch_wake_kernel<<<dim3((unsigned)blocks, few ? 32 / kBatchWarps : 1), kBatchWarps * 32,
                        0, st>>>(sets, nb, S, nk);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return set_error(PHK_ECUDA, "phk_wake_batch launch: %s",
                         cudaGetErrorString(e));
    count_launches(1);
    return PHK_OK;
}

}  // namespace phk
