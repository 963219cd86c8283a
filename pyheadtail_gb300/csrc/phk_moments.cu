// Per-slice moments for Slicer.add_statistics (phk_slice_moments,
// phk_slice_moments_all): the sums behind every statistic of a slice, two
// passes over the particles (sums and counts, then centred products).
//
// The values are summed per CTA as exact fixed-point digits in shared memory
// (add_digits; the window of each value from a sample of the CTA's particles)
// and the CTA adds its totals to the caller's FP64 arrays, one global atomic
// per slice and value; what the digits do not hold of a value (32 times the
// typical one, bits below 2^-69 of it, infinite, NaN) is added there on its own.  Before, every
// particle's value was a global FP64 atomic, one launch pair per statistic:
// 22 launches of 220 us for all statistics of 1e6 particles in 200 slices,
// now two.  The integer work and the shared-memory atomics bound it (52
// atomics a particle in the second pass); FP64 instructions are one
// subtraction per coordinate and one product per pair.
#include "phk_track.cuh"

namespace phk {

constexpr int kMomThreads = 512;

// Which products a second pass forms of NQ quantities: the pairs of
// phk_slice_moments (three quantities) and of phk_slice_moments_all (six).
struct Pairs3 {
    static constexpr int NQ = 3, NP = 6;
    static __device__ constexpr int a(int p) { return p == 2 || p == 4 ? 1 : p == 5 ? 2 : 0; }
    static __device__ constexpr int b(int p) { return p == 0 ? 0 : p <= 2 ? 1 : 2; }
};
// (x,x) (y,y) (z,z) (dp,dp)  (x,xp) (y,yp) (z,dp)  (xp,xp) (yp,yp)
// (x,dp) (y,dp)  (xp,dp) (yp,dp)
struct Pairs6 {
    static constexpr int NQ = 6, NP = 13;
    static __device__ constexpr int a(int p) {
        constexpr int v[13] = {0, 2, 4, 5, 0, 2, 4, 1, 3, 0, 2, 1, 3};
        return v[p];
    }
    static __device__ constexpr int b(int p) {
        constexpr int v[13] = {0, 2, 4, 5, 1, 3, 5, 1, 3, 5, 5, 5, 5};
        return v[p];
    }
};

struct MomentArgs {
    const void* z;
    const void* q[6];
    int64_t n;
    const double* means;    // [NQ][S], second pass
    double* sums;           // first pass [NQ][S], second pass [NP][S]
    int32_t* counts;
    int32_t n_q;            // quantities given (the others are skipped)
    int32_t in_smem;        // the digits fit in shared memory
};

// a float as a double, without the conversion unit of the FP64 pipe for
// normal values
__device__ __forceinline__ double widen(float v) {
    const unsigned b = __float_as_uint(v);
    const unsigned e = (b >> 23) & 0xffu;
    if (e == 0u || e == 255u) return (double)v;
    return __hiloint2double((int)((b & 0x80000000u) | ((((b & 0x7fffffffu) >> 3)) +
                                                       (896u << 20))),
                            (int)(b << 29));
}
__device__ __forceinline__ double widen(double v) { return v; }

// words per slice: the count (first pass) and four digits per value, odd so
// that neighbouring slices fall into different banks
template <class PAIRS, int PASS>
__host__ __device__ constexpr int moment_words() {
    return (PASS == 0 ? 1 + 4 * PAIRS::NQ : 4 * PAIRS::NP) | 1;
}

template <typename T, class PAIRS, int PASS>
__global__ void __launch_bounds__(kMomThreads, 1)
moments_kernel(const __grid_constant__ phk_slicer sl, const __grid_constant__ MomentArgs a) {
    constexpr int NQ = PAIRS::NQ, NV = PASS == 0 ? NQ : PAIRS::NP;
    constexpr int W = moment_words<PAIRS, PASS>(), D0 = PASS == 0 ? 1 : 0;
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int WARPS = kMomThreads / 32;
    __shared__ unsigned s_most[NV][WARPS];
    __shared__ int s_base[NV];
    const int S = sl.n_slices, tid = threadIdx.x;
    T* edges = reinterpret_cast<T*>(smem);
    int* words = reinterpret_cast<int*>(smem + align16(sizeof(T) * (S + 1)));
    for (int i = tid; i <= S; i += kMomThreads)
        stage_edge<T>(edges, i, reinterpret_cast<const T*>(sl.edges)[i]);
    if (a.in_smem)
        for (int i = tid; i < W * S; i += kMomThreads) words[i] = 0;
    __syncthreads();
    Bins<T> bins;
    bins.init(edges, S, sl.negate);
    vote_fast_path<T>(bins, true, tid, kMomThreads);
    const T* z = reinterpret_cast<const T*>(a.z);

    // slice (or -1) and values of particle i
    auto values = [&](int64_t i, double (&v)[NV]) {
        const int s = i < a.n ? bins.index(z[i]) : -1;
        double d[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            d[q] = 0.0;
            if (s >= 0 && q < a.n_q) {
                d[q] = widen(reinterpret_cast<const T*>(a.q[q])[i]);
                if (PASS == 1) d[q] -= __ldg(a.means + q * S + s);
            }
        }
#pragma unroll
        for (int p = 0; p < NV; ++p)
            v[p] = PASS == 0 ? d[p < NQ ? p : 0] : d[PAIRS::a(p)] * d[PAIRS::b(p)];
        return s;
    };

    // ---- the window of every value, from a sample; particles outside the
    // cuts count as zeros
    double v[NV];
    int64_t i = own_sample<kMomThreads, kMomThreads>(tid, a.n);
    int s = values(i < 0 ? a.n : i, v);
#pragma unroll
    for (int p = 0; p < NV; ++p) {
        const unsigned m = __reduce_max_sync(0xffffffffu, finite_high(v[p]));
        if ((tid & 31) == 0) s_most[p][tid >> 5] = m;
    }
    __syncthreads();
    for (int p = tid >> 5; p < NV; p += WARPS) {
        const int base = digit_base(typical_of<WARPS>(s_most[p][tid & (WARPS - 1)]), 17);
        if ((tid & 31) == 0) s_base[p] = base;
    }
    __syncthreads();
    int base[NV];
#pragma unroll
    for (int p = 0; p < NV; ++p) base[p] = s_base[p];

    const int64_t step = (int64_t)gridDim.x * kMomThreads;
    const int64_t rounds = (a.n + step - 1) / step;
    i = (int64_t)blockIdx.x * kMomThreads + tid;
    for (int64_t it = 0; it < rounds; ++it, i += step) {
        s = values(i, v);
        if (s >= 0) {
            int* w = words + s * W;
            if (PASS == 0) atomicAdd(a.in_smem ? w : a.counts + s, 1);
#pragma unroll
            for (int p = 0; p < NV; ++p) {
                if (PASS == 0 ? p < a.n_q : PAIRS::b(p) < a.n_q) {
                    double r = v[p];            // what the digits do not hold
                    if (a.in_smem) {
                        int* d = w + D0 + 4 * p;
                        r = add_digits(d, base[p], r) ? 0.0 : add_outside(d, base[p], r);
                    }
                    if (r != 0.0) atomicAdd(a.sums + p * S + s, r);
                }
            }
        }
        if (a.in_smem && (it + 1) % (kDigitValues / kMomThreads) == 0) {
            __syncthreads();
            for (int j = tid; j < S * NV; j += kMomThreads) {
                const int p = j / S, sj = j - p * S;
                const int top = carry_digits(words + sj * W + D0 + 4 * p);
                if (top) atomicAdd(a.sums + j, top_value(top, s_base[p]));
            }
            __syncthreads();
        }
    }
    if (!a.in_smem) return;
    // ---- this CTA's totals to the caller's sums
    __syncthreads();
    for (int j = tid; j < S * NV; j += kMomThreads) {
        const int p = j / S, sj = j - p * S;
        const double t = digits_value(words + sj * W + D0 + 4 * p, s_base[p]);
        if (t != 0.0) atomicAdd(a.sums + j, t);
    }
    if (PASS == 0)
        for (int sj = tid; sj < S; sj += kMomThreads)
            if (words[sj * W]) atomicAdd(a.counts + sj, words[sj * W]);
}

template <typename T, class PAIRS, int PASS>
static int launch_moments_t(const phk_slicer* sl, MomentArgs a, cudaStream_t st) {
    auto kern = moments_kernel<T, PAIRS, PASS>;
    const DeviceInfo& d = device_info();
    const size_t edges = align16(sizeof(T) * (sl->n_slices + 1));
    size_t smem = edges + (size_t)4 * moment_words<PAIRS, PASS>() * sl->n_slices;
    const size_t limit = (size_t)d.max_smem_optin - 1024;
    a.in_smem = smem <= limit;
    if (!a.in_smem) smem = edges;
    // on every launch: the attribute belongs to the current device's kernel
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)limit) != cudaSuccess)
        cudaGetLastError();
    // one CTA per SM: every CTA's total is a rounding of the caller's sum, and two
    // per SM are hardly faster
    int64_t blocks = (a.n + kMomThreads - 1) / kMomThreads;
    if (blocks > d.sm_count) blocks = d.sm_count;
    kern<<<(unsigned)(blocks < 1 ? 1 : blocks), kMomThreads, smem, st>>>(*sl, a);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return set_error(PHK_ECUDA, "phk_slice_moments launch: %s", cudaGetErrorString(e));
    count_launches(1);
    return PHK_OK;
}

template <class PAIRS>
static int launch_moments_pairs(const phk_slicer* sl, int32_t dtype, int32_t pass,
                                const MomentArgs& a, cudaStream_t st) {
    if (dtype == PHK_F64)
        return pass == 0 ? launch_moments_t<double, PAIRS, 0>(sl, a, st)
                         : launch_moments_t<double, PAIRS, 1>(sl, a, st);
    return pass == 0 ? launch_moments_t<float, PAIRS, 0>(sl, a, st)
                     : launch_moments_t<float, PAIRS, 1>(sl, a, st);
}

int launch_moments(const phk_slicer* sl, const void* z, int64_t n,
                   int32_t dtype, const void* const* q, int32_t n_q,
                   int32_t pass, const double* means, double* sums,
                   int32_t* counts, cudaStream_t st) {
    MomentArgs a;
    memset(&a, 0, sizeof(a));
    a.z = z;
    for (int i = 0; i < n_q; ++i) a.q[i] = q[i];
    a.n = n;
    a.means = means;
    // the second pass's sums follow the three of the first
    a.sums = pass == 0 ? sums : sums + (int64_t)3 * sl->n_slices;
    a.counts = counts;
    a.n_q = n_q;
    return launch_moments_pairs<Pairs3>(sl, dtype, pass, a, st);
}

int launch_moments_all(const phk_slicer* sl, const phk_coords* c, int32_t pass,
                       const double* means, double* sums, int32_t* counts,
                       cudaStream_t st) {
    MomentArgs a;
    memset(&a, 0, sizeof(a));
    a.z = c->z;
    a.q[0] = c->x; a.q[1] = c->xp; a.q[2] = c->y;
    a.q[3] = c->yp; a.q[4] = c->z; a.q[5] = c->dp;
    a.n = c->n;
    a.means = means;
    a.sums = sums;
    a.counts = counts;
    a.n_q = 6;
    return launch_moments_pairs<Pairs6>(sl, c->dtype, pass, a, st);
}

}  // namespace phk
