// Dot-product wakes: wake samples of a resistive wall and the matrix-vector
// products of every kick.
//
// Slices that are not a fixed uniform grid (uniform charge, bunch-dependent
// cuts with several turns) need the S x S samples of the wake anew every turn.
#include <cuda_runtime.h>

#include "phk_internal.h"

namespace phk {

namespace {

__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }

}  // namespace

// One thread per sample [j][i], dt = target[i] - source[j]; every operation is
// the reference's, in its order and correctly rounded, so the tables have the
// bits of the host's.  coef[.][1 + sign] are the products in front of the
// square root for the three signs of dt + dt_min (host values); the root is
// shared by all tables of the launch.  Samples ahead of the source
// (sign +1, half of them) are a zero coefficient times the root at -dt_min,
// one value.  Bound by FP64: a division and a square root, about 25 operations
// of 19 cycles per warp (500 slices, four tables: 24 us).  As NumPy on the host,
// with the upload of every table, it was 7 ms a turn.
__global__ void wall_table_kernel(const __grid_constant__ phk_wall_tables w) {
    const int S = w.n_slices;
    const double ahead = __dsqrt_rn(__ddiv_rn(w.num, -w.dt_min));
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
         t < (int64_t)S * S; t += (int64_t)gridDim.x * blockDim.x) {
        const int j = (int)(t / S), i = (int)(t - (int64_t)j * S);
        const double dt = add(w.times[i], -w.times[S + j]);
        const double u = add(dt, w.dt_min);
        double r = ahead;
        if (!(u > 0.0)) {
            const double lim = -w.dt_min;
            r = __dsqrt_rn(__ddiv_rn(w.num, dt > lim ? lim : dt));
        }
        const int s = u > 0.0 ? 2 : u < 0.0 ? 0 : 1;
        for (int k = 0; k < w.n_tables; ++k) {
            const double v = mul(mul(w.table[k].coef[s], r), w.post);
            w.table[k].out[t] = v;
        }
    }
}

int launch_wall_tables(const phk_wall_tables* w, cudaStream_t st) {
    const int64_t n = (int64_t)w->n_slices * w->n_slices;
    const int64_t blocks = (n + 255) / 256;
    wall_table_kernel<<<(unsigned)(blocks < 65536 ? blocks : 65536), 256, 0, st>>>(*w);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return set_error(PHK_ECUDA, "phk_wall_tables launch: %s",
                         cudaGetErrorString(e));
    count_launches(1);
    return PHK_OK;
}

// One CTA per (kick, 16 target slices): its 32 half-warps take the sources in
// turn and read 128-byte rows of the table, the lags one after another; a
// warp then adds the 32 partial sums of each target in a fixed order.
// Latency-bound at these sizes: a thread per target with all S sources in one
// chain kept 16 CTAs busy (500 slices, 4 kicks: 202 us); this split has
// 128 CTAs and chains of S / 32 (8 us), whose rounding errors are smaller.
constexpr int kDenseTargets = 16;
constexpr int kDenseThreads = 512;

__global__ void __launch_bounds__(kDenseThreads)
wake_dense_kernel(const __grid_constant__ phk_wake_set w) {
    __shared__ double part[kDenseTargets][33];
    const int S = w.n_slices;
    const int blocks = (S + kDenseTargets - 1) / kDenseTargets;
    const int k = blockIdx.x / blocks;
    const phk_wake_kick& kk = w.kick[k];
    if (!kk.dense) return;
    const int i0 = (blockIdx.x - k * blocks) * kDenseTargets;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = threadIdx.x & (kDenseTargets - 1);
    const int row = threadIdx.x / kDenseTargets;       // 0 .. 31
    const int i = i0 + t;
    double acc = 0.0;
    if (i < S)
        for (int a = 0; a < kk.n_lags; ++a) {
            const int slot = ((w.head - a) % w.ring_len + w.ring_len) % w.ring_len;
            const double* m = w.moments + ((int64_t)slot * 3 + kk.source) * S;
            const double* W = kk.table + (int64_t)a * S * S + i;
#pragma unroll 4
            for (int j = row; j < S; j += 32)
                acc = fma(m[j], W[(int64_t)j * S], acc);
        }
    part[t][row] = acc;
    __syncthreads();
    double v = part[warp][lane];                       // warp = target
#pragma unroll
    for (int d = 16; d; d >>= 1) v = add(v, __shfl_xor_sync(~0u, v, d));
    if (lane == 0 && i0 + warp < S) {
        const double r = mul(kk.factor, v);
        if (w.out_dtype == PHK_F64)
            reinterpret_cast<double*>(kk.out)[i0 + warp] = r;
        else
            reinterpret_cast<float*>(kk.out)[i0 + warp] = (float)r;
    }
}

void launch_wake_dense(const phk_wake_set* w, cudaStream_t st) {
    const int blocks = (w->n_slices + kDenseTargets - 1) / kDenseTargets;
    wake_dense_kernel<<<w->n_kicks * blocks, kDenseThreads, 0, st>>>(*w);
}

}  // namespace phk
