// The plain form's fused pass: pending kicks, element program, slicing, one
// read and one write of the coordinates.  Included by phk_track_f64.cu.
//
// GB300 starts an FP64 instruction of a warp every 19 cycles per SM, so this
// kernel is built around having few of them: the slice sums (FixHist64) and
// the RF sine (sine_turn) are integer arithmetic, the slice lookup compares
// integer keys.
#pragma once

#include "phk_track.cuh"

namespace phk {

struct Track64Args {
    TrackArgs t;
    OpFix op[PHK_MAX_OPS];
    DetFix det[PHK_MAX_DETUNERS];
    int32_t sine;          // the program needs the quarter wave
    int32_t share_edges;   // the kicks' slicing is the accumulation's
};

// shared memory, every region 16-byte aligned: FixHist64 words [Sa][9] int,
// accumulation edges [Sa + 1] (keys), pending-kick edges [Sp + 1] (keys; the
// same table with `share`), kick tables [n_tables][Sp], the quarter wave
// (`sine`)
struct Track64Smem {
    size_t words, eacc, epk, ktab, sine, bytes;
};
__host__ __device__ inline Track64Smem track64_smem(int Sa, int Sp, int n_tables,
                                                    bool share, bool sine) {
    Track64Smem m;
    size_t b = 0;
    m.words = b; b = align16(b + (size_t)4 * kFix64Words * Sa);
    m.eacc = b; b = align16(b + (size_t)8 * (Sa > 0 ? Sa + 1 : 0));
    m.epk = share ? m.eacc : b;
    if (!share) b = align16(b + (size_t)8 * (Sp > 0 ? Sp + 1 : 0));
    m.ktab = b; b = align16(b + (size_t)8 * n_tables * Sp);
    m.sine = b; b += sine ? kSineBytes : 0;
    m.bytes = b;
    return m;
}

// Carries the digits of the slices with more than `most` values (all threads)
static __device__ __noinline__ void carry_slices(int* words, int S, int most,
                                                 Spill64* sp, const unsigned* typ) {
    __syncthreads();
    for (int s = threadIdx.x; s < S; s += kTrackThreads) {
        int* w = words + s * kFix64Words;
        if (w[0] <= most) continue;
        for (int q = 0; q < 2; ++q) {
            const int top = carry_digits(w + 1 + 4 * q);
            if (top) spill64(sp, q, s, top_value(top, digit_base(typ[q], 18)));
        }
    }
    __syncthreads();
}

// Three CTAs per SM (80 registers): the FP64 pipe is three quarters busy, the
// integer pipes half, and the more warps, the better their phases overlap; at
// four the exact sums spill (three / four CTAs: RF and a 50-turn wake, 3e6
// macroparticles 157 / 161 us a turn; 1e6 detuned 94 / 101; 1e6 linear 60 / 64).
template <int VEC, int SHAPE>
__global__ void __launch_bounds__(kTrackThreads, 3)
track64_kernel(const __grid_constant__ phk_program prog,
               const __grid_constant__ phk_kick_set pk,
               const __grid_constant__ phk_accum acc,
               const __grid_constant__ Track64Args ka) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int WARPS = kTrackThreads / 32;
    __shared__ Seen<WARPS> s_seen;
    __shared__ unsigned s_typ[2];   // typical |x|, |y|
    __shared__ Spill64 s_spill;
    constexpr int TILE = kTrackThreads * VEC;
    const TrackArgs& a = ka.t;
    const int Sa = a.has_acc ? acc.slicer.n_slices : 0;
    const int Sp = a.has_pk ? pk.slicer.n_slices : 0;
    const Track64Smem lay = track64_smem(Sa, Sp, a.n_tables, ka.share_edges, ka.sine);
    int* words = reinterpret_cast<int*>(smem + lay.words);
    double* eacc = reinterpret_cast<double*>(smem + lay.eacc);
    double* epk = reinterpret_cast<double*>(smem + lay.epk);
    double* ktab = reinterpret_cast<double*>(smem + lay.ktab);
    u64* sine = reinterpret_cast<u64*>(smem + lay.sine);
    const int tid = threadIdx.x;

    TrackCtx<double, VEC> cx;
#pragma unroll
    for (int q = 0; q < 6; ++q) cx.cp[q] = reinterpret_cast<double*>(a.c[q]);
    // the first tile is on its way while the CTA stages its tables
    int64_t i0 = (int64_t)blockIdx.x * TILE + tid * VEC;
    Tile<double, VEC> t;
    load_tile_plain<double, VEC>(a, cx, t, i0, i0 + VEC <= a.n);

    // so is a sample of its x and y
    unsigned m_in[2] = {0u, 0u};
    if (a.has_acc) {
        const int64_t i = own_sample<kTrackThreads, TILE>(tid, a.n);
        if (i >= 0) {
            m_in[0] = finite_high(cx.cp[PHK_X][i]);
            m_in[1] = finite_high(cx.cp[PHK_Y][i]);
        }
    }

    if (a.has_acc) {
        const double* e = reinterpret_cast<const double*>(acc.slicer.edges);
        for (int i = tid; i <= Sa; i += kTrackThreads) stage_edge<double>(eacc, i, e[i]);
        for (int i = tid; i < kFix64Words * Sa; i += kTrackThreads) words[i] = 0;
    }
    if (a.has_pk)
        stage_pending<double>(pk, a, epk, ktab, tid, kTrackThreads, ka.share_edges);
    if (ka.sine) stage_sine(sine, tid, kTrackThreads);
    if (a.has_acc) note_seen<WARPS>(s_seen.in, m_in[0], m_in[1]);
    if (tid < 2) s_typ[tid] = 0u;
    __syncthreads();
    if (a.has_pk) cx.bpk.init(epk, Sp, pk.slicer.negate);
    if (a.has_acc) cx.bac.init(eacc, Sa, acc.slicer.negate);
    cx.ktab = ktab;
    cx.aux = Aux64{sine, ka.op, ka.det};

    // partial column of this CTA's cluster
    const bool clustered = a.has_acc && a.cluster > 1;
    const unsigned crank = clustered ? cg::this_cluster().block_rank() : 0u;
    const int column = clustered ? (int)(blockIdx.x / a.cluster) : (int)blockIdx.x;
    const int64_t G = acc.grid;
    double* P = acc.partials + column;

    if (a.has_acc) {
        // rank 0 clears its column's sums before any member adds
        if (crank == 0)
            for (int s = tid; s < 2 * Sa; s += kTrackThreads) P[(Sa + s) * G] = 0.0;
        if (tid == 0) {
            s_spill.sum[0] = P + Sa * G;
            s_spill.sum[1] = P + 2 * Sa * G;
            s_spill.stride = G;
            s_spill.any = 0;
        }
        if (clustered) cg::this_cluster().sync();   // orders the clears, see kCluster
        else __syncthreads();
        cx.fix.w = words;
        cx.fix.sp = &s_spill;
        cx.fix.base[0] = cx.fix.base[1] = kNoBase;
    }

    // ---- the tiles: every warp runs whole ones (lanes past the end carry
    // dead particles)
    constexpr int kTiles = kDigitValues / TILE;
    int until_carry = kTiles;
    bool open = a.has_acc;          // a window is still to be set
    const int64_t step = (int64_t)gridDim.x * TILE;
    const int64_t rounds = (a.n_tiles + gridDim.x - 1) / gridDim.x;
    for (int64_t it = 0; it < rounds; ++it, i0 += step) {
        tile_advance<double, VEC, SHAPE, false>(prog, pk, a, cx, t, i0);
        if (open) {
            unsigned m[2] = {0u, 0u};
#pragma unroll
            for (int j = 0; j < VEC; ++j)
                if (i0 + j < a.n) {
                    m[0] = max(m[0], finite_high(t.c[PHK_X][j]));
                    m[1] = max(m[1], finite_high(t.c[PHK_Y][j]));
                }
            open = find_typical<WARPS>(&s_seen, s_typ, m[0], m[1]);
            cx.fix.base[0] = digit_base(s_typ[0], 18);
            cx.fix.base[1] = digit_base(s_typ[1], 18);
        }
        tile_finish<double, VEC, false, true>(acc, a, cx, t, i0, i0 + VEC <= a.n);
        load_tile_plain<double, VEC>(a, cx, t, i0 + step, i0 + step + VEC <= a.n);
        if (a.has_acc && --until_carry == 0) {
            // before a counter can overflow in the next kTiles tiles
            until_carry = kTiles;
            carry_slices(words, Sa, kDigitValues - kTiles * TILE, &s_spill, s_typ);
        }
    }
    if (!a.has_acc) return;

    // ---- rank 0 writes the partial column: every CTA's exact sums, and what
    // lay outside their windows
    unsigned nb = 1;
    if (clustered) {
        // adds to the column before the barrier (see kCluster)
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        nb = cl.num_blocks();
    } else {
        __syncthreads();
    }
    if (crank == 0) {
        // the column is read only if values lay outside
        const bool outside = clustered || s_spill.any;
        for (int s = tid; s < Sa; s += kTrackThreads) {
            long long c = 0;
            double v[2] = {0.0, 0.0};
            if (outside) {
                v[0] = __ldcg(P + (Sa + s) * G);
                v[1] = __ldcg(P + (2 * Sa + s) * G);
            }
            // unrolled over the cluster's members, so that the loads of
            // every member are in flight together
#pragma unroll
            for (int r = 0; r < kCluster; ++r) {
                if (r >= (int)nb) break;
                const int* w = words;
                const unsigned* typ = s_typ;
                if (clustered) {
                    w = cg::this_cluster().map_shared_rank(words, r);
                    typ = cg::this_cluster().map_shared_rank(s_typ, r);
                }
                w += s * kFix64Words;
                c += w[0];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const double t = digits_value(w + 1 + 4 * q, digit_base(typ[q], 18));
                    // mostly the first: no FP64 instruction
                    v[q] = __double_as_longlong(v[q]) == 0 ? t : add_cold(v[q], t);
                }
            }
            P[s * G] = (double)c;
            P[(Sa + s) * G] = v[0];
            P[(2 * Sa + s) * G] = v[1];
        }
    }
    if (clustered) cg::this_cluster().sync();  // members keep their counters until read
}

// ===================================================================
// launch
// ===================================================================

// Kick tables and shared memory of a launch; thousands of slices leave the
// kick tables in global memory.
static inline size_t track64_plan(const phk_kick_set* pk, const phk_accum* acc,
                                  bool sine, size_t limit, Track64Args* ka) {
    TrackArgs& a = ka->t;
    const int Sa = acc ? acc->slicer.n_slices : 0;
    const int Sp = pk ? pk->slicer.n_slices : 0;
    // a turn's kicks come from the slicing that is about to be repeated: one
    // staged edge table serves both
    ka->share_edges = pk && acc && pk->slicer.edges == acc->slicer.edges &&
                      Sp == Sa && pk->slicer.negate == acc->slicer.negate;
    plan_kick_tables<double>(pk, &a);
    if (!a.kicks_smem) a.n_tables = 0;
    size_t b = track64_smem(Sa, Sp, a.n_tables, ka->share_edges, sine).bytes;
    if (b > limit && a.kicks_smem) {
        a.kicks_smem = a.kick_comb = a.n_tables = 0;
        a.comb_slot[0] = a.comb_slot[1] = a.comb_slot[2] = -1;
        b = track64_smem(Sa, Sp, 0, ka->share_edges, sine).bytes;
    }
    return b;
}

// dynamic shared memory a launch may request; opts in once per
// instantiation and device
template <int VEC, int SHAPE>
static size_t track64_limit() {
    static size_t limit[64] = {0};
    const DeviceInfo& d = device_info();
    const int dev = d.device < 64 ? d.device : 63;
    if (!limit[dev]) {
        auto kern = track64_kernel<VEC, SHAPE>;
        cudaFuncAttributes fa;
        size_t l = (size_t)d.max_smem_optin - 1024;
        if (cudaFuncGetAttributes(&fa, kern) == cudaSuccess)
            l = (size_t)d.max_smem_optin - fa.sharedSizeBytes;
        else
            cudaGetLastError();
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)l) != cudaSuccess)
            cudaGetLastError();
        limit[dev] = l;
    }
    return limit[dev];
}

template <int VEC, int SHAPE>
static int launch_track64_t(const phk_program* prog, const phk_coords* c,
                            const phk_kick_set* pk, const phk_accum* acc,
                            int load_mask, int store_mask, cudaStream_t st) {
    Track64Args ka;
    memset(&ka, 0, sizeof(ka));
    TrackArgs& a = ka.t;
    a.c[0] = c->x; a.c[1] = c->xp; a.c[2] = c->y;
    a.c[3] = c->yp; a.c[4] = c->z; a.c[5] = c->dp;
    a.n = c->n;
    a.has_pk = pk != nullptr;
    a.has_acc = acc != nullptr;
    a.load_mask = load_mask;
    a.store_mask = store_mask;
    a.cluster = 1;
    const int64_t per_tile = (int64_t)kTrackThreads * VEC;
    a.n_tiles = (c->n + per_tile - 1) / per_tile;
    ka.sine = program_has_phase(*prog);
    for (int o = 0; o < prog->n_ops; ++o) op_fix(prog->op[o], ka.op + o);
    for (int d = 0; d < prog->n_det; ++d) det_fix(prog->det[d], ka.det + d);
    const size_t limit = track64_limit<VEC, SHAPE>();
    const size_t smem = track64_plan(pk, acc, ka.sine, limit, &ka);
    if (smem > limit)
        return set_error(PHK_ESIZE, "phk_track: %zu bytes of shared memory "
                         "needed for %d + %d slices", smem,
                         acc ? acc->slicer.n_slices : 0,
                         pk ? pk->slicer.n_slices : 0);
    static phk_kick_set zero_pk;
    static phk_accum zero_acc;
    auto kern = track64_kernel<VEC, SHAPE>;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kTrackThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    if (acc) {
        // One partial column per CTA: folding four CTAs into a column costs two
        // cluster barriers, and only 440 of 456 CTAs found room (a turn with
        // linear maps of 1e5 macroparticles at 50 / 500 / 1000 slices 24.8 / 63 /
        // 97 us against 22.8 / 37 / 53; 1e7 with RF and a 50-turn wake 371 against
        // 354, when this was chosen).  A caller with fewer columns than SMs and tiles (the
        // workspace-free pass) gets clusters of kCluster CTAs per column.
        // Launched as clusters of one too: their CTAs are spread better than
        // those of a plain launch (1e6 with detuning 90.1 / 92.2 us).
        const int64_t sms = device_info().sm_count;
        a.cluster = acc->grid < (a.n_tiles < sms ? a.n_tiles : sms) ? kCluster : 1;
        cfg.gridDim = dim3((unsigned)acc->grid * a.cluster, 1, 1);
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = a.cluster;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
    } else {
        int bps = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, kTrackThreads,
                                                          smem) != cudaSuccess)
            bps = 1;
        int64_t g = (int64_t)device_info().sm_count * (bps < 1 ? 1 : bps);
        if (a.n_tiles < g) g = a.n_tiles;
        cfg.gridDim = dim3((unsigned)(g < 1 ? 1 : g), 1, 1);
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, *prog, pk ? *pk : zero_pk,
                                             acc ? *acc : zero_acc, ka);
    if (e != cudaSuccess)
        return set_error(PHK_ECUDA, "phk_track launch: %s", cudaGetErrorString(e));
    count_launches(1);
    note_track_launch(0, 0, smem);
    return PHK_OK;
}

// CTAs that can be resident at once (clusters of one)
template <int VEC, int SHAPE>
static int track64_ctas(size_t smem) {
    track64_limit<VEC, SHAPE>();
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &n, track64_kernel<VEC, SHAPE>, kTrackThreads, smem) != cudaSuccess ||
        n < 1) {
        cudaGetLastError();
        n = 1;
    }
    return n * device_info().sm_count;
}

}  // namespace phk
