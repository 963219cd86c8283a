// The plain form's fused pass: pending kicks, element program, slicing, one
// read and one write of the coordinates.  Included by phk_track_f64.cu.
//
// GB300 starts an FP64 instruction of a warp every 16 cycles per SM, so this
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
// flag bytes [Sa], accumulation edges [Sa + 1] (keys), pending-kick edges
// [Sp + 1] (keys; the same table with `share`), kick tables [n_tables][Sp],
// the quarter wave (`sine`)
struct Track64Smem {
    size_t words, flags, eacc, epk, ktab, sine, bytes;
};
__host__ __device__ inline Track64Smem track64_smem(int Sa, int Sp, int n_tables,
                                                    bool share, bool sine) {
    Track64Smem m;
    size_t b = 0;
    m.words = b; b = align16(b + (size_t)4 * kFix64Words * Sa);
    m.flags = b; b = align16(b + (size_t)4 * ((Sa + 3) / 4));
    m.eacc = b; b = align16(b + (size_t)8 * (Sa > 0 ? Sa + 1 : 0));
    m.epk = share ? m.eacc : b;
    if (!share) b = align16(b + (size_t)8 * (Sp > 0 ? Sp + 1 : 0));
    m.ktab = b; b = align16(b + (size_t)8 * n_tables * Sp);
    m.sine = b; b += sine ? kSineBytes : 0;
    m.bytes = b;
    return m;
}

// FixHist64: carries the digits of this CTA into the column's 64-bit words
// (counts of 2^48 units), leaving 16 bits in the lower three (all threads,
// between two barriers).
__device__ __forceinline__ void fix64_carry(const FixHist64& f, int S,
                                            long long* column, int64_t G,
                                            int tid, int nthreads) {
    for (int s = tid; s < S; s += nthreads) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            unsigned* d = reinterpret_cast<unsigned*>(f.w) + s * kFix64Words +
                          1 + 4 * q;
            long long c = 0;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                c += d[i];
                d[i] = (unsigned)c & 0xffffu;
                c >>= 16;
            }
            c += (int)d[3];
            d[3] = 0u;
            if (c != 0)
                atomicAdd(reinterpret_cast<unsigned long long*>(
                              column + ((int64_t)(q + 1) * S + s) * G),
                          (unsigned long long)c);
        }
    }
}

// Three CTAs per SM (80 registers): the FP64 pipe and the integer pipes are
// each about half busy, and the more warps, the better their phases overlap
// (two / three / four CTAs at 1e7 macroparticles with RF and a 50-turn wake:
// 406 / 371 / 358 us a turn; with detuning at 1e6: 107 / 92 / 96 us).
template <int VEC, int SHAPE>
__global__ void __launch_bounds__(kTrackThreads, 3)
track64_kernel(const __grid_constant__ phk_program prog,
               const __grid_constant__ phk_kick_set pk,
               const __grid_constant__ phk_accum acc,
               const __grid_constant__ Track64Args ka) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char smem[];
    // the sums' unit: smallest over the warps of their largest |x|, |y|
    // (high words)
    __shared__ unsigned s_typ[2];
    __shared__ int s_marked;        // FixHist64::any
    constexpr int TILE = kTrackThreads * VEC;
    const TrackArgs& a = ka.t;
    const int Sa = a.has_acc ? acc.slicer.n_slices : 0;
    const int Sp = a.has_pk ? pk.slicer.n_slices : 0;
    const Track64Smem lay = track64_smem(Sa, Sp, a.n_tables, ka.share_edges, ka.sine);
    int* words = reinterpret_cast<int*>(smem + lay.words);
    unsigned* flags = reinterpret_cast<unsigned*>(smem + lay.flags);
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

    if (tid == 0) {
        s_typ[0] = s_typ[1] = ~0u;
        s_marked = 0;
    }
    if (a.has_acc) {
        const double* e = reinterpret_cast<const double*>(acc.slicer.edges);
        for (int i = tid; i <= Sa; i += kTrackThreads) stage_edge<double>(eacc, i, e[i]);
        for (int i = tid; i < kFix64Words * Sa; i += kTrackThreads) words[i] = 0;
        for (int i = tid; i < (Sa + 3) / 4; i += kTrackThreads) flags[i] = 0u;
    }
    if (a.has_pk)
        stage_pending<double>(pk, a, epk, ktab, tid, kTrackThreads, ka.share_edges);
    if (ka.sine) stage_sine(sine, tid, kTrackThreads);
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
    long long* PL = reinterpret_cast<long long*>(P);

    if (a.has_acc) {
        // ---- the cluster's unit, from the finite |x|, |y| of the inputs of
        // every member's first tile (the maps change them by factors of
        // order one; much larger values mark their slice)
        unsigned m[2] = {0u, 0u};
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {      // zeros past the end
                const unsigned b =
                    (unsigned)__double2hiint(t.c[q ? PHK_Y : PHK_X][j]) & 0x7fffffffu;
                if (b < 0x7ff00000u && b > m[q]) m[q] = b;
            }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            m[q] = __reduce_max_sync(0xffffffffu, m[q]);
            if ((tid & 31) == 0 && m[q]) atomicMin(&s_typ[q], m[q]);
        }
        // rank 0 clears its column's 64-bit words before any member adds
        if (crank == 0)
            for (int s = tid; s < 2 * Sa; s += kTrackThreads) PL[(Sa + s) * G] = 0;
        unsigned M[2];
        if (clustered) {
            cg::cluster_group cl = cg::this_cluster();
            cl.sync();                   // orders the clears, see kCluster
            M[0] = M[1] = ~0u;
            for (unsigned r = 0; r < cl.num_blocks(); ++r) {
                const unsigned* sm = cl.map_shared_rank(s_typ, r);
                M[0] = min(M[0], sm[0]);
                M[1] = min(M[1], sm[1]);
            }
        } else {
            __syncthreads();
            M[0] = s_typ[0];
            M[1] = s_typ[1];
        }
        cx.fix.w = words;
        cx.fix.flag = flags;
        cx.fix.any = &s_marked;
        cx.fix.k[0] = fix64_k(M[0]);
        cx.fix.k[1] = fix64_k(M[1]);
    }

    // ---- the tiles: every warp runs whole ones (lanes past the end carry
    // dead particles)
    const int64_t step = (int64_t)gridDim.x * TILE;
    const int64_t rounds = (a.n_tiles + gridDim.x - 1) / gridDim.x;
    for (int64_t it = 0; it < rounds; ++it, i0 += step) {
        run_tile<double, VEC, SHAPE, false, true>(prog, pk, acc, a, cx, t, i0,
                                                  i0 + VEC <= a.n);
        load_tile_plain<double, VEC>(a, cx, t, i0 + step, i0 + step + VEC <= a.n);
        if (a.has_acc && (it + 1) % fix_flush_tiles<TILE>() == 0) {
            __syncthreads();
            fix64_carry(cx.fix, Sa, PL, G, tid, kTrackThreads);
            __syncthreads();
        }
    }
    if (!a.has_acc) return;

    // ---- rank 0 adds its cluster's counters and 64-bit words as integers
    // and writes the partial column in FP64
    unsigned nb = 1;
    int any = 0;
    if (clustered) {
        // adds to the column before the barrier (see kCluster)
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        nb = cl.num_blocks();
        for (unsigned r = 0; r < nb; ++r) any |= *cl.map_shared_rank(&s_marked, r);
        if (crank == 0 && any) {
            // this CTA's flags become the cluster's
            for (int i = tid; i < (Sa + 3) / 4; i += kTrackThreads)
                for (unsigned r = 1; r < nb; ++r)
                    flags[i] |= cl.map_shared_rank(flags, r)[i];
            __syncthreads();
        }
    } else {
        __syncthreads();
        any = s_marked;
    }
    if (crank == 0) {
        for (int s = tid; s < Sa; s += kTrackThreads) {
            long long c = 0, L1[2] = {0, 0}, d2[2] = {0, 0}, d3[2];
            d3[0] = __ldcg(PL + (Sa + s) * G);
            d3[1] = __ldcg(PL + (2 * Sa + s) * G);
            // unrolled over the cluster's members, so that the loads of
            // every member are in flight together
#pragma unroll
            for (int r = 0; r < kCluster; ++r) {
                if (r >= (int)nb) break;
                const int* w = words;
                if (clustered) w = cg::this_cluster().map_shared_rank(words, r);
                w += s * kFix64Words;
                c += w[0];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const unsigned* d = reinterpret_cast<const unsigned*>(w) + 1 + 4 * q;
                    L1[q] += (long long)d[0] + ((long long)d[1] << 16);
                    d2[q] += d[2];
                    d3[q] += (int)d[3];
                }
            }
            P[s * G] = (double)c;
#pragma unroll
            for (int q = 0; q < 2; ++q)
                P[((q + 1) * Sa + s) * G] =
                    any && cx.fix.marked(s, q)
                        ? 0.0 : fix64_value(L1[q], d2[q], d3[q], cx.fix.k[q]);
        }
    }
    if (any) {
        // ---- marked slices: the cluster's CTAs add their particles'
        // updated values in FP64 (each thread reads what it stored)
        __threadfence();
        if (clustered) cg::this_cluster().sync(); else __syncthreads();
        const unsigned* fl = clustered ? cg::this_cluster().map_shared_rank(flags, 0)
                                       : flags;
        i0 = (int64_t)blockIdx.x * TILE + tid * VEC;
        for (int64_t it = 0; it < rounds; ++it, i0 += step) {
            for (int j = 0; j < VEC; ++j) {
                if (i0 + j >= a.n) continue;
                const int s = cx.bac.index(cx.cp[PHK_Z][i0 + j]);
                if (s < 0) continue;
                const unsigned f = fl[s >> 2] >> (8 * (s & 3));
                if (f & 1u) atomicAdd(P + (Sa + s) * G, cx.cp[PHK_X][i0 + j]);
                if (f & 2u) atomicAdd(P + (2 * Sa + s) * G, cx.cp[PHK_Y][i0 + j]);
            }
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
        // 97 us, now 22.8 / 37 / 53; 1e7 with RF and a 50-turn wake 371 us, now
        // 354).  A caller with fewer columns than SMs and tiles (the
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
