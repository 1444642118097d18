// sfg_cluster1d.cu -- whole runs of small 1-D grids in one launch: a single
// thread-block cluster of 16 (or 8) CTAs steps the grid from sfg_advance's
// start to its end time (or step limit) without returning to the host, with
// the state held in the cluster's distributed shared memory.
//
// A 1000-cell tube costs ~30 us per step on the graph path, almost all of it
// launch latency (dt, finalize, three stage launches, commit per step, each a
// few microseconds of work).  Here:
//   * CTA r owns the nodes [r per, (r + 1) per) of every stage buffer (qn,
//     qa, qb and the RK4 accumulator) in its shared memory for the whole run;
//     HBM is touched only to load the state at the start and store it at
//     the end;
//   * a face stencil reads its nodes from the owning CTA's shared memory
//     (its own, or a neighbour's through distributed shared memory);
//   * one lane computes one face; the upper face of a node comes from the
//     next lane by a warp shuffle, so a warp of 32 faces finishes up to 31
//     nodes (the face at a warp boundary is computed by both warps);
//   * one hardware cluster barrier (barrier.cluster: release / acquire at
//     cluster scope) closes each stage; in the last stage of a step every warp
//     also writes its CFL maximum and status bits into its slot of every CTA's
//     shared memory, so every CTA finds the same dt and stop decision in its
//     own after that barrier (slots double-buffered by step parity: a slot is
//     rewritten two steps later, after a barrier that every reader has passed).
// The clock arithmetic is that of finalize_dt_kernel and commit_kernel
// (Time::Driver, SF_time.cpp:42-93), replayed in every thread; the face flux
// and the stage update are the functions the other kernels use (face_flux,
// finish_node).
//
// FP64 (the plain path), transmissive / periodic / frozen ends, all fluxes
// but Lax-Wendroff, up to CL_MAX_NODES nodes (forward Euler: twice as many).
#include <cooperative_groups.h>

#include "sfg_internal.h"
#include "sfg_math.cuh"
#include "sfg_stage.cuh"

namespace cg = cooperative_groups;

namespace sfg {

constexpr int CL_CTAS_MAX = 16;     // the opt-in cluster size
constexpr int CL_WARPS_MAX = 8;
// One pass of eight warps (248 nodes) in each of 16 CTAs.  Beyond it a stage
// takes two passes and the graph path is as fast or faster for one scheme or
// another (us a step at 4100 nodes, cluster / graph: WENO5 17.9 / 20.2, WENO7 27.6 /
// 24.7, TENO5 25.0 / 23.9; at 3968 10.8 / 19.7, 15.5 / 23.8, 14.3 / 23.2).  An Euler
// step is one stage here and a stage, a copy and the launches' latency there:
// two passes win for every scheme (4100: WENO5 7.0 / 12.1, WENO7 10.2 / 13.5;
// 7900: 7.5 / 11.8, 10.5 / 13.1), three do not (8500: WENO7 14.3 / 13.5).
constexpr int CL_MAX_NODES = CL_CTAS_MAX * 31 * CL_WARPS_MAX;

namespace {

// Stage buffers (0 = qn, 1 = qa, 2 = qb, 3 = RK4 accumulator) read and
// written by each stage: the same roles stage_view gives the global arrays.
// Euler alternates qn / qa by step parity instead of copying back.
__device__ __forceinline__ void stage_buffers(int time_id, int stage, int parity, int& in, int& out) {
    if (time_id == T_EULER) {
        in = parity;
        out = 1 - parity;
    } else if (time_id == T_SSPRK3) {
        in = stage;
        out = stage == 2 ? 0 : stage + 1;
    } else {
        in = stage == 3 ? 1 : stage;
        out = stage == 0 ? 1 : stage == 1 ? 2 : stage == 2 ? 1 : 0;
    }
}

__host__ __device__ __forceinline__ int buffer_count(int time_id) {
    return time_id == T_EULER ? 2 : time_id == T_SSPRK3 ? 3 : 4;
}

}  // namespace

// A stage lasts as long as the FP64 chain of one warp of faces (about 1400
// instructions), and two warps on one SM sub-partition take turns on its FP64
// pipe.  So the cluster is as wide as it gets, and a CTA's nodes are dealt
// evenly to four warps, one a sub-partition, when they fit (124 nodes), else to
// eight.  WENO5, us a step, 8 CTAs with full warps of 31 nodes -> 16 CTAs: 1001
// nodes 11.8 -> 10.8, 3000 23.8 -> 12.2.
template <int CTAS, int SCHEME, int FLUX>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(CL_WARPS_MAX * 32)
    cluster1d_kernel(GridView g, ClusterRun run) {
    constexpr int NST = SchemeInfo<SCHEME>::NST;
    constexpr int CL_CTAS = CTAS;
    const int CL_THREADS = blockDim.x, CL_WARPS = blockDim.x >> 5;
    extern __shared__ double cl_smem[];                 // [buffer][5][per]
    __shared__ double slots[2][CL_CTAS * CL_WARPS_MAX];     // CFL maxima of every warp of the cluster, by step parity
    __shared__ unsigned fslots[2][CL_CTAS * CL_WARPS_MAX];  // and their status bits
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = g.n[0];
    const int per = (n + CL_CTAS - 1) / CL_CTAS;
    const int c0 = rank * per, c1 = min(n, c0 + per);        // owned nodes
    const int s0 = max(c0, g.lo[0]), s1 = min(c1, g.hi[0]);  // owned solved nodes (s1 <= s0: none)
    const int time_id = run.sv[0].time_id;
    const int nbuf = buffer_count(time_id);
    const int bstride = 5 * per;                              // doubles per buffer
    const long long vs = g.vs;
    GridView gl = g;                                          // node index = local index, stride per
    gl.vs = per;

    // load the owned chunk of qn into every buffer (unsolved nodes -- frozen
    // ghost values -- stay as loaded in all of them)
    for (int i = c0 + threadIdx.x; i < c1; i += CL_THREADS) {
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            const double x = __ldcg(run.sv[0].qs + v * vs + i);
            for (int b = 0; b < nbuf; ++b) cl_smem[b * bstride + v * per + (i - c0)] = x;
        }
    }

    // largest of the warp's non-negative doubles: high words, then the low words
    // of those that share the largest
    auto warp_largest = [](double x) {
        const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
        const unsigned h = __reduce_max_sync(0xffffffffu, hi);
        const unsigned l = __reduce_max_sync(0xffffffffu, hi == h ? lo : 0u);
        return __hiloint2double((int)h, (int)l);
    };
    // Every warp writes its CFL maximum and status bits into its slot of every
    // CTA (remote stores, one lane a CTA: nothing waits for them but the next
    // cluster barrier, and the reads after it are local).
    auto publish = [&](double sr, unsigned fl, int par) {
        sr = warp_largest(sr);
        fl = __reduce_or_sync(0xffffffffu, fl);
        const int slot = rank * CL_WARPS + warp;
        if (lane < CL_CTAS) {
            cluster.map_shared_rank(&slots[par][0], lane)[slot] = sr;
            cluster.map_shared_rank(&fslots[par][0], lane)[slot] = fl;
        }
        if (lane == 0 && fl) atomicOr(run.flags, fl);
    };
    // after the barrier: the cluster's maximum and status bits (every thread)
    auto gather = [&](int par, double& m, unsigned& f) {
        double x = 0.0;
        unsigned b = 0;
        for (int k = lane; k < CL_CTAS * CL_WARPS; k += 32) {
            x = fmax(x, slots[par][k]);
            b |= fslots[par][k];
        }
        m = warp_largest(x);
        f = __reduce_or_sync(0xffffffffu, b);
    };

    // the CFL maximum of the state the run starts from (slot parity 1; step
    // `it` publishes into parity it & 1)
    {
        double sr = 0.0;
        unsigned fl = 0;
        __syncthreads();
        for (int i = s0 + threadIdx.x; i < s1; i += CL_THREADS) {
            double q[5];
#pragma unroll
            for (int v = 0; v < 5; ++v) q[v] = cl_smem[v * per + (i - c0)];
            const double r = cfl_rate(g, q);
            if (!(r > 0.0) || !isfinite(r)) fl |= FLAG_NONFINITE;  // as dt_kernel
            sr = fmax(sr, r);
        }
        cluster.sync();  // every CTA of the cluster runs before its shared memory is written
        publish(sr, fl, 1);
    }
    cluster.sync();  // the loaded chunks and the first slots are visible cluster-wide
    double sr_max;
    unsigned bad;
    gather(1, sr_max, bad);
    if (bad) sr_max = 0.0;  // an invalid state: no step

    Clock c = *run.clock;
    const long long first = c.steps;
    const double eps = 2.220446049250313e-16;
    bool more = false;  // stopped by the per-launch step bound, not by the run's end
    int parity = 0;     // Euler: buffer holding the current state
    unsigned cores = 0, cut = 0;
    // nodes of a warp per pass: the CTA's dealt evenly, at most 31 (its faces are one more)
    const int share = min(31, max(1, (s1 - s0 + CL_WARPS - 1) / CL_WARPS));
    const int per_pass = share * CL_WARPS;
    const int passes = s1 > s0 ? (s1 - s0 + per_pass - 1) / per_pass : 0;
    for (int it = 0;; ++it) {
        // finalize_dt_kernel
        const double remaining = c.t_end - c.t;
        double scale = fmax(fabs(c.t), fabs(c.t_end));
        scale = scale < 1.0 ? 1.0 : scale;
        if (!(remaining > 64.0 * eps * scale) || c.steps >= c.max_steps || !(sr_max > 0.0)) break;
        if (c.steps - first >= run.launch_steps) {
            more = true;
            break;
        }
        double limit = remaining;
        if (c.write_interval > 0.0 && c.next_out - c.t < limit) limit = c.next_out - c.t;
        if (c.limit < limit) limit = c.limit;
        double dt = __ddiv_rn(g.cfl, sr_max);
        if (c.max_dt < dt) dt = c.max_dt;
        if (limit < dt) dt = limit;

        double sr = 0.0;
        unsigned flags = 0;
        for (int s = 0; s < run.stages; ++s) {
            int bin, bout;
            stage_buffers(time_id, s, parity, bin, bout);
            StageView sv = run.sv[s];
            sv.qout = cl_smem + bout * bstride;
            sv.q0 = cl_smem;                  // qn
            sv.k = cl_smem + 3 * bstride;     // RK4 only
            sv.mode = MODE_FINAL | (s == run.stages - 1 ? MODE_CFL : 0);
            const double* in_local = cl_smem + bin * bstride;
            for (int p = 0; p < passes; ++p) {
                const int f0 = s0 + p * per_pass + warp * share;
                const int f = f0 + lane;  // face f: lower face of node f
                const int fend = min(s1, f0 + share);
                double Fa[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
                if (f <= fend && f0 < s1) {
                    double st[NST][5];
#pragma unroll
                    for (int k = 0; k < NST; ++k) {
                        const int j = map_index(f - NST / 2 + k, n, g.bc_lo[0], g.bc_hi[0]);
                        const double* src = in_local + (j - c0);
                        if ((unsigned)(j - c0) >= (unsigned)(c1 - c0)) {  // a neighbour's node
                            const int owner = j / per;
                            src = cluster.map_shared_rank(in_local, owner) + (j - owner * per);
                        }
#pragma unroll
                        for (int v = 0; v < 5; ++v) st[k][v] = src[v * per];
                    }
                    double F[5];
                    face_flux<0, SCHEME, FLUX>(st, g.gamma, F, flags, cut, 0.0);
#pragma unroll
                    for (int v = 0; v < 5; ++v) Fa[v] = F[v] * g.area[0];
                    if (SCHEME == TENO5 && (lane < share || f == s1)) cores += 10;
                }
                double div[5];
#pragma unroll
                for (int v = 0; v < 5; ++v) div[v] = __shfl_down_sync(0xffffffffu, Fa[v], 1) - Fa[v];
                if (lane < share && f < fend) {
                    const int li = f - c0;
                    double qn[5];
#pragma unroll
                    for (int v = 0; v < 5; ++v) qn[v] = in_local[v * per + li];
                    finish_node(gl, sv, dt, li, qn, div, flags, sr);
                }
            }
            if (s == run.stages - 1) publish(sr, flags, it & 1);
            cluster.sync();  // the stage's output is visible cluster-wide
        }
        if (time_id == T_EULER) parity ^= 1;
        // commit_kernel
        if (rank == 0 && threadIdx.x == 0 && run.dt_log && c.steps - c.log_base < run.dt_cap &&
            c.steps >= c.log_base)
            run.dt_log[c.steps - c.log_base] = dt;
        c.t += dt;
        c.steps += 1;
        double sc = fabs(c.t);
        sc = sc < 1.0 ? 1.0 : sc;
        if (c.write_interval > 0.0 && c.t >= c.next_out - 1.0e-11 * sc) c.next_out += c.write_interval;
        c.limit = __longlong_as_double(0x7FF0000000000000ll);
        c.dt = dt;
        gather(it & 1, sr_max, bad);
        if (bad) break;  // an invalid state stops the run (the same bits in every CTA)
    }
    // the owned solved nodes of the current state back to qn
    const double* cur = cl_smem + (time_id == T_EULER ? parity : 0) * bstride;
    double* qn_out = const_cast<double*>(run.sv[0].qs);
    for (int i = s0 + threadIdx.x; i < s1; i += CL_THREADS) {
#pragma unroll
        for (int v = 0; v < 5; ++v) qn_out[v * vs + i] = cur[v * per + (i - c0)];
    }
    if (rank == 0 && threadIdx.x == 0) {
        c.active = more ? 1 : 0;
        c.dt_ready = 0;
        c.dt_bits = 0x7FEFFFFFFFFFFFFFull;
        *run.clock = c;
    }
    if (run.sv[0].counters && (cores | cut)) {
        atomicAdd(run.sv[0].counters + 0, (unsigned long long)cores);
        atomicAdd(run.sv[0].counters + 1, (unsigned long long)cut);
    }
    cluster.sync();  // no CTA leaves while another may still read its shared memory
}

template <int CTAS, int SCHEME, int FLUX>
static cudaError_t launch_cluster_n(const GridView& g, const ClusterRun& run, cudaStream_t st) {
    const int per = (g.n[0] + CTAS - 1) / CTAS;
    const size_t smem = sizeof(double) * 5 * (size_t)per * buffer_count(run.sv[0].time_id);
    auto kern = cluster1d_kernel<CTAS, SCHEME, FLUX>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if (CTAS > 8) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
    }
    kern<<<CTAS, per <= 124 ? 128 : 256, smem, st>>>(g, run);
    return cudaGetLastError();
}

template <int SCHEME, int FLUX>
static cudaError_t launch_cluster(const GridView& g, const ClusterRun& run, cudaStream_t st) {
    // 16 CTAs from 8 nodes each on: below that there is nothing to spread
    if (g.hi[0] - g.lo[0] >= CL_CTAS_MAX * 8) return launch_cluster_n<CL_CTAS_MAX, SCHEME, FLUX>(g, run, st);
    return launch_cluster_n<8, SCHEME, FLUX>(g, run, st);
}

template <int SCHEME>
static cudaError_t launch_cluster_f(int flux, const GridView& g, const ClusterRun& run, cudaStream_t st) {
    switch (flux) {
    case RUSANOV: return launch_cluster<SCHEME, RUSANOV>(g, run, st);
    case ROE: return launch_cluster<SCHEME, ROE>(g, run, st);
    case STEGER: return launch_cluster<SCHEME, STEGER>(g, run, st);
    case LAXF: return launch_cluster<SCHEME, LAXF>(g, run, st);
    }
    return cudaErrorInvalidValue;
}

// Whether a 1-D grid can run in the cluster kernel.
bool cluster1d_eligible(const GridView& g, int flux, int prec64, int time_id) {
    return g.dim == 1 && prec64 && flux != LAXW && !g.curv && g.hi[0] - g.lo[0] >= 8 &&
           g.n[0] <= (time_id == T_EULER ? 2 : 1) * CL_MAX_NODES;
}

cudaError_t launch_cluster1d(int scheme, int flux, const GridView& g, const ClusterRun& run, cudaStream_t st) {
    switch (scheme) {
    case WENO5: return launch_cluster_f<WENO5>(flux, g, run, st);
    case TENO5: return launch_cluster_f<TENO5>(flux, g, run, st);
    case WENO3: return launch_cluster_f<WENO3>(flux, g, run, st);
    case WENO7: return launch_cluster_f<WENO7>(flux, g, run, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace sfg
