// Many ticks of a small model in one launch.
//
// A tick of a small grid is a chain of latencies: as the three kernels of the
// stream schedule it takes about 9.5 us whatever the grid size, of which the
// grid's memory traffic (populations in L2) is a fraction of a microsecond.
// Here resident CTAs run tick after tick (tick!, src/gpu/fluids.jl:132-226,
// moveParticles!, src/gpu/particles.jl:7-92) with ONE barrier between ticks:
//   bulk CTAs     collide and push their nodes, src -> dst (both in L2).  Pushes
//                 into link slots and wall nodes are left out (pmask, wmask: per
//                 source node, the directions not to push), so that those values
//                 can be written in the same phase: a node next to a wall writes
//                 its own bounce-back (it holds f*_i and rho), and
//   boundary CTA  (the last one, where there is a particle) the particle's link
//                 slots: it re-collides the link nodes from src, forms and stores
//                 the slot values, sums the momentum exchange and decides whether
//                 the particle's geometry stays before it arrives at the barrier;
//                 the rest of the particle update and the slip velocities of the
//                 next tick run behind the barrier.
// Where the geometry changes (one tick in tens), the CTA rebuilds it, the slot
// list and pmask before it arrives, and the others wait.
// The arithmetic of a node, a link slot and a particle, and the order of the
// FP64 sums, are those of k_bulk, k_fixup and k_particles: the populations are
// equal bit for bit.
//
// Measured with a squirmer, per tick, against the stream schedule: 64^2 FP32
// 3.1 us (9.4), 256 x 128 FP64 3.8 (10.2), 201 x 65 with walls 3.6 (10.4),
// 512 x 256 FP32 3.9 (10.0).  The chain that bounds it: barrier and fence 1.0,
// link nodes 0.8, slots and their sums 0.7, the verdict on the geometry 0.4 us.
// (Two barriers per tick, with the slots stored between them over the pushes,
// took 3.4 to 5.6 us for the same grids.)
//
// The barrier is the hardware barrier of one thread-block cluster (up to 16
// CTAs), or for larger grids a counter in global memory (a cooperative launch;
// every wait bounded).  Both cost mostly the same thing, the fence that makes
// the pushes visible (about 1,500 cycles).
#pragma once
#include "fixup.cuh"
#include "particles.cuh"

namespace lbm {

constexpr int kResThreads = 512;      // threads per CTA
constexpr int kResHalf = 256;         // threads per chunk of link entries (= the fix-up's CTA: sums in the same order)
constexpr int kResMaxCluster = 16;
constexpr int kResMaxEntries = 1024;  // link entries of the particle, where their shared memory fits
constexpr size_t kResMaxSmem = 200 * 1024;
constexpr int kResMaxChunks = kResMaxEntries / kFixBlock;
constexpr long long kResSpinLimit = 1LL << 22;  // polls of the grid barrier before it gives up (about a second)

struct ResidentJob {
    StepArgs a[2];          // by tick parity
    ParticleArgs pa;
    unsigned* pmask;        // [N] directions a node does not push: the particle's link slots (zero between launches)
    const unsigned* wmask;  // [N] the same for wall nodes and wall links (static), or null
};

struct ResidentArgs {
    const ResidentJob* job;
    int ticks;
    int max_entries;     // link entries the boundary CTA's shared memory holds
    unsigned* bar;       // grid barrier counter, zero at launch (null: cluster barrier)
    int* err;            // of the grid barrier
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_size() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// The cluster's barrier in two halves; every thread of every CTA takes both.
// The loops before it leave warps diverged, and the compiler does not know
// that inline assembly wants them together: the warp is joined first, and the
// forms without .aligned are used, which count threads however a warp arrives.
__device__ __forceinline__ void cluster_arrive() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_arrive_relaxed() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    __syncwarp();
}

// The barrier between ticks.  arrive(): after a __syncthreads that follows the
// CTA's stores, by every thread; the last warp makes them visible and arrives
// for the CTA.  wait(): by every thread; false when a bounded wait gave up
// (every CTA then leaves at its next wait).
struct ResidentBarrier {
    unsigned* ctr;      // null: cluster barrier
    int* err;
    unsigned target;    // arrivals that complete the current phase
    unsigned ctas;
    __device__ __forceinline__ void arrive() {
        if (ctr) {
            if (threadIdx.x == kResThreads - 32) {
                __threadfence();
                atomicAdd(ctr, 1u);
            }
        } else if (threadIdx.x >= kResThreads - 32) {
            __threadfence();
            cluster_arrive();
        } else {
            cluster_arrive_relaxed();
        }
    }
    __device__ __forceinline__ bool wait() {
        if (!ctr) {
            cluster_wait();
            return true;
        }
        target += ctas;
        __shared__ int s_ok;
        if (threadIdx.x == 0) {
            int ok = 1;
            long long it = 0;
            unsigned v;
            while (true) {
                asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
                if ((int)(v - target) >= 0) break;
                if (++it > kResSpinLimit) {
                    atomicOr(err, kErrSpinTimeout);
                    ok = 0;
                    break;
                }
            }
            s_ok = ok;
        }
        __syncthreads();
        return s_ok != 0;
    }
};

// load_pops through L2: the buffers change roles every tick, so the loads must
// not use the read-only path that plain const __restrict__ loads may take
template <class L, int ST>
__device__ __forceinline__ void load_pops_l2(const StepArgs& a, int cell, typename Store<ST>::R* g) {
    using SS = Store<ST>;
    using T = typename SS::T;
    const T* src = static_cast<const T*>(a.src);
#pragma unroll
    for (int i = 0; i < L::Q; ++i) g[i] = SS::dec(__ldcg(src + i * a.g.N + cell), typename SS::R(1));
}

// One node of the bulk phase (k_bulk), after its populations are loaded: pushes
// except into link slots and wall nodes, and the node's own wall links.
template <class L, int ST, bool TRT, bool WALLS>
__device__ __forceinline__ bool resident_node(const StepArgs& a, const unsigned* pmask, const unsigned* wmask,
                                              int cell, int x, int y, int z, typename Store<ST>::R* g, bool first) {
    using SS = Store<ST>;
    using T = typename SS::T;
    using R = typename SS::R;
    constexpr int Q = L::Q;
    const int nx = a.g.n[0], ny = a.g.n[1], nz = a.g.n[2];
    const long long N = a.g.N;
    T* dst = static_cast<T*>(a.dst);
    unsigned skip = pmask ? __ldcg(pmask + cell) : 0u;
    unsigned wm = 0;
    if (WALLS) {
        wm = wmask[cell];
        if (wm & 1u) {  // a wall node: f = 0, never pushed into; written in both buffers once per launch
            if (first) {
                const T zero = SS::enc(R(-a.rho0), R(a.scale));
#pragma unroll
                for (int i = 0; i < Q; ++i) dst[i * N + cell] = zero;
            }
            return false;
        }
        skip |= wm;
    }
    const R rho = collide_node<L, ST, TRT>(a, cell, true, g);
    const int xs[3] = {x == 0 ? nx - 1 : x - 1, x, x == nx - 1 ? 0 : x + 1};
    const int ys[3] = {y == 0 ? ny - 1 : y - 1, y, y == ny - 1 ? 0 : y + 1};
    const int zs[3] = {z == 0 ? nz - 1 : z - 1, z, z == nz - 1 ? 0 : z + 1};
#pragma unroll
    for (int i = 0; i < Q; ++i)
        if (!(skip >> i & 1u))
            dst[i * N + (xs[L::cx(i) + 1] + nx * (ys[L::cy(i) + 1] + ny * zs[L::cz(i) + 1]))] = SS::enc(g[i], R(1));
    if (WALLS && wm) {
#pragma unroll
        for (int i = 1; i < Q; ++i) {
            if (!(wm >> i & 1u)) continue;  // x + c_i is a wall node: f_j(x) = f*_i(x), j = opp(i)
            const int j = L::opp(i);
            const int t = xs[L::cx(i) + 1] + nx * (ys[L::cy(i) + 1] + ny * zs[L::cz(i) + 1]);
            if (pmask && (__ldcg(pmask + t) >> j & 1u)) continue;  // also the particle's link: the boundary CTA's
            double v = (double)(g[i] * R(a.inv_scale));
            if (a.uw) {  // moving walls (fluids.jl:168-174)
                const double dot = -(L::cx(i) * a.uw[t] + L::cy(i) * a.uw[N + t] +
                                     (L::D == 3 ? L::cz(i) * a.uw[2 * N + t] : 0.0));
                v += 6.0 * (double)rho * dot;
            }
            dst[j * N + cell] = SS::enc((R)v, R(a.scale));
        }
    }
    return bad_density(rho);
}

// nodes first, first + stride, ... of the grid, two at a time: the loads of
// both are in flight together
template <class L, int ST, bool TRT, bool WALLS>
__device__ __forceinline__ void resident_bulk(const StepArgs& a, const unsigned* pmask, const unsigned* wmask,
                                              int first, int stride, int x, int y, int z, bool init) {
    using R = typename Store<ST>::R;
    const int nx = a.g.n[0], ny = a.g.n[1], N = (int)a.g.N;
    bool bad = false;
    for (int cell = first; cell < N; cell += 2 * stride) {
        const int c2 = cell + stride;
        const bool two = c2 < N;
        R g[2][L::Q];
        load_pops_l2<L, ST>(a, cell, g[0]);
        load_pops_l2<L, ST>(a, two ? c2 : cell, g[1]);
        if (cell != first) {
            x = cell % nx;
            y = L::D == 2 ? cell / nx : (cell / nx) % ny;
            z = L::D == 2 ? 0 : cell / (nx * ny);
        }
        bad |= resident_node<L, ST, TRT, WALLS>(a, pmask, wmask, cell, x, y, z, g[0], init);
        if (!two) break;
        x = c2 % nx;
        y = L::D == 2 ? c2 / nx : (c2 / nx) % ny;
        z = L::D == 2 ? 0 : c2 / (nx * ny);
        bad |= resident_node<L, ST, TRT, WALLS>(a, pmask, wmask, c2, x, y, z, g[1], init);
    }
    if (bad) atomicOr(a.err, kErrNumeric);
}

// wmask of every node: bit i where x + c_i is a wall node; all bits at wall nodes
template <class L>
__global__ void k_resident_wmask(const unsigned char* wall, GridDesc g, unsigned* wmask) {
    const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (c >= g.N) return;
    unsigned m = 0;
    if (wall[c]) {
        m = ~0u;
    } else {
        const int nx = g.n[0], ny = g.n[1], nz = g.n[2];
        const int x = (int)(c % nx), y = (int)((c / nx) % ny), z = (int)(c / ((long long)nx * ny));
#pragma unroll
        for (int i = 1; i < L::Q; ++i)
            if (wall[wrap_idx(x + L::cx(i), nx) +
                     (long long)nx * (wrap_idx(y + L::cy(i), ny) + (long long)ny * wrap_idx(z + L::cz(i), nz))])
                m |= 1u << i;
    }
    wmask[c] = m;
}

// shared memory of the boundary CTA, in a fixed layout for `max_entries` entries
template <class L, int ST>
struct ResidentBoundary {
    using R = typename Store<ST>::R;
    static constexpr int Q = L::Q, D = L::D;
    int E;            // max_entries
    double* C;        // [D][3][E] coordinates of x - 1, x, x + 1 per axis
    double* rho;      // [E]
    double* cu;       // [E Q] c_i . slip velocity of the slots' source nodes
    R* g;             // [Q][E] post-collision populations (f/w - rho0)
    int* cell;        // [E]
    int* mask;        // [E]
    unsigned short* list;  // [E Q] (entry << 5) | j, chunk by chunk of kFixBlock entries
    static __host__ __device__ size_t bytes(int E) {
        return (size_t)E * (sizeof(double) * (3 * D + 1 + Q) + sizeof(R) * Q + 2 * sizeof(int) +
                            sizeof(unsigned short) * Q);
    }
    __device__ __forceinline__ ResidentBoundary(unsigned char* p, int e) : E(e) {
        C = reinterpret_cast<double*>(p);
        rho = C + 3 * D * E;
        cu = rho + E;
        g = reinterpret_cast<R*>(cu + Q * E);
        cell = reinterpret_cast<int*>(g + Q * E);
        mask = cell + E;
        list = reinterpret_cast<unsigned short*>(mask + E);
    }
};

// Range of positions of a particle in which its index box (solid_box) and its
// solid nodes are certainly those of the stored intervals.
struct ResidentKeep {
    double lo[3], hi[3];  // per axis
    double d2;            // squared distance from vR (negative: unknown)
};

// by one thread, after the intervals were looked at
template <int D>
__device__ __forceinline__ void resident_keep(const ParticleArgs& a, const ParticleDev& P, ResidentKeep* k) {
    double dmax2 = 0.0;
    bool ok = P.valid && P.slack > 0.0;
    for (int q = 0; q < D; ++q) {
        // solid_box: floor(c - r) - 1 and ceil(c + r) + 1 with c = (R - x0)/dx, clipped
        // to the grid; inside (lo + 1, lo + 2) and (hi - 2, hi - 1) by a margin that
        // covers the rounding of c, the box stays (a clipped side is left to the full update)
        const int n = a.g.n[q];
        const double rr = P.radius / a.dx, eps = 1e-9 * (fabs(P.vR[q] - a.x0[q]) / a.dx + rr + 1.0);
        ok = ok && P.slo[q] > 0 && P.shi[q] < n - 1 && P.slo[q] <= P.shi[q];
        const double l = fmax(P.slo[q] + 1 + rr, P.shi[q] - 2 - rr) + eps, h = fmin(P.slo[q] + 2 + rr, P.shi[q] - 1 - rr) - eps;
        k->lo[q] = a.x0[q] + a.dx * l;
        k->hi[q] = a.x0[q] + a.dx * h;
        if (ok) {
            const double e0 = fabs(a.coord[q][P.slo[q]] - P.vR[q]), e1 = fabs(a.coord[q][P.shi[q]] - P.vR[q]);
            dmax2 += e0 > e1 ? e0 * e0 : e1 * e1;
        }
    }
    // the displacement d that particles_core accepts: 2 dmax d + d^2 < slack less the rounding of the nodes' d^2
    const double s = P.slack - 2e-9 * (P.r2 + dmax2);
    if (!ok || !(s > 0.0)) {
        k->d2 = -1.0;
        return;
    }
    const double d = s / (sqrt(dmax2) + sqrt(dmax2 + s));
    k->d2 = d * d * (1.0 - 1e-9);
}

// The particle update of a tick that changes no geometry (particles_core with
// the intervals kept), by two warps: one the translation (lane k < D component
// k), one the rotation.  The new state goes to a ResidentNew; nothing of the
// record changes before every thread has seen the verdict (keep).
struct ResidentNew {
    double v[3], R[3], w[3], e[3], F[3], T[3];
    int moved, alpha, keep;
};
// the chunks' sums in the order of particles_core: a butterfly over 32 lanes of one chunk each
__device__ __forceinline__ double resident_sum(const double (*part)[kPartialStride], int nch, int k) {
    double v[kResMaxChunks];
#pragma unroll
    for (int c = 0; c < kResMaxChunks; ++c) v[c] = c < nch ? part[c][k] : 0.0;
    // lanes 8, 4, 2, 1 apart; chunks past the list are zero
#pragma unroll
    for (int o = kResMaxChunks / 2; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < o; ++c) v[c] += v[c + o];
    static_assert(kResMaxChunks <= 32, "one lane per chunk");
    return v[0];
}
template <int D>
__device__ __forceinline__ void resident_translate(const ParticleArgs& a, const ParticleDev& P, const ResidentKeep& K,
                                                   const double (*part)[kPartialStride], int nch, int lane,
                                                   ResidentNew* N) {
    const int k = lane & 3;  // lanes 4.. repeat lanes 0..3; component 3 (and 2 in 2D) is idle
    const bool on = k < D;
    const int q = on ? k : 0;
    const double F = resident_sum(part, nch, q);
    const double dt = a.dt;
    double v = P.v[q], R = P.R[q];
    bool moved = false;
    if (P.rules == 1) {  // the CPU module's rules: a step whenever v != 0 (see particles_core)
        v = v + P.inv_mass * (dt * F);
        moved = __any_sync(0xffffffffu, v != 0.0);
        if (moved) R = R + dt * v;
    } else if (P.coupleF) {
        v = v + dt * (F * P.inv_mass);
        R = R + dt * v;
        moved = __any_sync(0xffffffffu, v != 0.0);
    }
    // every lane takes part in the shuffles, whatever the tests say
    const double d = on ? R - P.vR[q] : 0.0;
    double d2 = d * d;
    d2 += __shfl_xor_sync(0xffffffffu, d2, 1);
    d2 += __shfl_xor_sync(0xffffffffu, d2, 2);
    const int ok = __all_sync(0xffffffffu, R > K.lo[q] && R < K.hi[q] && d2 < K.d2);
    if (lane < D) {
        N->v[k] = v;
        N->R[k] = R;
        N->F[k] = P.rules == 1 ? dt * F : F;
    }
    if (lane == 0) {
        N->moved = moved;
        N->keep = ok || !moved;
    }
}
template <int D>
__device__ __forceinline__ void resident_rotate(const ParticleArgs& a, const ParticleDev& P,
                                                const double (*part)[kPartialStride], int nch, int lane,
                                                ResidentNew* N) {
    constexpr int NW = D == 2 ? 1 : 3;
    double T[3] = {0, 0, 0}, w[3] = {P.w[0], P.w[1], P.w[2]}, e[3] = {P.e[0], P.e[1], P.e[2]};
#pragma unroll
    for (int k = 0; k < NW; ++k) T[k] = resident_sum(part, nch, 3 + k);
    const double dt = a.dt;
    bool alpha = false;
    if (P.rules == 1) {
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            const double dL = dt * T[k];
            w[k] = w[k] + P.inv_inertia * dL;
            alpha = alpha || dL != 0.0;
        }
    } else if (P.coupleT) {
        double Al[3] = {0, 0, 0};
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            Al[k] = T[k] * P.inv_inertia;
            w[k] = w[k] + dt * Al[k];
            alpha = alpha || Al[k] != 0.0;
        }
        if (P.kind == 1) rotate_direction<D>(w, dt, e);
    }
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            N->w[k] = w[k];
            N->e[k] = e[k];
            N->T[k] = P.rules == 1 ? dt * T[k] : T[k];
        }
        N->alpha = alpha;
    }
}
// the kept update into the record, by one warp
template <int D>
__device__ __forceinline__ void resident_commit(const ParticleArgs& a, ParticleDev& P, const ResidentNew& N, int lane) {
    constexpr int NW = D == 2 ? 1 : 3;
    const bool nv = N.moved || N.alpha;  // getNodeVelocity: the snapshot of the slip velocity
    if (lane < D) {
        P.v[lane] = N.v[lane];
        P.R[lane] = N.R[lane];
        P.e[lane] = N.e[lane];
        if (N.moved) P.mR[lane] = N.R[lane];
        if (nv) {
            P.sR[lane] = N.R[lane];
            P.sV[lane] = N.v[lane];
            P.sE[lane] = N.e[lane];
        }
    }
    if (lane >= 4 && lane < 4 + NW) {
        P.w[lane - 4] = N.w[lane - 4];
        if (nv) P.sW[lane - 4] = N.w[lane - 4];
    }
    if (lane >= 8 && lane < 11) {
        P.lastF[lane - 8] = lane - 8 < D ? N.F[lane - 8] : 0.0;
        P.lastT[lane - 8] = N.T[lane - 8];
    }
    if (lane == 11) {
        P.relink = 0;
        P.valid = 1;
    }
    __syncwarp();
    if (lane == 0 && a.trj) {
        double* r = a.trj + (P.nrec % a.trj_cap) * a.nparts * 9;
        for (int q = 0; q < 3; ++q) {
            r[q] = P.R[q];
            r[3 + q] = P.v[q];
            r[6 + q] = P.w[q];
        }
        P.nrec += 1;
    }
}

// Ladd term and momentum exchange of one slot with the slip velocity's c_i . u
// already known (ladd_link)
template <int D>
__device__ __forceinline__ void resident_exchange(const StepArgs& a, const ParticleDev& P, const int* ci,
                                                  const double* Xc, double gi, double wi, double v, double* acc) {
    const double cs = a.coeff * (wi * (2.0 * a.rho0 + gi + v));
    if (P.coupleF || P.recordF) {
#pragma unroll
        for (int k = 0; k < D; ++k) acc[k] += cs * ci[k];
    }
    if (P.coupleT) {
        const double r0 = Xc[0] - P.mR[0], r1 = Xc[1] - P.mR[1], r2 = D == 3 ? Xc[2] - P.mR[2] : 0.0;
        if (D == 2) {
            acc[3] += cs * (r0 * ci[1] - r1 * ci[0]);
        } else {
            acc[3] += cs * (r1 * ci[2] - r2 * ci[1]);
            acc[4] += cs * (-r0 * ci[2] + r2 * ci[0]);
            acc[5] += cs * (r0 * ci[1] - r1 * ci[0]);
        }
    }
}

// One CTA per SM (128 registers): the chain of latencies gains nothing from
// occupancy.
template <class L, int ST, bool TRT>
__global__ void __launch_bounds__(kResThreads, 1) k_resident(const __grid_constant__ ResidentArgs ra) {
    using SS = Store<ST>;
    using T = typename SS::T;
    using R = typename SS::R;
    constexpr int Q = L::Q, D = L::D;
    constexpr int kHalves = kResThreads / kResHalf;
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ StepArgs s_a[2];
    __shared__ ParticleArgs s_pa;
    __shared__ unsigned *s_pmask;
    __shared__ const unsigned* s_wmask;
    __shared__ ParticleDev sP;
    __shared__ ResidentKeep s_keep;
    __shared__ ResidentNew s_new;
    __shared__ double s_part[kResMaxChunks][kPartialStride];
    __shared__ double s_red[kResThreads / 32][6];
    __shared__ int s_off[kResMaxChunks + 1];  // first slot of each chunk
    __shared__ int s_wcnt[2];
    __shared__ int s_lat[4][Q];  // c_i (3) and i of the slot direction j, i = opp(j)
    __shared__ double s_w[Q];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool grid = ra.bar != nullptr;
    const int rank = grid ? (int)blockIdx.x : (int)cluster_rank();
    const int csize = grid ? (int)gridDim.x : (int)cluster_size();
    ResidentBarrier bar{ra.bar, ra.err, 0u, (unsigned)csize};
    for (int j = tid; j < Q; j += kResThreads) {
        s_lat[0][j] = -L::cx(j);
        s_lat[1][j] = -L::cy(j);
        s_lat[2][j] = -L::cz(j);
        s_lat[3][j] = L::opp(j);
        s_w[j] = L::w(j);
    }
    const ResidentJob& J = *ra.job;
    for (int k = tid; k < (int)(2 * sizeof(StepArgs) / 4); k += kResThreads)
        reinterpret_cast<int*>(s_a)[k] = reinterpret_cast<const int*>(J.a)[k];
    for (int k = tid; k < (int)(sizeof(ParticleArgs) / 4); k += kResThreads)
        reinterpret_cast<int*>(&s_pa)[k] = reinterpret_cast<const int*>(&J.pa)[k];
    if (tid == 0) {
        s_pmask = J.pmask;
        s_wmask = J.wmask;
    }
    __syncthreads();
    const bool part = s_a[0].nparts > 0;
    const bool walls = s_a[0].nwnodes > 0;
    const int bulk_ctas = part && csize > 1 ? csize - 1 : csize;
    const bool does_bulk = rank < bulk_ctas, boundary = part && rank == csize - 1;
    const int nx = s_a[0].g.n[0], ny = s_a[0].g.n[1], nz = s_a[0].g.n[2];
    unsigned* pmask = part ? s_pmask : nullptr;
    const unsigned* wmask = s_wmask;
    const int first = rank * kResThreads + tid, stride = bulk_ctas * kResThreads;
    const int x0 = first % nx, y0 = D == 2 ? first / nx : (first / nx) % ny, z0 = D == 2 ? 0 : first / (nx * ny);
    ResidentBoundary<L, ST> B(s_dyn, ra.max_entries);
    int entries = 0, nch = 0;
    // the source node of slot `item` (the node pushed from by plain streaming)
    auto source = [&](int item) -> int {
        const int cell = B.cell[item >> 5], j = item & 31;
        const int x = wrap_idx(cell % nx + s_lat[0][j], nx), y = wrap_idx((cell / nx) % ny + s_lat[1][j], ny);
        const int z = D == 2 ? 0 : wrap_idx(cell / (nx * ny) + s_lat[2][j], nz);
        return x + nx * (y + ny * z);
    };
    // entries, coordinates and slot list of the current links, and pmask with them
    auto relist = [&]() {
        const int old = nch > 0 ? s_off[nch] : 0;
        for (int l = tid; l < old; l += kResThreads) pmask[source(B.list[l])] = 0u;
        __syncthreads();
        const int nl = sP.nlinks;
        entries = min(nl, B.E);
        if (nl > B.E && tid == 0) atomicOr(s_a[0].err, kErrLinkOverflow);
        nch = (entries + kFixBlock - 1) / kFixBlock;
        for (int e = tid; e < entries; e += kResThreads) {
            const int2 ent = s_a[0].links[sP.link_off + e];
            B.cell[e] = ent.x;
            B.mask[e] = ent.y;
            const int xyz[3] = {ent.x % nx, (ent.x / nx) % ny, ent.x / (nx * ny)};
#pragma unroll
            for (int k = 0; k < D; ++k)
#pragma unroll
                for (int o = 0; o < 3; ++o)
                    B.C[(k * 3 + o) * B.E + e] = s_a[0].coord[k][wrap_idx(xyz[k] + o - 1, s_a[0].g.n[k])];
        }
        if (tid == 0) {
            s_off[0] = 0;
            resident_keep<D>(s_pa, sP, &s_keep);
        }
        __syncthreads();
        for (int c = 0; c < nch; ++c) {  // slots in entry order, as fixup_body lists them
            const int e = c * kFixBlock + tid;
            const unsigned mask = tid < kFixBlock && e < entries ? (unsigned)B.mask[e] : 0u;
            int off = __popc(mask);
            const int cnt = off;
            if (tid < kFixBlock) {
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, off, o);
                    if (lane >= o) off += v;
                }
                if (lane == 31) s_wcnt[tid >> 5] = off;
            }
            __syncthreads();
            if (tid < kFixBlock) {
                off += s_off[c] - cnt + (tid >= 32 ? s_wcnt[0] : 0);
                for (unsigned m = mask; m; m &= m - 1) B.list[off++] = (unsigned short)((e << 5) | (__ffs(m) - 1));
            }
            if (tid == 0) s_off[c + 1] = s_off[c] + s_wcnt[0] + s_wcnt[1];
            __syncthreads();
        }
        const int now = nch > 0 ? s_off[nch] : 0;
        for (int l = tid; l < now; l += kResThreads) atomicOr(pmask + source(B.list[l]), 1u << (B.list[l] & 31));
    };
    // c_i . slip velocity at every slot's source node, for the record's snapshot
    auto slip = [&]() {
        const int now = nch > 0 ? s_off[nch] : 0;
        for (int l = tid; l < now; l += kResThreads) {
            const int item = B.list[l], e = item >> 5, j = item & 31;
            const int ci0 = s_lat[0][j], ci1 = s_lat[1][j], ci2 = s_lat[2][j];
            const double Tc[3] = {B.C[(1 + ci0) * B.E + e], B.C[(4 + ci1) * B.E + e],
                                  D == 3 ? B.C[(7 + ci2) * B.E + e] : 0.0};
            double up[3];
            if (sP.rules == 1)
                slip_velocity_cpu<D>(sP.sR, sP.sV, sP.sW, sP.sE, sP.B1, sP.B2, sP.kind, sP.radius,
                                     2.0 * s_a[0].half_dt, Tc[0], Tc[1], Tc[2], up);
            else
                slip_velocity<D>(sP.sR, sP.sV, sP.sW, sP.sE, sP.B1, sP.B2, sP.kind, Tc[0], Tc[1], Tc[2], up);
            B.cu[l] = ci0 * up[0] + ci1 * up[1] + ci2 * up[2];
        }
    };
    if (boundary) {
        const unsigned long long* from = reinterpret_cast<const unsigned long long*>(s_pa.parts);
        for (int k = tid; k < (int)(sizeof(ParticleDev) / 8); k += kResThreads)
            reinterpret_cast<unsigned long long*>(&sP)[k] = from[k];
        __syncthreads();
        if (tid == 0) s_pa.partial = &s_part[0][0] - (long long)sP.part_off * kPartialStride;  // from part_off on
        relist();
        slip();
        __syncthreads();
    }
    if (part) {  // pmask is set before the first push
        bar.arrive();
        if (!bar.wait()) return;
    }
    for (int t = 0; t < ra.ticks; ++t) {
        const StepArgs& a = s_a[t & 1];
        if (does_bulk) {
            if (walls) resident_bulk<L, ST, TRT, true>(a, pmask, wmask, first, stride, x0, y0, z0, t < 2);
            else resident_bulk<L, ST, TRT, false>(a, pmask, wmask, first, stride, x0, y0, z0, false);
        }
        if (boundary) {
            // the link nodes, collided from src
            for (int e = tid; e < entries; e += kResThreads) {
                R g[Q];
                const int cell = B.cell[e];
                load_pops_l2<L, ST>(a, cell, g);
                B.rho[e] = (double)collide_node<L, ST, TRT>(a, cell, true, g);
#pragma unroll
                for (int i = 0; i < Q; ++i) B.g[i * B.E + e] = g[i] * R(a.inv_scale);
            }
            __syncthreads();
            // slot values, stored at once (nobody else writes them), and the momentum exchange:
            // each half of the CTA a chunk
            T* dst = static_cast<T*>(a.dst);
            for (int c0 = 0; c0 < nch; c0 += kHalves) {
                const int c = c0 + tid / kResHalf;
                double acc[6] = {0, 0, 0, 0, 0, 0};
                if (c < nch) {
                    const int l1 = s_off[c + 1];
                    for (int l = s_off[c] + tid % kResHalf; l < l1; l += kResHalf) {
                        const int item = B.list[l], e = item >> 5, j = item & 31, cell = B.cell[e];
                        if (walls && a.wall[cell]) continue;  // wall nodes hold f = 0 (fluids.jl:154)
                        const int ci[3] = {s_lat[0][j], s_lat[1][j], s_lat[2][j]};
                        const double rhoL = B.rho[e], gi = (double)B.g[s_lat[3][j] * B.E + e];
                        double v = gi;  // halfway bounce-back: f_j(x) = f*_i(x)
                        if (a.uw) {     // moving walls (fluids.jl:168-174)
                            const int q = source(item);
                            const double dot = -(ci[0] * a.uw[q] + ci[1] * a.uw[a.g.N + q] +
                                                 (D == 3 ? ci[2] * a.uw[2 * a.g.N + q] : 0.0));
                            v += 6.0 * rhoL * dot;
                        }
                        if (sP.dirlinks >> j & 1u) {
                            v += 6.0 * rhoL * -B.cu[l];
                            if (sP.coupleF || sP.coupleT || sP.recordF) {
                                const double Xc[3] = {B.C[B.E + e], B.C[4 * B.E + e], D == 3 ? B.C[7 * B.E + e] : 0.0};
                                resident_exchange<D>(a, sP, ci, Xc, gi, s_w[j], v, acc);
                            }
                        }
                        dst[j * a.g.N + cell] = SS::enc((R)v, R(a.scale));
                    }
                    // as fixup_body: butterfly inside warps, then the warps in order
#pragma unroll
                    for (int k = 0; k < (D == 2 ? 4 : 6); ++k) {
                        if (D == 2 && k == 2) continue;  // (2D: two force components and one torque)
                        for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
                        if (lane == 0) s_red[warp][k] = acc[k];
                    }
                }
                __syncthreads();
                if (tid < 6 * kHalves && c0 + tid / 6 < nch) {
                    const int h = tid / 6, k = tid % 6;
                    double sum = 0.0;
                    if (D == 3 || (k < 4 && k != 2))
                        for (int w = 0; w < kResHalf / 32; ++w) sum += s_red[h * (kResHalf / 32) + w][k];
                    s_part[c0 + h][k] = sum;
                }
                __syncthreads();
            }
            if (warp == 0) resident_translate<D>(s_pa, sP, s_keep, s_part, nch, lane, &s_new);
            else if (warp == 1) resident_rotate<D>(s_pa, sP, s_part, nch, lane, &s_new);
            __syncthreads();
            if (!s_new.keep) {  // the geometry may change: the full update, and pmask before the barrier
                if (particles_core<L, 128>(s_pa, 0, sP)) {
                    __syncthreads();
                    relist();
                }
                __syncthreads();
                bar.arrive();
            } else {
                bar.arrive();
                if (warp == 0) resident_commit<D>(s_pa, sP, s_new, lane);
            }
            __syncthreads();
            slip();
        } else {
            __syncthreads();
            bar.arrive();
        }
        if (!bar.wait()) return;
    }
    if (boundary) {  // pmask back to zero, the record back to global memory
        __syncthreads();
        const int now = nch > 0 ? s_off[nch] : 0;
        for (int l = tid; l < now; l += kResThreads) pmask[source(B.list[l])] = 0u;
        store_record(s_pa, 0, sP);
        if (tid == 0) publish_box(s_pa, 0, sP);
    }
}

}  // namespace lbm
