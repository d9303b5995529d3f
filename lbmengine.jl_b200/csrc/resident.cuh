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
// The operations of a node, a link slot and a particle, and the order of the
// FP64 sums, are those of k_bulk, k_fixup and k_particles.  The compiler may
// contract the particle's here otherwise than there: its state agrees with the
// stream schedule's to 1e-12 of itself while the stored populations round
// alike, and these to a unit in the last place (1e-7 FP32, 1e-13 FP64; tested).
//
// Measured in calls of 2,000 ticks, us per tick, against the stream schedule:
// with a squirmer 64^2 FP32 3.4 (9.0), 256 x 128 FP64 4.0 (9.5), 201 x 65 FP64 with
// walls 4.2 (9.6), 512 x 256 FP32 4.0 (9.4), 724^2 FP32 8.9 (10.2); with a bead
// 201 x 65 FP64 with walls 3.8 (9.4), with a moving lid 5.0 (9.6); faster swimmers, whose
// geometry changes more often, 0.2-0.6 more.  The chain that bounds it: barrier and fence 1.0,
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
#include "interactions.cuh"

namespace lbm {

constexpr int kResThreads = 512;      // threads per CTA
constexpr int kResHalf = 256;         // threads per chunk of link entries (= the fix-up's CTA: sums in the same order)
constexpr int kResMaxCluster = 16;
constexpr int kResMaxChunks = 32;                            // one lane per chunk in resident_sum
constexpr int kResMaxEntries = kResMaxChunks * kFixBlock;    // link entries of a particle
constexpr int kResMaxParts = 32;
constexpr int kResMaxInter = 128;                            // interaction contributions to one particle
constexpr size_t kResMaxSmem = 200 * 1024;                   // dynamic shared memory per CTA

struct ResidentJob {
    StepArgs a[2];          // by tick parity
    ParticleArgs pa;
    InterArgs in;           // particle interactions (nitems 0: none)
    unsigned* pmask;        // [2][N] directions a node does not push, the particles' link slots, by tick parity
                            // (a geometry change of tick t goes to tick t + 1's mask while the bulk phase still
                            // reads tick t's); zero between launches
    const unsigned* wmask;  // [N] the same for wall nodes and wall links (static), or null
    int* box;               // [nparts][6] solid boxes, kept current while the launch runs
    double* pos;            // [2][nparts][3] positions at the start of a tick, by its parity
};

struct ResidentArgs {
    const ResidentJob* job;
    int ticks;
    int cap_entries, cap_slots, cap_box;  // shared memory of a boundary CTA (ResidentBoundary)
    unsigned* bar;       // grid barrier: counter (zero at launch) and the phase the launch ends at (all
                         // ones at launch); null: cluster barrier
    int* err;            // of the grid barrier
    int spin_limit;        // polls before a wait at the grid barrier gives up (2^22: about a second)
    unsigned wait_extra;   // test knob: added to the count it waits for
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
// for the CTA.  stop (grid barrier only): every CTA leaves after this phase;
// the counter's top bit says that some phase was named, the second word which
// one (a CTA still waiting for an earlier phase must not leave at it).
// wait(): by every thread; kGoOn, kStop, or kGaveUp when the bounded wait ran
// out (every CTA then gives up at its next wait).
struct ResidentBarrier {
    enum { kGoOn = 0, kStop = 1, kGaveUp = 2 };
    unsigned* ctr;      // null: cluster barrier
    int* err;
    unsigned phase;     // phases completed
    unsigned ctas;
    int limit;          // polls of a wait
    unsigned goal;      // arrivals that the last wait waited for (at first: wait_extra)
    __device__ __forceinline__ void arrive(bool stop = false) {
        if (ctr) {
            if (threadIdx.x == kResThreads - 32) {
                if (stop) atomicMin(ctr + 1, phase + 1);
                __threadfence();
                if (stop) atomicOr(ctr, 0x80000000u);  // before the arrival: who sees the one sees the other
                atomicAdd(ctr, 1u);
            }
        } else if (threadIdx.x >= kResThreads - 32) {
            __threadfence();
            cluster_arrive();
        } else {
            cluster_arrive_relaxed();
        }
    }
    static __device__ __forceinline__ unsigned load(const unsigned* p) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        return v;
    }
    __device__ __forceinline__ int wait() {
        ++phase;
        if (!ctr) {
            cluster_wait();
            return kGoOn;
        }
        goal += ctas;
        __shared__ int s_state;
        if (threadIdx.x == 0) {
            int state = kGoOn, it = 0;
            while (true) {
                const unsigned v = load(ctr);
                if ((v & 0x7fffffffu) >= goal) {
                    if ((v & 0x80000000u) && load(ctr + 1) <= phase) state = kStop;
                    break;
                }
                if (++it > limit) {
                    atomicOr(err, kErrSpinTimeout);
                    state = kGaveUp;
                    break;
                }
            }
            s_state = state;
        }
        __syncthreads();
        return s_state;
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
                                              int cell, int x, int y, typename Store<ST>::R* g, bool first) {
    using SS = Store<ST>;
    using T = typename SS::T;
    using R = typename SS::R;
    constexpr int Q = L::Q;
    const int nx = a.g.n[0], ny = a.g.n[1];
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
#pragma unroll
    for (int i = 0; i < Q; ++i)
        if (!(skip >> i & 1u))
            dst[i * N + (xs[L::cx(i) + 1] + nx * ys[L::cy(i) + 1])] = SS::enc(g[i], R(1));
    if (WALLS && wm) {
#pragma unroll
        for (int i = 1; i < Q; ++i) {
            if (!(wm >> i & 1u)) continue;  // x + c_i is a wall node: f_j(x) = f*_i(x), j = opp(i)
            const int j = L::opp(i);
            const int t = xs[L::cx(i) + 1] + nx * ys[L::cy(i) + 1];
            if (pmask && (__ldcg(pmask + t) >> j & 1u)) continue;  // also the particle's link: the boundary CTA's
            double v = (double)(g[i] * R(a.inv_scale));
            if (a.uw) {  // moving walls (fluids.jl:168-174)
                const double dot = -(L::cx(i) * a.uw[t] + L::cy(i) * a.uw[N + t]);
                v += 6.0 * (double)rho * dot;
            }
            dst[j * N + cell] = SS::enc((R)v, R(a.scale));
        }
    }
    return bad_density(rho);
}

// Nodes first, first + stride, ... of the grid, two at a time, so that the loads
// of both are in flight together.
template <class L, int ST, bool TRT, bool WALLS>
__device__ __forceinline__ void resident_bulk(const StepArgs& a, const unsigned* pmask, const unsigned* wmask,
                                              int first, int stride, int x, int y, const int* step, bool init) {
    using R = typename Store<ST>::R;
    const int nx = a.g.n[0], N = (int)a.g.N;
    bool bad = false;
    auto advance = [&]() {  // (x, y) of the node `stride` further on
        x += step[0];
        y += step[1];
        if (x >= nx) {
            x -= nx;
            ++y;
        }
    };
    for (int cell = first; cell < N; cell += 2 * stride) {
        const int c2 = cell + stride;
        const bool two = c2 < N;
        R g[2][L::Q];
        load_pops_l2<L, ST>(a, cell, g[0]);
        load_pops_l2<L, ST>(a, two ? c2 : cell, g[1]);
        bad |= resident_node<L, ST, TRT, WALLS>(a, pmask, wmask, cell, x, y, g[0], init);
        if (!two) break;
        advance();
        bad |= resident_node<L, ST, TRT, WALLS>(a, pmask, wmask, c2, x, y, g[1], init);
        advance();
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
        const int nx = g.n[0], ny = g.n[1], x = (int)(c % nx), y = (int)(c / nx);
#pragma unroll
        for (int i = 1; i < L::Q; ++i)
            if (wall[wrap_idx(x + L::cx(i), nx) + (long long)nx * wrap_idx(y + L::cy(i), ny)]) m |= 1u << i;
    }
    wmask[c] = m;
}

// Shared memory of a boundary CTA: capacities E (link entries), S (slots) and
// B (nodes per axis of the near box and one more on each side).
template <int ST>
struct ResidentBoundary {
    using R = typename Store<ST>::R;
    int E, S, B;
    double* cu;       // [S] c_i . slip velocity of the slots' source nodes
    double* rho;      // [E] density of the entries
    double* X;        // [3][B] node coordinates per axis, from slo - 2 on (periodic)
    R* gi;            // [S] f*_i/w - rho0 of the slots' directions i = opp(j)
    int* cell;        // [E]
    int* mask;        // [E]
    int* loc;         // [E] position in the near box, 10 bits per axis
    int* slot;        // [E] first slot
    int* src;         // [2][S] source nodes whose pushes pmask leaves out, by tick parity
    unsigned short* list;  // [S] (entry << 5) | j, chunk by chunk of kFixBlock entries
    static __host__ __device__ size_t bytes(int E, int S, int B) {
        return sizeof(double) * ((size_t)S + E + 3 * B) + sizeof(R) * (size_t)S +
               sizeof(int) * (4 * (size_t)E + 2 * (size_t)S) + sizeof(unsigned short) * (size_t)S;
    }
    __device__ __forceinline__ ResidentBoundary(unsigned char* p, int e, int s, int b) : E(e), S(s), B(b) {
        cu = reinterpret_cast<double*>(p);
        rho = cu + S;
        X = rho + E;
        gi = reinterpret_cast<R*>(X + 3 * B);
        cell = reinterpret_cast<int*>(gi + S);
        mask = cell + E;
        loc = mask + E;
        slot = loc + E;
        src = slot + E;
        list = reinterpret_cast<unsigned short*>(src + 2 * S);
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
    double v[2], R[2], e[2], F[2], w, T;
    int moved, alpha, keep;
};
// the chunks' sums in the order of particles_core: a butterfly over the lanes of one chunk each (a whole warp)
__device__ __forceinline__ double resident_sum(const double (*part)[kPartialStride], int nch, int k, int lane) {
    static_assert(kResMaxChunks == 32, "one lane per chunk");
    if (nch <= 2) return nch == 0 ? 0.0 : (nch == 1 ? part[0][k] : part[0][k] + part[1][k]);  // the same sum
    double v = lane < nch ? part[lane][k] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <int D>
__device__ __forceinline__ void resident_translate(const ParticleArgs& a, const ParticleDev& P, const ResidentKeep& K,
                                                   const double (*part)[kPartialStride], int nch, int lane,
                                                   const double* fint, ResidentNew* N) {
    const int k = lane & 3;  // lanes 4.. repeat lanes 0..3; component 3 (and 2 in 2D) is idle
    const bool on = k < D;
    const int q = on ? k : 0;
    double F = 0.0;
#pragma unroll
    for (int c = 0; c < D; ++c) {
        const double f = resident_sum(part, nch, c, lane);
        if (q == c) F = f;
    }
    if (fint) F += fint[q];  // the interactions' share of the force input
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
    const double T = resident_sum(part, nch, 3, lane), dt = a.dt;
    double w = P.w[0], e[3] = {P.e[0], P.e[1], P.e[2]};
    bool alpha = false;
    if (P.rules == 1) {
        const double dL = dt * T;
        w = w + P.inv_inertia * dL;
        alpha = dL != 0.0;
    } else if (P.coupleT) {
        const double Al = T * P.inv_inertia;
        w = w + dt * Al;
        alpha = Al != 0.0;
        if (P.kind == 1) rotate_direction<D>(&w, dt, e);
    }
    if (lane == 0) {
        for (int k = 0; k < 2; ++k) N->e[k] = e[k];
        N->w = w;
        N->T = P.rules == 1 ? dt * T : T;
        N->alpha = alpha;
    }
}
// the kept update into the record, by one warp
template <int D>
__device__ __forceinline__ void resident_commit(const ParticleArgs& a, int p, ParticleDev& P, const ResidentNew& N,
                                                int lane) {
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
    if (lane == 4) {
        P.w[0] = N.w;
        if (nv) P.sW[0] = N.w;
    }
    if (lane >= 8 && lane < 11) {
        P.lastF[lane - 8] = lane - 8 < D ? N.F[lane - 8] : 0.0;
        P.lastT[lane - 8] = lane == 8 ? N.T : 0.0;
    }
    if (lane == 11) {
        P.relink = 0;
        P.valid = 1;
    }
    __syncwarp();
    if (lane == 0 && a.trj) {
        double* r = a.trj + ((P.nrec % a.trj_cap) * a.nparts + p) * 9;
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
__device__ __forceinline__ void resident_exchange(const StepArgs& a, const ParticleDev& P, const int* ci,
                                                  const double* Xc, double gi, double wi, double v, double* acc) {
    const double cs = a.coeff * (wi * (2.0 * a.rho0 + gi + v));
    if (P.coupleF || P.recordF) {
        acc[0] += cs * ci[0];
        acc[1] += cs * ci[1];
    }
    if (P.coupleT) {
        const double r0 = Xc[0] - P.mR[0], r1 = Xc[1] - P.mR[1];
        acc[3] += cs * (r0 * ci[1] - r1 * ci[0]);
    }
}

// do the periodic index ranges of the near box of `b` grown by two nodes and the
// near box of `o` meet (boxes as lo[3], hi[3] of the solid nodes)?
template <int D>
__device__ __forceinline__ bool resident_close(const int* b, const int* o, const int* n) {
    bool meet = true;
    for (int k = 0; k < D; ++k) {
        if (b[k] > b[3 + k] || o[k] > o[3 + k]) return true;  // an empty region: left to the general path
        meet = meet && ranges_meet(b[k] - 3, b[3 + k] - b[k] + 7, o[k] - 1, o[3 + k] - o[k] + 3, n[k]);
    }
    return meet;
}

// One CTA per SM (128 registers): the chain of latencies gains nothing from
// occupancy.  The last nparts CTAs are the particles' boundary CTAs.
//
// With several particles each must be alone (no other particle's near box close
// to its own) with links in every direction, so that a slot belongs to one
// particle; a boundary CTA that finds otherwise, or whose links outgrow its
// shared memory, ends the launch after the tick (the caller goes on with the
// stream schedule).  Boxes of the others are read while they may be moving: by
// at most a node per tick, which the margin of two nodes covers.
template <class L, int ST, bool TRT>
__global__ void __launch_bounds__(kResThreads, 1) k_resident(const __grid_constant__ ResidentArgs ra) {
    using SS = Store<ST>;
    using T = typename SS::T;
    using R = typename SS::R;
    constexpr int Q = L::Q, D = L::D;
    static_assert(D == 2, "a 2D kernel");
    constexpr int kHalves = kResThreads / kResHalf;
    constexpr unsigned kAllDirs = (Q == 32 ? 0u : (1u << Q)) - 2u;
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ StepArgs s_a[2];
    __shared__ ParticleArgs s_pa;
    __shared__ ParticleDev sP;
    __shared__ ResidentKeep s_keep;
    __shared__ ResidentNew s_new;
    __shared__ double s_part[kResMaxChunks][kPartialStride];
    __shared__ double s_red[kResThreads / 32][6];
    __shared__ int s_off[kResMaxChunks + 1];  // first slot of each chunk
    __shared__ int s_wcnt[2], s_stop, s_quit, s_box[6];
    __shared__ int s_nsrc[2];  // source nodes set in each parity's pmask
    __shared__ int s_lat[2][Q];  // c_i of the slot direction j, i = opp(j)
    __shared__ double s_w[Q];
    __shared__ double s_fi[kResMaxInter][3], s_fint[3];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool grid = ra.bar != nullptr;
    const int rank = grid ? (int)blockIdx.x : (int)cluster_rank();
    const int csize = grid ? (int)gridDim.x : (int)cluster_size();
    ResidentBarrier bar{ra.bar, ra.err, 0u, (unsigned)csize, ra.spin_limit, ra.wait_extra};
    for (int j = tid; j < Q; j += kResThreads) {
        s_lat[0][j] = -L::cx(j);
        s_lat[1][j] = -L::cy(j);
        s_w[j] = L::w(j);
    }
    const ResidentJob& J = *ra.job;
    for (int k = tid; k < (int)(2 * sizeof(StepArgs) / 4); k += kResThreads)
        reinterpret_cast<int*>(s_a)[k] = reinterpret_cast<const int*>(J.a)[k];
    for (int k = tid; k < (int)(sizeof(ParticleArgs) / 4); k += kResThreads)
        reinterpret_cast<int*>(&s_pa)[k] = reinterpret_cast<const int*>(&J.pa)[k];
    if (tid == 0) {
        s_stop = s_nsrc[0] = s_nsrc[1] = 0;
        // a launch before this one of the same call gave up: what it left is undefined
        s_quit = grid && (*(volatile const int*)ra.err & kErrSpinTimeout) != 0;
    }
    __syncthreads();
    if (s_quit) return;
    const int np = s_a[0].nparts;
    const bool walls = s_a[0].nwnodes > 0;
    const int bulk_ctas = csize - np;
    const bool boundary = rank >= bulk_ctas;
    const int p = rank - bulk_ctas;  // the boundary CTA's particle
    const int nx = s_a[0].g.n[0], ny = s_a[0].g.n[1];
    const long long N = s_a[0].g.N;
    unsigned* const pmask = np > 0 ? J.pmask : nullptr;
    const unsigned* const wmask = J.wmask;
    const int first = rank * kResThreads + tid, stride = bulk_ctas * kResThreads;
    const int x0 = first % nx, y0 = first / nx, step[2] = {stride % nx, stride / nx};
    ResidentBoundary<ST> B(s_dyn, ra.cap_entries, ra.cap_slots, ra.cap_box);
    int entries = 0, nch = 0;
    // the source node of slot `item` (the node pushed from by plain streaming)
    auto source = [&](int item) -> int {
        const int cell = B.cell[item >> 5], j = item & 31;
        const int x = wrap_idx(cell % nx + s_lat[0][j], nx), y = wrap_idx(cell / nx + s_lat[1][j], ny);
        return x + nx * y;
    };
    auto slots = [&]() -> int { return nch > 0 ? s_off[nch] : 0; };
    // pmask of parity b: cleared, and set for the current slots
    auto unmask = [&](int b) {
        for (int l = tid; l < s_nsrc[b]; l += kResThreads) pmask[(size_t)b * N + B.src[b * B.S + l]] = 0u;
    };
    auto set_mask = [&](int b) {
        unmask(b);
        __syncthreads();
        const int now = slots();
        for (int l = tid; l < now; l += kResThreads) {
            const int item = B.list[l], at = source(item);
            B.src[b * B.S + l] = at;
            atomicOr(pmask + (size_t)b * N + at, 1u << (item & 31));
        }
        if (tid == 0) s_nsrc[b] = now;
    };
    // The links outgrew the shared memory (ResidentCaps says that they cannot).
    // Several particles: the launch ends after the tick.  One: a cluster cannot
    // end early, so the call fails instead of going on without the particle.
    auto outgrown = [&]() {
        s_stop = 1;
        if (np == 1) atomicOr(s_a[0].err, kErrLinkOverflow);
    };
    // Entries, coordinates and slot list of the current links; sets s_stop
    // where this launch cannot go on with them.
    auto relist = [&](bool check_move) {
        const int nl = sP.nlinks;
        bool fits = nl <= B.E;
        const int ex = near_extent(sP, s_a[0].g, 0, D), ey = near_extent(sP, s_a[0].g, 1, D),
                  ez = near_extent(sP, s_a[0].g, 2, D);
        fits = fits && ex + 2 <= B.B && ey + 2 <= B.B && ez + 2 <= B.B;
        entries = fits ? nl : 0;
        nch = (entries + kFixBlock - 1) / kFixBlock;
        for (int e = tid; e < entries; e += kResThreads) {
            const int2 ent = s_a[0].links[sP.link_off + e];
            B.cell[e] = ent.x;
            B.mask[e] = ent.y;
            const int xyz[3] = {ent.x % nx, (ent.x / nx) % ny, ent.x / (nx * ny)};
            int loc = 0;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const int n = s_a[0].g.n[k], l = xyz[k] - (sP.slo[k] - 1);
                loc |= (l < 0 ? l + n : (l >= n ? l - n : l)) << (10 * k);
            }
            B.loc[e] = loc;
        }
        if (entries > 0) {
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const int n = s_a[0].g.n[k];
                for (int i = tid; i < near_extent(sP, s_a[0].g, k, D) + 2; i += kResThreads)
                    B.X[k * B.B + i] = s_a[0].coord[k][((sP.slo[k] - 2 + i) % n + n) % n];
            }
        }
        if (tid == 0) {
            s_off[0] = 0;
            resident_keep<D>(s_pa, sP, &s_keep);
            if (!fits) outgrown();
            if (np > 1) {
                if ((sP.dirlinks & kAllDirs) != kAllDirs) s_stop = 1;
                for (int k = 0; k < 3; ++k) {
                    // more than a node per tick: the margin does not hold
                    if (check_move && (abs(sP.slo[k] - s_box[k]) > 1 || abs(sP.shi[k] - s_box[3 + k]) > 1)) s_stop = 1;
                    s_box[k] = sP.slo[k];
                    s_box[3 + k] = sP.shi[k];
                }
                for (int k = 0; k < 6; ++k) __stcg(J.box + 6 * p + k, s_box[k]);
            }
        }
        __syncthreads();
        if (np > 1 && tid < np && tid != p) {
            int o[6];
            for (int k = 0; k < 6; ++k) o[k] = __ldcg(J.box + 6 * tid + k);
            if (resident_close<D>(s_box, o, s_a[0].g.n)) s_stop = 1;
        }
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
            const int base = s_off[c], end = base + s_wcnt[0] + s_wcnt[1];
            if (end > B.S) {  // the same in every thread
                if (tid == 0) outgrown();
                entries = 0;
                nch = 0;
                break;
            }
            if (tid < kFixBlock) {
                off += base - cnt + (tid >= 32 ? s_wcnt[0] : 0);
                if (e < entries) B.slot[e] = off;
                for (unsigned m = mask; m; m &= m - 1) B.list[off++] = (unsigned short)((e << 5) | (__ffs(m) - 1));
            }
            if (tid == 0) s_off[c + 1] = end;
            __syncthreads();
        }
        __syncthreads();
    };
    // the coordinate of entry e's node along axis k, o nodes further on
    auto coord = [&](int e, int k, int o) -> double { return B.X[k * B.B + (B.loc[e] >> (10 * k) & 1023) + 1 + o]; };
    // c_i . slip velocity at every slot's source node, for the record's snapshot
    auto slip = [&]() {
        const int now = slots();
        for (int l = tid; l < now; l += kResThreads) {
            const int item = B.list[l], e = item >> 5, j = item & 31;
            const int ci0 = s_lat[0][j], ci1 = s_lat[1][j];
            const double Tc[2] = {coord(e, 0, ci0), coord(e, 1, ci1)};
            double up[3];
            if (sP.rules == 1)
                slip_velocity_cpu<D>(sP.sR, sP.sV, sP.sW, sP.sE, sP.B1, sP.B2, sP.kind, sP.radius,
                                     2.0 * s_a[0].half_dt, Tc[0], Tc[1], 0.0, up);
            else
                slip_velocity<D>(sP.sR, sP.sV, sP.sW, sP.sE, sP.B1, sP.B2, sP.kind, Tc[0], Tc[1], 0.0, up);
            B.cu[l] = ci0 * up[0] + ci1 * up[1];
        }
    };
    // what the tick loop wants of the job, in registers: behind the barrier's
    // acquire every read of it would go to L2 again
    const bool inter = J.in.nitems > 0;
    const int inter0 = boundary && inter ? J.in.coff[p] : 0, ninter = boundary && inter ? J.in.coff[p + 1] - inter0 : 0;
    const int* const inter_cent = J.in.cent;
    const InterItem* const inter_items = J.in.items;
    double* const positions = J.pos;
    if (boundary) {
        const unsigned long long* from = reinterpret_cast<const unsigned long long*>(s_pa.parts + p);
        for (int k = tid; k < (int)(sizeof(ParticleDev) / 8); k += kResThreads)
            reinterpret_cast<unsigned long long*>(&sP)[k] = from[k];
        __syncthreads();
        if (tid == 0) {  // the CTA's own partial sums and interaction force, indexed as the global arrays
            s_pa.partial = &s_part[0][0] - (long long)sP.part_off * kPartialStride;
            s_pa.fint = J.in.nitems > 0 ? s_fint - 3 * p : nullptr;
        }
        if (tid < 3) __stcg(J.pos + 3 * p + tid, sP.R[tid]);
        if (tid < np && tid != p) {  // the others as the launch finds them
            const ParticleDev& O = s_pa.parts[tid];
            const int b[6] = {sP.slo[0], sP.slo[1], sP.slo[2], sP.shi[0], sP.shi[1], sP.shi[2]};
            const int o[6] = {O.slo[0], O.slo[1], O.slo[2], O.shi[0], O.shi[1], O.shi[2]};
            if ((O.dirlinks & kAllDirs) != kAllDirs || resident_close<D>(b, o, s_a[0].g.n)) s_stop = 1;
            for (int k = 0; k < 6; ++k) __stcg(J.box + 6 * tid + k, o[k]);  // every CTA writes the same
        }
        __syncthreads();
        relist(false);
        set_mask(0);
        set_mask(1);
        slip();
        __syncthreads();
    }
    bool stale = false;  // the other parity's mask is that of the links before the last change
    int t = 0, state = ResidentBarrier::kGoOn;
    if (np > 0) {  // pmask is set before the first push
        bar.arrive(s_stop != 0);
        state = bar.wait();
    }
    for (; t < ra.ticks && state == ResidentBarrier::kGoOn; ++t) {
        const StepArgs& a = s_a[t & 1];
        if (!boundary) {
            const unsigned* pm = pmask ? pmask + (size_t)(t & 1) * N : nullptr;
            if (walls) resident_bulk<L, ST, TRT, true>(a, pm, wmask, first, stride, x0, y0, step, t < 2);
            else resident_bulk<L, ST, TRT, false>(a, pm, wmask, first, stride, x0, y0, step, false);
            __syncthreads();
            bar.arrive();
        } else {
            // the link nodes, collided from src
            for (int e = tid; e < entries; e += kResThreads) {
                R g[Q];
                const int cell = B.cell[e];
                const unsigned mask = (unsigned)B.mask[e];
                load_pops_l2<L, ST>(a, cell, g);
                B.rho[e] = (double)collide_node<L, ST, TRT>(a, cell, true, g);
                int l = B.slot[e];
#pragma unroll
                for (int j = 1; j < Q; ++j)
                    if (mask >> j & 1u) B.gi[l++] = g[L::opp(j)] * R(a.inv_scale);
            }
            if (inter) {  // interactions: the positions at the start of the tick (interactions.cuh)
                const double* pos = positions + (size_t)(t & 1) * 3 * np;
                if (tid >= kResThreads - kResMaxInter && tid - (kResThreads - kResMaxInter) < ninter) {
                    const int q = tid - (kResThreads - kResMaxInter);
                    const int c = inter_cent[inter0 + q];
                    const InterItem it = inter_items[c >> 3];
                    double R1[3], R2[3], R3[3], out[9];
                    for (int k = 0; k < 3; ++k) {
                        R1[k] = __ldcg(pos + 3 * it.id1 + k);
                        R2[k] = __ldcg(pos + 3 * it.id2 + k);
                        R3[k] = it.kind == 2 ? __ldcg(pos + 3 * it.id3 + k) : 0.0;
                    }
                    interaction_force(it, D, R1, R2, R3, out);
                    const double* v = out + 3 * (c >> 1 & 3);
                    for (int k = 0; k < 3; ++k) s_fi[q][k] = c & 1 ? -v[k] : v[k];
                }
                __syncthreads();
                if (tid < 3) {
                    double f = 0.0;
                    for (int q = 0; q < ninter; ++q) f += s_fi[q][tid];
                    s_fint[tid] = f;
                }
            }
            __syncthreads();
            // slot values, stored at once (nobody else writes them), and the momentum exchange:
            // each half of the CTA a chunk
            T* dst = static_cast<T*>(a.dst);
            for (int c0 = 0; c0 < nch; c0 += kHalves) {
                const int c = c0 + tid / kResHalf;
                double acc[4] = {0, 0, 0, 0};  // two force components, (none), the torque
                if (c < nch) {
                    const int l1 = s_off[c + 1];
                    for (int l = s_off[c] + tid % kResHalf; l < l1; l += kResHalf) {
                        const int item = B.list[l], e = item >> 5, j = item & 31, cell = B.cell[e];
                        if (walls && a.wall[cell]) continue;  // wall nodes hold f = 0 (fluids.jl:154)
                        const int ci[2] = {s_lat[0][j], s_lat[1][j]};
                        const double rhoL = B.rho[e], gi = (double)B.gi[l];
                        double v = gi;  // halfway bounce-back: f_j(x) = f*_i(x)
                        if (a.uw) {     // moving walls (fluids.jl:168-174)
                            const int q = source(item);
                            v += 6.0 * rhoL * -(ci[0] * a.uw[q] + ci[1] * a.uw[a.g.N + q]);
                        }
                        if (sP.dirlinks >> j & 1u) {
                            v += 6.0 * rhoL * -B.cu[l];
                            if (sP.coupleF || sP.coupleT || sP.recordF) {
                                const double Xc[2] = {coord(e, 0, 0), coord(e, 1, 0)};
                                resident_exchange(a, sP, ci, Xc, gi, s_w[j], v, acc);
                            }
                        }
                        dst[j * a.g.N + cell] = SS::enc((R)v, R(a.scale));
                    }
                    // as fixup_body: butterfly inside warps, then the warps in order
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        if (k == 2) continue;
                        for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
                        if (lane == 0) s_red[warp][k] = acc[k];
                    }
                }
                __syncthreads();
                if (tid < 6 * kHalves && c0 + tid / 6 < nch) {
                    const int h = tid / 6, k = tid % 6;
                    double sum = 0.0;
                    if (k < 4 && k != 2)
                        for (int w = 0; w < kResHalf / 32; ++w) sum += s_red[h * (kResHalf / 32) + w][k];
                    s_part[c0 + h][k] = sum;
                }
                __syncthreads();
            }
            if (warp == 0)
                resident_translate<D>(s_pa, sP, s_keep, s_part, nch, lane, inter ? s_fint : nullptr, &s_new);
            else if (warp == 1)
                resident_rotate<D>(s_pa, sP, s_part, nch, lane, &s_new);
            __syncthreads();
            double* next = positions + (size_t)((t + 1) & 1) * 3 * np + 3 * p;
            if (!s_new.keep) {  // the geometry may change: the full update, and pmask before the barrier
                const bool changed = particles_core<L, 128>(s_pa, p, sP);
                __syncthreads();
                if (changed) relist(true);
                if (changed || stale) set_mask((t + 1) & 1);
                stale = changed;
                if (tid < 3) __stcg(next + tid, sP.R[tid]);
                __syncthreads();
                bar.arrive(s_stop != 0);
            } else {
                if (stale) {
                    set_mask((t + 1) & 1);
                    stale = false;
                    __syncthreads();
                }
                if (inter) {
                    if (tid < D) __stcg(next + tid, s_new.R[tid]);
                    else if (tid < 3) __stcg(next + tid, 0.0);
                    __syncthreads();
                }
                bar.arrive();
                if (warp == 0) resident_commit<D>(s_pa, p, sP, s_new, lane);
            }
            __syncthreads();
            slip();
        }
        state = bar.wait();
    }
    if (state == ResidentBarrier::kGaveUp) return;
    if (boundary) {  // pmask back to zero, the record back to global memory
        __syncthreads();
        unmask(0);
        unmask(1);
        store_record(s_pa, p, sP);
        if (tid == 0) publish_box(s_pa, p, sP);
    }
}

}  // namespace lbm
