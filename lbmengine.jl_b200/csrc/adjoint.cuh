// Discrete adjoint of one tick (reverse mode), for gradients of a particle
// observable with respect to the squirmer modes B1, B2, the relaxation times
// and the uniform body force.  No counterpart in the reference (it has no
// differentiation); the forward map differentiated is the tick of
// tick!/moveParticles! (src/gpu/fluids.jl:132-226, src/gpu/particles.jl:7-92)
// as this library runs it:
//   f*(x)        = collide(f^n(x); tau+, tau-, F)                (fluids.jl:58-127)
//   f^{n+1}_i(x+c_i) = f*_i(x)                                   (push streaming)
//   f^{n+1}_j(x) = f*_i(x) + 6 w_j rho^n(x) c_j.u_p(x-c_j),  i = opp(j),
//                  for the particle's boundary links (x fluid, x - c_j solid)
//   F = sum_links coeff (f*_i + f^{n+1}_j) c_i,  T = sum_links coeff (f*_i + f^{n+1}_j) (x - R) x c_i
// Walls (static, fluids.jl:147-174): wall nodes hold f = 0 after streaming,
// and a fluid node x whose source x - c_j is a wall node gets
//   f^{n+1}_j(x) = f*_i(x) + 6 w_j rho^n(x) c_j.u_w(x - c_j)  (+ the particles' Ladd terms),
// which the momentum exchange of a particle with the same link also sees.
// The solid masks are held as the forward run computed them (their
// derivative is zero almost everywhere).  Adjoint populations are FP64 and
// in f units; the forward populations are read in their storage format and
// the local linearisation is evaluated in FP64.
//
// A backward tick is three kernels in stream order, with no host round trip
// (the particle's share of the adjoint, a few hundred FP64 operations, runs on
// the device too):
//   k_adjoint_links     a warp per link entry, a lane per direction: the link
//                       terms of (x, j) are added to lam^{n+1}_i(x + c_i),
//                       i = opp(j), which only node x gathers in the next
//                       kernel, and to dmu(x); particle accumulators;
//   k_adjoint           a thread per node x, gathering ("pull" form of the
//                       transposed push):
//                         lam*_i(x) = lam^{n+1}_i(x + c_i)   unless (x + c_i, i) is a link slot
//                         lam^n(x)  = (d collide / d f)^T lam*(x) + (d rho / d f)^T mu_rho(x);
//   k_adjoint_particle  sums both kernels' accumulators in a fixed order and
//                       reverses the particle update of the tick before.
// With the link terms inside the node kernel the threads of link nodes ran up
// to 18 links x 14 dual directions in series while everyone else waited: the
// 64^3 D3Q19 backward tick took about 0.5 ms; now the node kernel is bound by
// its FP64 populations (19 gathered and 19 written per node).
#pragma once
#include "kernels.cuh"

namespace lbm {

// accumulators of the node kernel: dtau+, dtau-, dF (3)
constexpr int kAdjAcc = 5;
constexpr int kAdjBlock = 128;
// accumulators of the link kernel: particle snapshot sR, sV, sW, sE (12), dB1, dB2, torque arm mR (3)
constexpr int kAdjLinkAcc = 17;
constexpr int kAdjLinkWarps = 8;   // link entries a CTA has in hand
constexpr int kAdjLinkCtas = 296;  // two per SM; a list longer than 2,368 entries takes several rounds
constexpr int kAdjSumBlock = 32 * (kAdjAcc + kAdjLinkAcc);

// forward-mode dual number with one direction
struct DD1 {
    double v, d;
};
__device__ __forceinline__ DD1 dd(double v, double d = 0.0) { return DD1{v, d}; }
__device__ __forceinline__ DD1 operator+(DD1 a, DD1 b) { return {a.v + b.v, a.d + b.d}; }
__device__ __forceinline__ DD1 operator-(DD1 a, DD1 b) { return {a.v - b.v, a.d - b.d}; }
__device__ __forceinline__ DD1 operator-(DD1 a) { return {-a.v, -a.d}; }
__device__ __forceinline__ DD1 operator*(DD1 a, DD1 b) { return {a.v * b.v, a.d * b.v + a.v * b.d}; }
__device__ __forceinline__ DD1 operator/(DD1 a, DD1 b) {
    const double q = a.v / b.v;
    return {q, (a.d - q * b.d) / b.v};
}
__device__ __forceinline__ DD1 operator-(double b, DD1 a) { return {b - a.v, -a.d}; }
__device__ __forceinline__ DD1 operator*(double b, DD1 a) { return {b * a.v, b * a.d}; }
__device__ __forceinline__ DD1 dsqrt(DD1 a) {
    const double r = ::sqrt(a.v);
    return {r, a.d / (2.0 * r)};
}

// adjoint of the particle state carried backwards through the ticks, and the
// parameter gradients summed so far
struct AdjState {
    double R[3], v[3], w[3], e[3];
    double S[12];              // snapshot sR, sV, sW, sE
    double mR[3];
    double lamF[3], lamT[3];   // adjoints of the current tick's particle force and torque
    double dtp, dtm, dF[3], dB1, dB2;
};

// the forward state of one tick the linearisation needs
struct AdjArgs {
    const void* src;         // f^n in its storage format
    double* lam_in;          // lam^{n+1} [Q][N], f units (the link kernel adds to it)
    double* lam_out;         // lam^n [Q][N]
    double* dmu;             // [N] link terms of mu_rho, zero where none (reset by the node kernel)
    GridDesc g;
    const double* coord[3];
    const ParticleDev* part;  // the particle at tick n (one particle)
    const int2* ivl;
    const int2* links;          // its link entries (cell, direction mask)
    const unsigned char* wall;  // wall nodes (null: no walls)
    const double* uw;           // wall velocity [d][N] (null: static walls)
    double rho0, inv_scale;  // stored g' = S (f/w - rho0)
    double dt, tau_p, tau_m;  // tau_m unused for BGK
    double F[3];
    int guo, incompressible;
    double rho_inc;
    double coeff;             // dx^d / dt
    AdjState* st;
    double* partial;          // [kAdjAcc][CTAs of the node kernel]
    double* lpartial;         // [kAdjLinkAcc][CTAs of the link kernel]
    long long nblocks, nlblocks;
    // k_adjoint_particle: reverse the particle update of tick `n` (-1: none)
    const ParticleDev* rec;   // [ticks + 1] the particle after each tick
    long long n;
    long long window_begin, window_end;
    double dir[3];
    int observe_force;
    int finish;               // sum the accumulators of the two kernels before
};

// Link terms of one particle: a warp per link entry (fluid node x), lane j the
// direction j.  Lane j loads f_j, rho and u come from a butterfly over the
// lanes, and lane opp(j)'s f from a shuffle, so f*_i(x) of the lane's link is
// formed without the other directions.  For a link (x, j), i = opp(j), the
// term that multiplies lam*_i is added to lam_in at (i, x + c_i): node x is the
// only reader of that value, so the node kernel gathers it with the rest.
// Where x + c_i is also a wall node (its gathered value is void there) the
// term replaces the value.  The slip velocity is reversed in closed form.
template <class L, int ST, bool TRT>
__global__ void __launch_bounds__(32 * kAdjLinkWarps) k_adjoint_links(const AdjArgs a) {
    using SS = Store<ST>;
    using T = typename SS::T;
    constexpr int Q = L::Q, D = L::D;
    static_assert(Q <= 32, "one lane per direction");
    __shared__ double s_red[kAdjLinkWarps][kAdjLinkAcc];
    __shared__ int s_lat[4][Q];
    __shared__ double s_w[Q];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const ParticleDev& P = *a.part;
    const int nl = P.nlinks;
    for (int j = threadIdx.x; j < Q; j += blockDim.x) {
        s_lat[0][j] = L::cx(j);
        s_lat[1][j] = L::cy(j);
        s_lat[2][j] = L::cz(j);
        s_lat[3][j] = L::opp(j);
        s_w[j] = L::w(j);
    }
    __syncthreads();
    double acc[kAdjLinkAcc];
    for (int k = 0; k < kAdjLinkAcc; ++k) acc[k] = 0.0;
    for (int e = blockIdx.x * kAdjLinkWarps + warp; e < nl; e += gridDim.x * kAdjLinkWarps) {
        const int2 ent = a.links[P.link_off + e];
        const long long N = a.g.N;
        const int cell = ent.x, nx = a.g.n[0], ny = a.g.n[1], nz = a.g.n[2];
        const bool wx = a.wall && a.wall[cell];  // a wall node: everything it streams is discarded
        const int j = lane < Q ? lane : 0;
        const int i = s_lat[3][j];
        const int cj[3] = {s_lat[0][j], s_lat[1][j], s_lat[2][j]};
        const double w = s_w[j];
        double f = 0.0;
        if (lane < Q)
            f = w * ((double)SS::dec(static_cast<const T*>(a.src)[(long long)j * N + cell], typename SS::R(1)) *
                         a.inv_scale + a.rho0);
        double rho = f, J[3] = {f * cj[0], f * cj[1], f * cj[2]};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            rho += __shfl_xor_sync(0xffffffffu, rho, o);
            for (int k = 0; k < D; ++k) J[k] += __shfl_xor_sync(0xffffffffu, J[k], o);
        }
        const double fo = __shfl_sync(0xffffffffu, f, i);  // f_i
        double gmu = 0.0;
        if (lane < Q && !wx && ((unsigned)ent.y >> j & 1u)) {
            double u[3] = {0, 0, 0}, uu = 0.0, uc = 0.0, cF = 0.0, uF = 0.0;
            if (rho != 0.0)
                for (int k = 0; k < D; ++k) u[k] = (J[k] + (a.guo ? 0.5 * a.dt * a.F[k] : 0.0)) / rho;
            for (int k = 0; k < D; ++k) {
                uu += u[k] * u[k];
                uc -= u[k] * cj[k];  // u.c_i
                cF -= a.F[k] * cj[k];
                uF += u[k] * a.F[k];
            }
            // f*_i = collide(f)_i (collisionStep + guoForcingTerm, fluids.jl:58-127)
            const double m = a.incompressible ? a.rho_inc : rho;
            const double ev = w * (rho + m * (4.5 * uc * uc - 1.5 * uu)), od = w * m * 3.0 * uc;
            double fs;
            if (TRT) {
                fs = fo - a.dt / a.tau_p * (0.5 * (fo + f) - ev) - a.dt / a.tau_m * (0.5 * (fo - f) - od);
                if (a.guo)
                    fs += w * a.dt * ((1.0 - a.dt / (2.0 * a.tau_p)) * (-3.0 * uF + 9.0 * uc * cF) +
                                      (1.0 - a.dt / (2.0 * a.tau_m)) * 3.0 * cF);
            } else {
                fs = fo - a.dt / a.tau_p * (fo - ev - od);
                if (a.guo) fs += w * a.dt * (1.0 - a.dt / (2.0 * a.tau_p)) * (3.0 * (cF - uF) + 9.0 * uc * cF);
            }
            const int x = cell % nx, y = (cell / nx) % ny, z = cell / (nx * ny);
            const int sx = wrap_idx(x - cj[0], nx), sy = wrap_idx(y - cj[1], ny), sz = wrap_idx(z - cj[2], nz);
            const long long sc = sx + (long long)nx * (sy + (long long)ny * sz);  // source x - c_j
            const bool wlink = a.wall && a.wall[sc];
            const double lj = a.lam_in[(long long)j * N + cell];
            const double w6 = 6.0 * w;
            double cw = 0.0;  // moving wall term (fluids.jl:167-174)
            if (wlink && a.uw)
                for (int k = 0; k < D; ++k) cw += cj[k] * a.uw[(long long)k * N + sc];
            // slip velocity at the source node (slip_velocity), kept for its reverse
            const double xr[3] = {a.coord[0][sx] - P.sR[0], a.coord[1][sy] - P.sR[1],
                                  D == 3 ? a.coord[2][sz] - P.sR[2] : 0.0};
            double up[3];
            if (D == 2) {
                up[0] = P.sV[0] - P.sW[0] * xr[1];
                up[1] = P.sV[1] + P.sW[0] * xr[0];
                up[2] = 0.0;
            } else {
                up[0] = P.sV[0] + P.sW[1] * xr[2] - P.sW[2] * xr[1];
                up[1] = P.sV[1] - P.sW[0] * xr[2] + P.sW[2] * xr[0];
                up[2] = P.sV[2] + P.sW[0] * xr[1] - P.sW[1] * xr[0];
            }
            double ur[3] = {0, 0, 0}, inv = 1.0, edr = 0.0, first = 0.0, nrm = 1.0;
            const bool slip = P.kind != 0;
            if (slip) {
                nrm = sqrt(xr[0] * xr[0] + xr[1] * xr[1] + xr[2] * xr[2]);
                inv = nrm == 0.0 ? 1.0 : 1.0 / nrm;
                for (int k = 0; k < D; ++k) {
                    ur[k] = inv * xr[k];
                    edr += ur[k] * P.sE[k];
                }
                first = P.B1 + P.B2 * edr;
                for (int k = 0; k < D; ++k) up[k] += first * (edr * ur[k] - P.sE[k]);
            }
            const double cu = cj[0] * up[0] + cj[1] * up[1] + cj[2] * up[2] + cw;  // Ladd and wall terms
            const double s = 2.0 * fs + w6 * rho * cu;                              // f*_i + f^{n+1}_j
            double lsi = lj, gup = lj;  // lam*_i, and lam_up = gup w6 rho c_j; mu_rho gets gup w6 cu
            if (P.coupleF || P.recordF) {
                const double t = -a.coeff * (a.st->lamF[0] * cj[0] + a.st->lamF[1] * cj[1] + a.st->lamF[2] * cj[2]);
                lsi += 2.0 * t;
                gup += t;
            }
            if (P.coupleT) {
                const double r[3] = {a.coord[0][x] - P.mR[0], a.coord[1][y] - P.mR[1],
                                     D == 3 ? a.coord[2][z] - P.mR[2] : 0.0};
                const double* lT = a.st->lamT;
                double tq;  // lam_T . (r x c_i), c_i = -c_j; the arm r is x - mR
                if (D == 2) {
                    tq = -lT[0] * (r[0] * cj[1] - r[1] * cj[0]);
                    acc[14] += a.coeff * s * lT[0] * cj[1];
                    acc[15] -= a.coeff * s * lT[0] * cj[0];
                } else {
                    tq = -(lT[0] * (r[1] * cj[2] - r[2] * cj[1]) + lT[1] * (r[2] * cj[0] - r[0] * cj[2]) +
                           lT[2] * (r[0] * cj[1] - r[1] * cj[0]));
                    // d/dr lam_T.(r x c) = c x lam_T
                    acc[14] += a.coeff * s * (cj[1] * lT[2] - cj[2] * lT[1]);
                    acc[15] += a.coeff * s * (cj[2] * lT[0] - cj[0] * lT[2]);
                    acc[16] += a.coeff * s * (cj[0] * lT[1] - cj[1] * lT[0]);
                }
                lsi += 2.0 * a.coeff * tq;
                gup += a.coeff * tq;
            }
            double* lp = a.lam_in + (long long)i * N + sc;
            *lp = wlink ? lsi : *lp + lsi;
            gmu = gup * w6 * cu;
            gup *= w6 * rho;
            const double lup[3] = {gup * cj[0], gup * cj[1], gup * cj[2]};
            // reverse of the slip velocity: snapshot (sR, sV, sW, sE), B1, B2
            double gx[3] = {0, 0, 0};
            for (int k = 0; k < D; ++k) acc[3 + k] += lup[k];
            if (D == 2) {
                acc[6] += lup[1] * xr[0] - lup[0] * xr[1];
                gx[0] += lup[1] * P.sW[0];
                gx[1] -= lup[0] * P.sW[0];
            } else {
                acc[6] += xr[1] * lup[2] - xr[2] * lup[1];
                acc[7] += xr[2] * lup[0] - xr[0] * lup[2];
                acc[8] += xr[0] * lup[1] - xr[1] * lup[0];
                gx[0] += lup[1] * P.sW[2] - lup[2] * P.sW[1];
                gx[1] += lup[2] * P.sW[0] - lup[0] * P.sW[2];
                gx[2] += lup[0] * P.sW[1] - lup[1] * P.sW[0];
            }
            if (slip) {
                double gfirst = 0.0, lur = 0.0;
                for (int k = 0; k < D; ++k) {
                    gfirst += lup[k] * (edr * ur[k] - P.sE[k]);
                    lur += lup[k] * ur[k];
                }
                const double gedr = first * lur + P.B2 * gfirst;
                double gur[3] = {0, 0, 0}, dot = 0.0;
                for (int k = 0; k < D; ++k) {
                    gur[k] = first * edr * lup[k] + gedr * P.sE[k];
                    acc[9 + k] += gedr * ur[k] - first * lup[k];
                    dot += gur[k] * ur[k];
                }
                if (nrm == 0.0) dot = 0.0;
                for (int k = 0; k < D; ++k) gx[k] += inv * (gur[k] - dot * ur[k]);
                acc[12] += gfirst;
                acc[13] += gfirst * edr;
            }
            for (int k = 0; k < D; ++k) acc[k] -= gx[k];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) gmu += __shfl_xor_sync(0xffffffffu, gmu, o);
        if (lane == 0 && gmu != 0.0) a.dmu[cell] = gmu;
    }
#pragma unroll
    for (int k = 0; k < kAdjLinkAcc; ++k) {
        double v = acc[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) s_red[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < kAdjLinkAcc) {
        double v = 0.0;
        for (int q = 0; q < kAdjLinkWarps; ++q) v += s_red[q][threadIdx.x];
        a.lpartial[(long long)threadIdx.x * a.nlblocks + blockIdx.x] = v;
    }
}

// The node kernel: transposed streaming and collision.  With feq_i(rho, u), the
// Guo term G_i(u, F, tau+-) and
//   TRT  f*_i = f_i - w+ (f+_i - feq+_i) - w- (f-_i - feq-_i) + G_i,  w+- = dt / tau+-
//   BGK  the same with w- = w+ = dt / tau
// the pair (i, opp(i)) contributes through l+ = lam*_i + lam*_opp and
// l- = lam*_i - lam*_opp only, so every sum runs over the pairs:
//   lam^n_i = lam*_i - w+/2 l+ - w-/2 l- + mu_rho + mu_u.(c_i - u) / rho.
// Memory-bound by the FP64 lam values (16 of 20 bytes per direction and node
// with FP32 storage): f stays in its storage type in registers, lam* in FP64.
// What node (x, y, z) does not gather from x + c_i: bit i of *zero where slot
// (x + c_i, i) was overwritten by the fix-up (a particle's or a wall's link
// slot) or zeroed (a wall node); bit i of *copy where x + c_i is a wall node
// whose link back to x is a bounce-back copy of lam_opp(i)(x), whose moving-wall
// term is added to *mu_rho.  A wall node that is also a particle's link has its
// value from k_adjoint_links.  Only nodes inside a particle, and models with
// walls, come here; a called function keeps its registers out of the node kernel.
template <class L>
__device__ __noinline__ void adjoint_slots(const AdjArgs& a, int x, int y, int z, unsigned* zero, unsigned* copy,
                                           double* mu_rho) {
    const ParticleDev& P = *a.part;
    const int nx = a.g.n[0], ny = a.g.n[1], nz = a.g.n[2];
    const long long N = a.g.N;
    const long long cell = x + (long long)nx * (y + (long long)ny * z);
    const bool wx = a.wall && a.wall[cell], sx = solid_at(P, a.ivl, x, y, z);
#pragma unroll
    for (int i = 0; i < L::Q; ++i) {
        const int tx = wrap_idx(x + L::cx(i), nx), ty = wrap_idx(y + L::cy(i), ny), tz = wrap_idx(z + L::cz(i), nz);
        const long long t = tx + (long long)nx * (ty + (long long)ny * tz);
        const bool wt = a.wall && a.wall[t];
        const bool st = solid_at(P, a.ivl, tx, ty, tz);
        if (wx || (sx && (wt || !st))) {
            *zero |= 1u << i;
        } else if (wt && !st) {
            *copy |= 1u << i;
            if (a.uw) {
                const int j = L::opp(i);
                const int cj[3] = {L::cx(j), L::cy(j), L::cz(j)};
                double cw = 0.0;
                for (int k = 0; k < L::D; ++k) cw += cj[k] * a.uw[(long long)k * N + t];
                *mu_rho += a.lam_in[(long long)j * N + cell] * 6.0 * L::w(j) * cw;
            }
        }
    }
}

// CTAs per SM the node kernel is compiled for: as many as its registers (two
// per FP64 value of lam*, one or two per stored value) allow with a few spilled values at most
template <class L>
constexpr int adjoint_ctas_per_sm() {
    return L::Q <= 9 ? 5 : (L::Q <= 19 ? 3 : 2);
}

template <class L, int ST, bool TRT>
__global__ void __launch_bounds__(kAdjBlock, adjoint_ctas_per_sm<L>()) k_adjoint(const __grid_constant__ AdjArgs a) {
    using SS = Store<ST>;
    using T = typename SS::T;
    constexpr int Q = L::Q, D = L::D;
    __shared__ double s_red[kAdjBlock / 32][kAdjAcc];
    const long long N = a.g.N;
    const long long cell = (long long)blockIdx.x * kAdjBlock + threadIdx.x;
    const int nx = a.g.n[0], ny = a.g.n[1], nz = a.g.n[2];
    double acc[kAdjAcc];
    for (int k = 0; k < kAdjAcc; ++k) acc[k] = 0.0;
    if (cell < N) {
        const unsigned c32 = (unsigned)cell;  // N < 2^31
        const int x = (int)(c32 % nx), y = (int)((c32 / nx) % ny), z = (int)(c32 / (nx * ny));
        const int xs[3] = {x == 0 ? nx - 1 : x - 1, x, x == nx - 1 ? 0 : x + 1};
        const int ys[3] = {y == 0 ? ny - 1 : y - 1, y, y == ny - 1 ? 0 : y + 1};
        const int zs[3] = {z == 0 ? nz - 1 : z - 1, z, z == nz - 1 ? 0 : z + 1};
        const bool wx = a.wall && a.wall[cell];  // a wall node: everything it streams is discarded
        double mu_rho = a.dmu[cell];
        if (mu_rho != 0.0) a.dmu[cell] = 0.0;
        unsigned zero = 0, copy = 0;
        if (a.wall || solid_at(*a.part, a.ivl, x, y, z)) adjoint_slots<L>(a, x, y, z, &zero, &copy, &mu_rho);
        // the loads without a branch between them, so that their latencies overlap
        T raw[Q];
        double ls[Q];
        {
            const T* __restrict__ src = static_cast<const T*>(a.src);
            const double* __restrict__ lam = a.lam_in;
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                ls[i] = __ldcs(lam + i * N + (xs[L::cx(i) + 1] + nx * (ys[L::cy(i) + 1] + ny * zs[L::cz(i) + 1])));
                raw[i] = src[i * N + cell];
            }
        }
        if (zero | copy) {
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                if (copy >> i & 1u) ls[i] = a.lam_in[L::opp(i) * N + cell];
                if (zero >> i & 1u) ls[i] = 0.0;
            }
        }
        // Pair sums and differences.  The polynomials in c_i that the derivatives
        // contract lam* with are of second order, so they need only the moments
        //   m0 = sum w lam*, m1 = sum w lam* c, m2 = sum w lam* c c,
        // and the relaxation rates the products of lam* with the stored values.
        double rho = 0.0, J[3] = {0, 0, 0};  // sums of w g and w g c, then rho and j
        double m0 = 0.0, m1[3] = {0, 0, 0}, m2[6] = {0, 0, 0, 0, 0, 0};  // xx, yy, zz, xy, xz, yz
        double lf_e = 0.0, lf_o = 0.0;  // sums over pairs of w l+ g+/2 and w l- g-/2
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const int ib = L::opp(i);
            if (ib < i) continue;
            const double w = L::w(i);
            const double ga = (double)SS::dec(raw[i], typename SS::R(1));
            if (ib == i) {
                rho += w * ga;
                m0 += w * ls[i];
                lf_e += w * ls[i] * ga;
                continue;
            }
            const double gb = (double)SS::dec(raw[ib], typename SS::R(1));
            const double gp = ga + gb, gm = ga - gb;
            const double lp = ls[i] + ls[ib], lm = ls[i] - ls[ib];
            const double wlp = w * lp, wlm = w * lm, wgm = w * gm;
            rho += w * gp;
            m0 += wlp;
            lf_e += 0.5 * wlp * gp;
            lf_o += 0.5 * wlm * gm;
            const int c[3] = {L::cx(i), L::cy(i), L::cz(i)};
#pragma unroll
            for (int k = 0; k < D; ++k)
                if (c[k]) {
                    J[k] += c[k] > 0 ? wgm : -wgm;
                    m1[k] += c[k] > 0 ? wlm : -wlm;
                    m2[k] += wlp;
                }
            if (c[0] && c[1]) m2[3] += c[0] * c[1] > 0 ? wlp : -wlp;
            if (c[0] && c[2]) m2[4] += c[0] * c[2] > 0 ? wlp : -wlp;
            if (c[1] && c[2]) m2[5] += c[1] * c[2] > 0 ? wlp : -wlp;
        }
        // wall nodes hold f = 0: rho is then exactly zero (g = -rho0, and the weights' sum is kept exact)
        rho = wx ? 0.0 : rho * a.inv_scale + a.rho0;
        const bool live = rho != 0.0;  // findFluidVelocity: u = 0 where rho == 0
        const double irho = live ? 1.0 / rho : 0.0;
        double u[3] = {0, 0, 0}, uu = 0.0, uF = 0.0;
        for (int k = 0; k < D; ++k) {
            u[k] = wx ? 0.0 : (J[k] * a.inv_scale + (a.guo ? 0.5 * a.dt * a.F[k] : 0.0)) * irho;
            uu += u[k] * u[k];
            uF += u[k] * a.F[k];
        }
        const double m2u[3] = {m2[0] * u[0] + m2[3] * u[1] + m2[4] * u[2], m2[3] * u[0] + m2[1] * u[1] + m2[5] * u[2],
                               m2[4] * u[0] + m2[5] * u[1] + m2[2] * u[2]};
        const double um2u = u[0] * m2u[0] + u[1] * m2u[1] + u[2] * m2u[2];
        const double m1u = m1[0] * u[0] + m1[1] * u[1] + m1[2] * u[2];
        const double wp = a.dt / a.tau_p, wm = TRT ? a.dt / a.tau_m : wp;
        const double m = a.incompressible ? a.rho_inc : rho;  // the factor of the velocity terms
        const double even = 4.5 * um2u - 1.5 * uu * m0;
        // sum of lam* times the relaxed deviations f+ - feq+ and f- - feq-
        acc[0] = (lf_e * a.inv_scale + (a.rho0 - rho) * m0 - m * even) * wp / a.tau_p;
        const double dm = (lf_o * a.inv_scale - 3.0 * m * m1u) * wm / (TRT ? a.tau_m : a.tau_p);
        if (TRT) acc[1] = dm;
        else acc[0] += dm;
        const double g_rho = a.incompressible ? wp * m0 : wp * (m0 + even) + 3.0 * wm * m1u;
        double g_u[3] = {0, 0, 0};
        for (int k = 0; k < D; ++k) g_u[k] = m * (3.0 * wm * m1[k] + 9.0 * wp * m2u[k] - 3.0 * wp * m0 * u[k]);
        if (a.guo) {  // G_i = w dt [a+ (-3 u.F + 9 uc cF) + a- 3 cF], a+- = 1 - dt/(2 tau+-) (BGK: a- = a+)
            const double m2F[3] = {m2[0] * a.F[0] + m2[3] * a.F[1] + m2[4] * a.F[2],
                                   m2[3] * a.F[0] + m2[1] * a.F[1] + m2[5] * a.F[2],
                                   m2[4] * a.F[0] + m2[5] * a.F[1] + m2[2] * a.F[2]};
            const double ap = 1.0 - 0.5 * wp, am = 1.0 - 0.5 * wm;
            double ge = -3.0 * uF * m0, go = 0.0;
            for (int k = 0; k < D; ++k) {
                ge += 9.0 * u[k] * m2F[k];
                go += 3.0 * a.F[k] * m1[k];
                g_u[k] += a.dt * ap * (9.0 * m2F[k] - 3.0 * m0 * a.F[k]);
                acc[2 + k] = a.dt * (ap * (9.0 * m2u[k] - 3.0 * m0 * u[k]) + 3.0 * am * m1[k]);
                if (live) acc[2 + k] += g_u[k] * irho * 0.5 * a.dt;  // u = (J + dt F / 2) / rho
            }
            acc[0] += a.dt * 0.5 * wp / a.tau_p * ge;
            const double to = a.dt * 0.5 * wm / (TRT ? a.tau_m : a.tau_p) * go;
            if (TRT) acc[1] += to;
            else acc[0] += to;
        }
        double mu_u[3] = {0, 0, 0};
        if (live) {
            mu_rho += g_rho;
            for (int k = 0; k < D; ++k) {
                mu_u[k] = g_u[k] * irho;
                mu_rho -= mu_u[k] * u[k];
            }
        }
        const double hp = 0.5 * wp, hm = 0.5 * wm;
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const int ib = L::opp(i);
            if (ib < i) continue;
            if (ib == i) {
                a.lam_out[i * N + cell] = (1.0 - wp) * ls[i] + mu_rho;
                continue;
            }
            const int c[3] = {L::cx(i), L::cy(i), L::cz(i)};
            double cu = 0.0;
            for (int k = 0; k < D; ++k)
                if (c[k]) cu += c[k] > 0 ? mu_u[k] : -mu_u[k];
            // (1 - hp - hm) l_i + (hm - hp) l_opp, by the pair's sum and difference
            const double e = mu_rho - hp * (ls[i] + ls[ib]), o = cu - hm * (ls[i] - ls[ib]);
            a.lam_out[i * N + cell] = ls[i] + (e + o);
            a.lam_out[ib * N + cell] = ls[ib] + (e - o);
        }
    }
    // fixed-order reduction of the accumulators of this CTA
    for (int k = 0; k < kAdjAcc; ++k) {
        double v = acc[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < kAdjAcc) {
        double v = 0.0;
        for (int w = 0; w < kAdjBlock / 32; ++w) v += s_red[w][threadIdx.x];
        a.partial[(long long)threadIdx.x * a.nblocks + blockIdx.x] = v;
    }
}

// the swimming-direction update of moveParticles! (particles.jl:48-70:
// Rodrigues rotation by |w| dt about w, then normalised), as the particle
// kernel does it, with one forward-mode direction
template <int D>
__device__ __forceinline__ void rodrigues_dual(const DD1* e, const DD1* w, double dt, DD1* out) {
    for (int k = 0; k < 3; ++k) out[k] = e[k];
    DD1 theta;
    if (D == 2) theta = w[0].v < 0 ? -w[0] : w[0];
    else theta = dsqrt(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
    if (theta.v == 0.0) return;
    const DD1 th = dt * theta;
    double sn, cs;
    sincos(th.v, &sn, &cs);
    const DD1 ct = dd(cs, -sn * th.d), st = dd(sn, cs * th.d);
    DD1 vr[3];
    if (D == 2) {
        const DD1 k = w[0] / theta;
        vr[0] = e[0] * ct - k * e[1] * st;
        vr[1] = e[1] * ct + k * e[0] * st;
        vr[2] = dd(0.0);
    } else {
        const DD1 k[3] = {w[0] / theta, w[1] / theta, w[2] / theta};
        const DD1 cr[3] = {k[1] * e[2] - k[2] * e[1], k[2] * e[0] - k[0] * e[2], k[0] * e[1] - k[1] * e[0]};
        const DD1 kv = k[0] * e[0] + k[1] * e[1] + k[2] * e[2];
        for (int q = 0; q < 3; ++q) vr[q] = e[q] * ct + cr[q] * st + k[q] * kv * (1.0 - ct);
    }
    DD1 n2 = dd(0.0);
    for (int q = 0; q < D; ++q) n2 = n2 + vr[q] * vr[q];
    const DD1 nr = dsqrt(n2);
    for (int q = 0; q < D; ++q) out[q] = vr[q] / nr;
}

// the adjoint of the particle update of tick a.n, by one warp; P0, P1: the
// particle before and after it
template <int D>
__device__ __forceinline__ void adjoint_particle_update(const AdjArgs& a, const ParticleDev& P0, const ParticleDev& P1,
                                                        AdjState& S, int lane) {
    __syncwarp();
    const double dt = a.dt;
    // the observable reads the velocity after tick n + 1, or the force of tick n + 1
    const bool in_window = a.n + 1 >= a.window_begin && a.n + 1 <= a.window_end;
    const double K = (double)(a.window_end - a.window_begin + 1);
    if (lane == 0) {
        if (in_window && !a.observe_force)
            for (int k = 0; k < D; ++k) S.v[k] += a.dir[k] / K;
        bool moved = false, alpha = false;
        if (P0.coupleF)
            for (int k = 0; k < D; ++k) moved = moved || P1.v[k] != 0.0;
        if (P0.coupleT)
            for (int k = 0; k < (D == 2 ? 1 : 3); ++k) alpha = alpha || P1.lastT[k] * P0.inv_inertia != 0.0;
        if (moved || alpha) {  // the snapshot after the update is the updated state
            for (int k = 0; k < 3; ++k) {
                S.R[k] += S.S[k];
                S.v[k] += S.S[3 + k];
                S.w[k] += S.S[6 + k];
                S.e[k] += S.S[9 + k];
            }
            for (int k = 0; k < 12; ++k) S.S[k] = 0.0;
        }
        if (moved)  // the torque arm after the update is the new position
            for (int k = 0; k < 3; ++k) {
                S.R[k] += S.mR[k];
                S.mR[k] = 0.0;
            }
    }
    __syncwarp();
    if (P0.coupleT && P0.kind == 1) {  // e' = rot(e, w'): lane q < 6 differentiates along e_q or w_(q-3)
        DD1 e[3], w[3], o[3];
        for (int k = 0; k < 3; ++k) {
            e[k] = dd(P0.e[k], lane == k ? 1.0 : 0.0);
            w[k] = dd(P1.w[k], lane == 3 + k ? 1.0 : 0.0);
        }
        rodrigues_dual<D>(e, w, dt, o);
        double g = 0.0;
        for (int k = 0; k < D; ++k) g += S.e[k] * o[k].d;
        __syncwarp();
        if (lane < 3) S.e[lane] = g;
        else if (lane < 6) S.w[lane - 3] += g;
    }
    __syncwarp();
    if (lane == 0) {
        for (int k = 0; k < 3; ++k) S.lamF[k] = S.lamT[k] = 0.0;
        if (P0.coupleT)
            for (int k = 0; k < (D == 2 ? 1 : 3); ++k) S.lamT[k] = dt * P0.inv_inertia * S.w[k];  // w' = w + dt T / I
        if (P0.coupleF) {
            for (int k = 0; k < D; ++k) S.v[k] += dt * S.R[k];                   // R' = R + dt v'
            for (int k = 0; k < D; ++k) S.lamF[k] = dt * P0.inv_mass * S.v[k];   // v' = v + dt F / m
        }
        if (in_window && a.observe_force)
            for (int k = 0; k < D; ++k) S.lamF[k] += a.dir[k] / K;  // J += e.F / K
    }
}

// One CTA, a warp per accumulator.  First (a.finish) the sums of the two
// kernels' per-CTA accumulators, each by its warp in a fixed order; then, for
// a.n >= 0, the adjoint of the particle update of tick a.n (moveParticles!,
// particles.cuh) up to the adjoints of that tick's force and torque.  The
// records and the adjoint state are staged in shared memory, so that the
// chain does not wait for L2 at every step.
template <int D>
__global__ void __launch_bounds__(kAdjSumBlock) k_adjoint_particle(const AdjArgs a) {
    __shared__ double s_sum[kAdjAcc + kAdjLinkAcc];
    __shared__ ParticleDev s_P[2];
    __shared__ AdjState S;
    static_assert(sizeof(AdjState) % 8 == 0 && sizeof(ParticleDev) % 8 == 0, "staged in 8-byte words");
    constexpr int kWordsS = (int)(sizeof(AdjState) / 8), kWordsP = (int)(sizeof(ParticleDev) / 8);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int k = tid; k < kWordsS; k += kAdjSumBlock)
        reinterpret_cast<unsigned long long*>(&S)[k] = reinterpret_cast<const unsigned long long*>(a.st)[k];
    if (a.n >= 0)
        for (int k = tid; k < 2 * kWordsP; k += kAdjSumBlock)
            reinterpret_cast<unsigned long long*>(s_P)[k] = reinterpret_cast<const unsigned long long*>(a.rec + a.n)[k];
    if (a.finish) {
        const bool node = warp < kAdjAcc;
        const long long nb = node ? a.nblocks : a.nlblocks;
        const double* p = node ? a.partial + warp * nb : a.lpartial + (warp - kAdjAcc) * nb;
        double v = 0.0;
#pragma unroll 16
        for (long long b = lane; b < nb; b += 32) v += p[b];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) s_sum[warp] = v;
    }
    __syncthreads();
    if (warp != 0) return;
    if (a.finish && lane == 0) {
        const double* l = s_sum + kAdjAcc;
        S.dtp += s_sum[0];
        S.dtm += s_sum[1];
        for (int k = 0; k < 3; ++k) S.dF[k] += s_sum[2 + k];
        for (int k = 0; k < 12; ++k) S.S[k] += l[k];  // the snapshot that tick used
        S.dB1 += l[12];
        S.dB2 += l[13];
        for (int k = 0; k < 3; ++k) S.mR[k] += l[14 + k];
    }
    if (a.n >= 0) adjoint_particle_update<D>(a, s_P[0], s_P[1], S, lane);
    __syncwarp();
    for (int k = lane; k < kWordsS; k += 32)
        reinterpret_cast<unsigned long long*>(a.st)[k] = reinterpret_cast<const unsigned long long*>(&S)[k];
}

// d/dF of the initial populations f^0 = feq(rho, u0 - dt F / (2 rho))
// (findInitialConditions, initMethods.jl:417-438), contracted with lam^0
template <class L, int ST>
__global__ void __launch_bounds__(kAdjBlock) k_adjoint_init(const AdjArgs a) {
    using SS = Store<ST>;
    using T = typename SS::T;
    constexpr int Q = L::Q, D = L::D;
    __shared__ double s_red[kAdjBlock / 32][3];
    const long long N = a.g.N;
    const long long cell = (long long)blockIdx.x * kAdjBlock + threadIdx.x;
    double acc[3] = {0, 0, 0};
    if (cell < N && a.guo) {
        const T* __restrict__ src = static_cast<const T*>(a.src);
        double rho = 0.0, J[3] = {0, 0, 0};
        for (int i = 0; i < Q; ++i) {
            const double fi = L::w(i) * ((double)SS::dec(src[i * N + cell], typename SS::R(1)) * a.inv_scale + a.rho0);
            rho += fi;
            J[0] += fi * L::cx(i);
            J[1] += fi * L::cy(i);
            J[2] += fi * L::cz(i);
        }
        if (rho != 0.0) {
            for (int k = 0; k < D; ++k) {
                double g = 0.0;
                for (int i = 0; i < Q; ++i) {  // d feq_i / d u_k at (rho, J / rho)
                    const int c[3] = {L::cx(i), L::cy(i), L::cz(i)};
                    double uc = 0.0;
                    for (int q = 0; q < D; ++q) uc += (J[q] / rho) * c[q];
                    const double dsec = 3.0 * c[k] + 9.0 * uc * c[k] - 3.0 * (J[k] / rho);
                    const double dfeq = a.incompressible ? L::w(i) * a.rho_inc * dsec : L::w(i) * rho * dsec;
                    g += a.lam_in[i * N + cell] * dfeq;
                }
                acc[k] = g * (-0.5 * a.dt / rho);
            }
        }
    }
    for (int k = 0; k < 3; ++k) {
        double v = acc[k];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < kAdjAcc) {
        double v = 0.0;  // accumulators 2..4: dF
        if (threadIdx.x >= 2)
            for (int w = 0; w < kAdjBlock / 32; ++w) v += s_red[w][threadIdx.x - 2];
        a.partial[(long long)threadIdx.x * a.nblocks + blockIdx.x] = v;
    }
}

// A model's state to or from a stored state: the regions of one copy in one
// launch (a memcpy per region took about 25 us per 64^3 restore, most of it
// the six small ones).  Regions start 16-byte aligned on both sides.
constexpr int kCopyRegions = 7;
struct CopyArgs {
    const void* src[kCopyRegions];
    void* dst[kCopyRegions];
    size_t bytes[kCopyRegions];
};
static __global__ void __launch_bounds__(512) k_copy_regions(const __grid_constant__ CopyArgs a) {
    const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x, n = (size_t)gridDim.x * blockDim.x;
    for (int r = 0; r < kCopyRegions; ++r) {
        const size_t v = a.bytes[r] / 16;
        const uint4* s = static_cast<const uint4*>(a.src[r]);
        uint4* d = static_cast<uint4*>(a.dst[r]);
        size_t k = t;
        for (; k + 3 * n < v; k += 4 * n) {  // four loads in flight
            const uint4 q0 = s[k], q1 = s[k + n], q2 = s[k + 2 * n], q3 = s[k + 3 * n];
            d[k] = q0;
            d[k + n] = q1;
            d[k + 2 * n] = q2;
            d[k + 3 * n] = q3;
        }
        for (; k < v; k += n) d[k] = s[k];
        for (size_t b = v * 16 + t; b < a.bytes[r]; b += n)
            static_cast<char*>(a.dst[r])[b] = static_cast<const char*>(a.src[r])[b];
    }
}

}  // namespace lbm
