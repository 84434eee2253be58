// engine.cu - sm_103a kernels of the hot path and the context that runs them.
//
// Data layout in HBM (N beads of all replicas packed, replica r owning the
// contiguous range [begin_r, begin_r + n_r)):
//   pos[2]   double4_32a (x, y, z, charge), double-buffered: one step reads
//            pos[cur] and writes pos[cur^1]; y0 of the predictor-corrector IS
//            the position.
//   yh       y1..y5 as 15 SoA double arrays (coalesced per component).
//   orig     double4_32a positions of the last Verlet rebuild (skin test).
//   bonded   per-centre parameters (bond i->i+1, angle at i, dihedral with
//            second bead i) and a flag word per bead; chains are contiguous,
//            so bonded partners are i-3..i+3 and come from a shared-memory
//            tile of the block.
//   natives  CSR per bead (both directions) with an "in Go list" byte.
//   Verlet   ELL rows nl_row[k*N + i] = j | flags<<30 holding only pairs that
//            some enabled pair term keeps (Pauli r < r_excl+pad, ES r < 2D+pad
//            with q_i q_j != 0); pairs no term keeps are dropped at build time.
//   cells    per-replica grids (cell budget fixed per replica), counting sort
//            with a deterministic in-cell order.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <stdexcept>

#include "device.cuh"
#include "engine.h"
#include "qa.cuh"

namespace xmdg {

std::string &last_error() {
    static thread_local std::string e;
    return e;
}

#define CK(call)                                                                     \
    do {                                                                             \
        cudaError_t e_ = (call);                                                     \
        if (e_ != cudaSuccess)                                                       \
            throw std::runtime_error(std::string("CUDA error ") + cudaGetErrorString(e_) + \
                                     " at " #call);                                  \
    } while (0)

constexpr int NL_MASK = 0x1FFFFFFF;
constexpr int NL_PID = 1 << 29;
constexpr int NL_PAULI = 1 << 30;
constexpr int NL_ES = (int)(1u << 31);

enum : int { ST_CAPACITY = 1, ST_NONFINITE = 2 };

// ---- generator jump-ahead (host) ---------------------------------------------
using GF2 = std::array<uint64_t, 64>;
static uint64_t xs_step(uint64_t s) {
    s ^= s >> 11;
    s ^= s << 31;
    s ^= s >> 18;
    return s;
}
static uint64_t gf2_apply_h(const GF2 &m, uint64_t x) {
    uint64_t y = 0;
    for (int k = 0; k < 64; ++k)
        if ((x >> k) & 1) y ^= m[k];
    return y;
}
static GF2 gf2_mul(const GF2 &a, const GF2 &b) {
    GF2 c;
    for (int k = 0; k < 64; ++k) c[k] = gf2_apply_h(a, b[k]);
    return c;
}
// matrix of `draws` generator steps
static GF2 gf2_jump(uint64_t draws) {
    GF2 m, r;
    for (int k = 0; k < 64; ++k) {
        m[k] = xs_step(1ull << k);
        r[k] = 1ull << k;
    }
    while (draws) {
        if (draws & 1) r = gf2_mul(m, r);
        m = gf2_mul(m, m);
        draws >>= 1;
    }
    return r;
}

uint64_t rng_jump(uint64_t state, uint64_t n_draws) { return gf2_apply_h(gf2_jump(n_draws), state); }

// ---- exact squared-distance thresholds (host) ---------------------------------
// The list tests of the reference take a square root (and a reciprocal) of
// the squared distance and compare.  Both are correctly rounded and monotone
// in IEEE FP64, so each test equals s < S for one threshold S on the squared
// distance, found here by stepping through adjacent doubles; the builds then
// compare squared distances (no FP64 square root or division per pair).
// smallest s with RN(sqrt(s)) >= T: sqrt(s) < T <=> s < sq_below(T)
static double sq_below(double T) {
    if (!(T > 0.0)) return 0.0;
    double s = T * T;
    while (s > 0.0 && std::sqrt(s) >= T) s = std::nextafter(s, 0.0);
    while (std::sqrt(s) < T) s = std::nextafter(s, INFINITY);
    return s;
}
// smallest x with RN(1/x) <= v: 1/x > v <=> x < inv_above(v)
static double inv_above(double v) {
    if (!(v > 0.0)) return INFINITY;
    double x = 1.0 / v;
    while (x > 0.0 && 1.0 / x <= v) x = std::nextafter(x, 0.0);
    while (1.0 / x > v) x = std::nextafter(x, INFINITY);
    return x;
}

// ---- device helpers -----------------------------------------------------------
// maximum over the warp of non-negative doubles, compared as their bit
// patterns (the same order) on the integer pipe
__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long v) {
    for (int o = 16; o; o >>= 1) {
        const unsigned long long u = __shfl_xor_sync(0xffffffffu, v, o);
        v = u > v ? u : v;
    }
    return v;
}

// finiteness from the exponent bits (integer pipe)
__device__ __forceinline__ bool finite_bits(double x) {
    return ((unsigned long long)__double_as_longlong(x) & 0x7ff0000000000000ull) != 0x7ff0000000000000ull;
}

// ---- external forces ---------------------------------------------------------------
// Wall forces on one bead at its wrapped position rw.  ljw points at the bead's state for the first LJ attractive
// wall (stride N); step = true advances the pair states.
struct WallOut { double fx, fy, fz, vs, vl; };
__device__ __forceinline__ WallOut wall_forces(const double *wall, LjWallState *ljw, size_t N, V3<double> rw,
                                            double tt, bool step, int n_solid, int n_ljw, double solid_eps,
                                            double solid_cutoff, double min_dist, double factor, double cycle,
                                            double cycle_inv, double depth) {
    WallOut o{0.0, 0.0, 0.0, 0.0, 0.0};
    for (int w = 0; w < n_solid; ++w) {
        // eval_solid_wall_forces::iter (walls/solid.cpp:12-27): V = eps /
        // (9 x^9) inside the cutoff, its force -dV/dx along the normal [the
        // shipped dV_dx = V (-9 x), added along +normal]
        const double *pl = wall + 6 * w;
        const double x = pl[3] * (rw.x - pl[0]) + pl[4] * (rw.y - pl[1]) + pl[5] * (rw.z - pl[2]);
        if (x < solid_cutoff) {
            const double x3 = x * x * x, V_ = solid_eps / (9.0 * (x3 * x3 * x3));
            const double mdV = 9.0 * V_ / x;   // -dV/dx
            o.vs += V_;
            o.fx += mdV * pl[3]; o.fy += mdV * pl[4]; o.fz += mdV * pl[5];
        }
    }
    for (int w = 0; w < n_ljw; ++w) {
        // eval_lj_attr_wall_forces::loop (walls/lj_attr.cpp:5-43)
        const double *pl = wall + 6 * (XMD_MAX_WALLS + w);
        LjWallState st = ljw[(size_t)w * N];
        if (st.status == 0) {
            const double x = pl[3] * (rw.x - pl[0]) + pl[4] * (rw.y - pl[1]) + pl[5] * (rw.z - pl[2]);
            if (step && fabs(x) < min_dist) {
                st.status = 1;
                st.jx = rw.x - pl[3] * x; st.jy = rw.y - pl[4] * x; st.jz = rw.z - pl[5] * x;
                st.ref_t = tt;
                ljw[(size_t)w * N] = st;
            }
        } else {
            double sat = fmin(tt - st.ref_t, cycle) * cycle_inv;
            if (st.status == 2) sat = 1.0 - sat;
            const V3<double> r12{st.jx - rw.x, st.jy - rw.y, st.jz - rw.z};
            const double r12_rn = 1.0 / norm(r12);
            double V_, dV;
            lj_eval<double>(depth, min_dist, r12_rn, &V_, &dV);
            o.vl += V_ * sat;
            const double f = sat * dV;
            o.fx += f * (r12_rn * r12.x); o.fy += f * (r12_rn * r12.y); o.fz += f * (r12_rn * r12.z);
            if (step) {
                if (st.status == 1 && sat == 1.0) {
                    if (factor * min_dist * r12_rn < 1.0) { st.status = 2; st.ref_t = tt; }
                } else if (st.status == 2 && sat == 0.0) {
                    st.status = 0;
                }
                ljw[(size_t)w * N] = st;
            }
        }
    }
    return o;
}

// External forces of the step, one thread per bead, before the step kernel
// (contexts with AFM tips or walls only): the AFM pulls and the wall forces
// at the step's positions, into fext; MODE 0 adds their energies, MODE 1
// advances the LJ attractive wall pairs.  Kept out of the step kernel, whose
// registers they would raise for every context.
template <int MODE>
__global__ void __launch_bounds__(256) k_ext(Dev d, TermP p, int cur) {
    step_order();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.N || (MODE == 1 && d.gate[0])) return;
    double *fo = d.fext + 3 * (size_t)i;
    fo[0] = fo[1] = fo[2] = 0.0;
    const int r = d.rep_of[i];
    if (r < 0) return;
    if (MODE == 1 && d.rep[r].steps_left == 0) return;
    const double4_32a pi = d.pos[cur][i];
    const double tt = d.rep[r].t;
    V3<double> f{0.0, 0.0, 0.0};
    if (d.rep[r].afm) {
        const uint32_t fl_i = d.bflags[i];
        if (fl_i & BF_AFM) {
            const AfmTip tp = d.afm[fl_i >> BF_AFM_SHIFT];
            if (tp.has_vel && p.on[XMD_TERM_VEL_AFM]) {
                // eval_velocity_afm_forces::iter (velocity_afm.cpp): a
                // harmonic(H1, H2, 0) spring to the tip at orig + t vel
                const V3<double> ra{tp.ox + tt * tp.vx - pi.x, tp.oy + tt * tp.vy - pi.y, tp.oz + tt * tp.vz - pi.z};
                const double rn = norm(ra), rrn = 1.0 / rn;
                const double dr2 = rn * rn;
                double dV = rn * (p.vel_afm_H1 + 2.0 * p.vel_afm_H2 * dr2);
                dV = clampv<double>(dV, -1.0e3, 1.0e3);
                // the spring at rest pulls nothing (0 * inf in the shipped code)
                if (rn > 0.0) f = f + dV * (rrn * ra);
            }
            if (p.on[XMD_TERM_FORCE_AFM]) f = f + V3<double>{tp.fx, tp.fy, tp.fz};
        }
    }
    if (p.n_solid | p.n_ljw) {
        // walls act on the position wrapped into the box (box::wrap)
        const BoxD bx = d.rep[r].box;
        V3<double> rw{pi.x, pi.y, pi.z};
        rw.x -= bx.cell[0] * rint(rw.x * bx.cell_inv[0]);
        rw.y -= bx.cell[1] * rint(rw.y * bx.cell_inv[1]);
        rw.z -= bx.cell[2] * rint(rw.z * bx.cell_inv[2]);
        const WallOut wo = wall_forces(d.wall, d.ljw + i, (size_t)d.N, rw, tt, MODE == 1, p.n_solid, p.n_ljw,
                                       p.solid_eps, p.solid_cutoff, p.ljw_min_dist, p.ljw_factor, p.ljw_cycle,
                                       p.ljw_cycle_inv, p.ljw_depth);
        f = f + V3<double>{wo.fx, wo.fy, wo.fz};
        if (MODE == 0) {
            if (p.n_solid) atomicAdd(&d.Vrep[r * XMD_NUM_TERMS + XMD_TERM_SOLID_WALL], wo.vs);
            if (p.n_ljw) atomicAdd(&d.Vrep[r * XMD_NUM_TERMS + XMD_TERM_LJ_WALL], wo.vl);
        }
    }
    fo[0] = f.x; fo[1] = f.y; fo[2] = f.z;
}

// ---- pseudo-improper dihedral potential: eval_pid_forces::iter
// (pid/eval_forces.cpp:14-141), bundles from update_pid_bundles
// (pid/bundle.cpp:6-29) ------------------------------------------------------------
// Evaluated in FP64 on both paths with every operation rounded on its own
// (DN), in the operation order of the oracle's restatement; the forces are
// the energy's gradient (the shipped kernel leaves one side's derivatives
// unset and scales the others by 1/|m|, 1/|n| for 1/|m|^2, 1/|n|^2).
using D3N = V3<DN>;
constexpr double PID_PI = 3.14159265358979323846;

// lambda_func (pid/lambda.h:29-56): inside the support, value and derivative
__device__ __forceinline__ bool pid_supp(DN alpha, DN psi0, DN psi) { return dn_fabs(alpha * (psi - psi0)) < DN(PID_PI); }
__device__ __forceinline__ void pid_lam(int version, DN alpha, DN psi0, DN psi, DN *val, DN *deriv) {
    const DN sv = alpha * (psi - psi0);
    if (version == 0) {
        *val = DN(0.5) * dn_cos(sv) + DN(0.5);
        *deriv = (DN(-0.5) * alpha) * sin(sv);
    } else {
        const DN t = dn_fabs(sv / DN(PID_PI));
        const DN x_inv = DN(1.0) / (DN(2.0) * t * t - DN(2.0) * t - DN(1.0));
        *val = (t * t - DN(2.0) * t + DN(1.0)) * x_inv;
        DN dv = (DN(2.0) * (t - DN(1.0)) * (t - DN(2.0))) * x_inv * x_inv * alpha / DN(PID_PI);
        if (sv < DN(0.0)) dv = -dv;
        *deriv = dv;
    }
}
__device__ __forceinline__ D3N d3n(double4_32a p) { return D3N{DN(p.x), DN(p.y), DN(p.z)}; }
__device__ __forceinline__ D3N pid_ruv(const BoxD &b, D3N u, D3N w) {
    D3N d = w - u;
    d.x = d.x - DN(b.cell[0]) * dn_rint(d.x * DN(b.cell_inv[0]));
    d.y = d.y - DN(b.cell[1]) * dn_rint(d.y * DN(b.cell_inv[1]));
    d.z = d.z - DN(b.cell[2]) * dn_rint(d.z * DN(b.cell_inv[2]));
    return d;
}
// one side: psi of (previous, bead, next; partner) and its derivatives along
// the four beads (d1 previous, d2 bead, d3 next, d4 partner)
__device__ __forceinline__ DN pid_psi(const BoxD &b, D3N r1_, D3N r2_, D3N r3_, D3N r4_, D3N *d1, D3N *d2, D3N *d3,
                                      D3N *d4) {
    const D3N r24 = pid_ruv(b, r2_, r4_);
    const D3N r12 = r2_ - r1_, r23 = r3_ - r2_, r13 = r3_ - r1_;
    const D3N r14 = r12 + r24;
    const D3N rij = -r23, rkj = -r13, rkl = -r14;
    const D3N rm = cross(r23, r12), rn = cross(r13, r14);
    const DN rm_rn = ninv(rm), rn_rn = ninv(rn), rkj_n = norm(rkj);
    const D3N gi = (rkj_n * rm_rn * rm_rn) * rm;
    const D3N gl = -((rkj_n * rn_rn * rn_rn) * rn);
    const DN a = dot(rij, rkj) / (rkj_n * rkj_n), bb = dot(rkl, rkj) / (rkj_n * rkj_n);
    *d1 = (bb - DN(1.0)) * gl - a * gi;
    *d2 = gi;
    *d3 = (a - DN(1.0)) * gi - bb * gl;
    *d4 = gl;
    DN psi = DN(acos((dot(rm, rn) * rm_rn * rn_rn).v));
    if (dot(rij, rn) < DN(0.0)) psi = -psi;
    return psi;
}

// One thread per bead: the bundles (i, j) of its Verlet row (both beads with
// their chain neighbours, r < PID cutoff + pad at the rebuild), each taken in
// its canonical order (i1, i2) = (min, max).  The bead keeps the forces of
// its side: on itself, its previous and its next bead, into pid_f; the step
// kernel adds to a bead its own part and its neighbours' parts for it.
// MODE 0 adds the energy of the bundles with i < j.
template <int MODE>
__global__ void __launch_bounds__(128) k_pid(Dev d, TermP p, int cur) {
    step_order();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.N || (MODE == 1 && d.gate[0])) return;
    const size_t N = d.N;
    double *Fs = d.pid_f, *Fp = d.pid_f + 3 * N, *Fn = d.pid_f + 6 * N;
    D3N fs{DN(0.0), DN(0.0), DN(0.0)}, fp = fs, fn = fs;
    double Vsum = 0.0;
    const int r = d.rep_of[i];
    const bool both = (d.bflags[i] & (BF_PREV | BF_NEXT)) == (BF_PREV | BF_NEXT);
    if (r >= 0 && both && !(MODE == 1 && d.rep[r].steps_left == 0)) {
        const double4_32a *pos = d.pos[cur];
        const BoxD bx = d.rep[r].box;
        const int cnt = d.nl_cnt[i];
        const DN bbq[2][4] = {{DN(p.pid_bbp[0]), DN(p.pid_bbp[1]), DN(p.pid_bbp[2]), DN(p.pid_bbp[3])},
                              {DN(p.pid_bbm[0]), DN(p.pid_bbm[1]), DN(p.pid_bbm[2]), DN(p.pid_bbm[3])}};
        const DN ssa = DN(p.pid_ss[0]), ssp = DN(p.pid_ss[1]);
        for (int k = 0; k < cnt; ++k) {
            const int e = d.nl_row[(size_t)k * N + i];
            if (!(e & NL_PID)) continue;
            const int j = e & NL_MASK;
            const int i1 = min(i, j), i2 = max(i, j);
            const D3N r1p = d3n(pos[i1 - 1]), r1 = d3n(pos[i1]), r1n = d3n(pos[i1 + 1]);
            const D3N r2p = d3n(pos[i2 - 1]), r2 = d3n(pos[i2]), r2n = d3n(pos[i2 + 1]);
            D3N a1p, a1, a1n, a2, b2p, b2, b2n, b1;
            const DN psi1 = pid_psi(bx, r1p, r1, r1n, r2, &a1p, &a1, &a1n, &a2);
            const DN psi2 = pid_psi(bx, r2p, r2, r2n, r1, &b2p, &b2, &b2n, &b1);
            const D3N r12 = pid_ruv(bx, r1, r2);
            const DN r12_n = norm(r12), r12_rn = DN(1.0) / r12_n;
            DN A(0.0), B(0.0), C(0.0), V(0.0);
            for (int q = 0; q < 2; ++q) {
                if (pid_supp(bbq[q][0], bbq[q][1], psi1) && pid_supp(bbq[q][0], bbq[q][1], psi2)) {
                    DN lam1, g1, lam2, g2, lV, ldV;
                    pid_lam(p.pid_lambda, bbq[q][0], bbq[q][1], psi1, &lam1, &g1);
                    pid_lam(p.pid_lambda, bbq[q][0], bbq[q][1], psi2, &lam2, &g2);
                    lj_eval<DN>(bbq[q][3], bbq[q][2], r12_rn, &lV, &ldV);
                    V = V + lam1 * lam2 * lV;
                    A = A + g1 * lam2 * lV;
                    B = B + g2 * lam1 * lV;
                    C = C + lam1 * lam2 * ldV;
                }
            }
            if (pid_supp(ssa, ssp, psi1) && pid_supp(ssa, ssp, psi2)) {
                // ss_ljs[type], type = atype1 * NUM_AA + atype2 (bundle.cpp:20-22)
                const int ty = (int)d.atype[i1] * XMD_NUM_AA + (int)d.atype[i2];
                DN lam1, g1, lam2, g2, lV, ldV;
                pid_lam(p.pid_lambda, ssa, ssp, psi1, &lam1, &g1);
                pid_lam(p.pid_lambda, ssa, ssp, psi2, &lam2, &g2);
                sink_lj_eval<DN>(DN(d.pid_sd[ty]), DN(d.pid_smin[ty]), DN(d.pid_smax[ty]), r12_n, r12_rn, &lV, &ldV);
                V = V + lam1 * lam2 * lV;
                A = A + g1 * lam2 * lV;
                B = B + g2 * lam1 * lV;
                C = C + lam1 * lam2 * ldV;
            }
            const D3N u = r12_rn * r12;
            if (i == i1) {
                fp = fp - A * a1p;
                fs = fs - ((A * a1 + B * b1) - C * u);
                fn = fn - A * a1n;
                if (MODE == 0) Vsum += V.v;
            } else {
                fp = fp - B * b2p;
                fs = fs - ((A * a2 + B * b2) + C * u);
                fn = fn - B * b2n;
            }
        }
    }
    Fs[3 * i] = fs.x.v; Fs[3 * i + 1] = fs.y.v; Fs[3 * i + 2] = fs.z.v;
    Fp[3 * i] = fp.x.v; Fp[3 * i + 1] = fp.y.v; Fp[3 * i + 2] = fp.z.v;
    Fn[3 * i] = fn.x.v; Fn[3 * i + 1] = fn.y.v; Fn[3 * i + 2] = fn.z.v;
    if (MODE == 0 && Vsum != 0.0) atomicAdd(&d.Vrep[r * XMD_NUM_TERMS + XMD_TERM_PID], Vsum);
}

}  // namespace xmdg
#include "step.cuh"
namespace xmdg {

// FP64 positions as float-float parts (mixed path).  The step kernel keeps
// them up to date; the host may have placed, restored or uploaded positions
// since, so every call that steps or evaluates starts with this pass (32 B
// read, 32 B written per bead).
__global__ void __launch_bounds__(256) k_split(Dev d, int cur) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.N) return;
    const double4_32a q = d.pos[cur][i];
    const P2 s = split_p(q);
    d.spl[cur][2 * (size_t)i] = make_float4(s.x.h, s.y.h, s.z.h, narrow_f(q.w));
    d.spl[cur][2 * (size_t)i + 1] = make_float4(s.x.l, s.y.l, s.z.l, 0.0f);
}

// ---- skin decision (nl::verify, verify.cpp:4-23) --------------------------------
// setc 1: also set the conditional handle of the graph's rebuild IF node;
// setc 2: count the step in the gate and halt the graph when a replica is
// flagged or the budget of steps is spent
enum : int { CHECK_PLAIN = 0, CHECK_COND = 1, CHECK_GATE = 2 };
template <int SETC>
__device__ __forceinline__ void nl_check_block(const Dev &d, int advance, double dt, cudaGraphConditionalHandle h) {
    __shared__ int any_s, nwork_s;
    if (threadIdx.x == 0) any_s = nwork_s = 0;
    __syncthreads();
    int any = 0;
    for (int r = threadIdx.x; r < d.R; r += blockDim.x) {
        RepDev &rp = d.rep[r];
        // every field the decision reads, loaded at once (one round trip)
        const int active = rp.active, fault = rp.fault, first = rp.first, tile = rp.tile;
        const int nchunk = rp.nchunk, chunk_off = rp.chunk_off;
        long long left = rp.steps_left;
        const unsigned long long mdb = rp.maxdisp;
        const double pad = rp.pad, tr = rp.t;
        if (!active) continue;
        if (fault) {   // frozen: no further step, no list
            rp.steps_left = 0;
            rp.rebuild = 0;
            continue;
        }
        if (advance && left == 0) {           // took no step (k_force kept it)
            rp.rebuild = 0;
            continue;
        }
        if (advance) {
            rp.t = tr + dt;                   // *t = (*true_t += dt)
            if (left > 0) rp.steps_left = --left;
        }
        const double md = __dsqrt_rn(__longlong_as_double((long long)mdb));
        rp.maxdisp = 0ull;
        int rb = first || (2.0 * md + 0.0 > pad);
        if (advance && left == 0 && !first) rb = 0;   // no further step uses a list
        rp.rebuild = rb;
        any |= rb;
        if (rb && !tile) {   // the cell build's bounding box starts empty
#pragma unroll
            for (int a = 0; a < 3; ++a) { rp.lo_key[a] = 0xffffffffu; rp.hi_key[a] = 0u; }
        }
        // the tile build's work list: every chunk of the flagged replicas
        // (order is free: each chunk writes its own rows)
        if (rb && tile) {
            const int at = atomicAdd(&nwork_s, nchunk);
            for (int c = 0; c < nchunk; ++c) d.work[at + c] = chunk_off + c;
        }
    }
    if (any) atomicOr(&any_s, 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        *d.any_rebuild = any_s;
        *d.nwork = nwork_s;
        if constexpr (SETC == CHECK_COND) cudaGraphSetConditional(h, any_s ? 1u : 0u);
        if constexpr (SETC == CHECK_GATE) {
            const int done = d.gate[1] + 1;
            d.gate[1] = done;
            if (any_s || done >= d.gate[2]) d.gate[0] = 1;
        }
    }
}
__global__ void k_nl_check(Dev d, int advance, double dt, cudaGraphConditionalHandle h, int setc) {
    step_order();
    if (setc == CHECK_GATE && d.gate[0]) return;
    if (setc == CHECK_COND) nl_check_block<CHECK_COND>(d, advance, dt, h);
    else if (setc == CHECK_GATE) nl_check_block<CHECK_GATE>(d, advance, dt, h);
    else nl_check_block<CHECK_PLAIN>(d, advance, dt, h);
}

// The quasi-adiabatic re-freeing (one block per replica).  With `check` (the
// gated graph steps) the last block to finish also takes the step's skin
// decision, which otherwise is a launch of its own.
__global__ void __launch_bounds__(1024) k_qa_refree(Dev d, double dt, int check) {
    step_order();
    if (d.gate[0]) return;
    qa_refree_block(d);
    if (!check) return;
    __shared__ int last_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last_s = atomicAdd(&d.ctr[2], 1ull) == (unsigned long long)(gridDim.x - 1);
    }
    __syncthreads();
    if (last_s) {
        __threadfence();
        nl_check_block<CHECK_GATE>(d, 1, dt, (cudaGraphConditionalHandle)0);
        if (threadIdx.x == 0) d.ctr[2] = 0ull;
    }
}

// The step kernel.  `fuse` (graph steps): FUSE_CHECK, the last block to
// finish also takes the skin decision of every replica (the next node, the
// row build, runs on the work list it leaves, empty or not); FUSE_CHECK_GATE,
// the same, and the decision keeps the gate: the kernel returns at once
// while the gate is closed; FUSE_GATE, no decision (a later kernel of the step
// takes it), and the kernel returns at once while the gate is closed.  The
// kernel holds no device-side graph call, so profilers see it in graphs.
// Resident blocks that the register allocation leaves room for: at most 64
// registers a thread in mixed precision (32 warps per SM), 80 in FP64 (25 warps),
// whatever the threads per slot
template <class FT, int FB, int LPB> constexpr int force_min_blocks() {
    return 65536 / (FB * LPB * (sizeof(FT) == 4 ? 64 : 80)) > 0 ? 65536 / (FB * LPB * (sizeof(FT) == 4 ? 64 : 80)) : 1;
}
enum : int { FUSE_NONE = 0, FUSE_CHECK = 1, FUSE_CHECK_GATE = 2, FUSE_GATE = 3 };
template <class FT, int MODE, int FB, int LPB>
__global__ void __launch_bounds__(FB * LPB, (force_min_blocks<FT, FB, LPB>())) k_force(Dev d, TermP p, int cur,
                                                                                  int fuse) {
    __shared__ int last_s;
    static_assert(LPB == 1 || LPB == 2 || LPB == 4 || LPB == 8, "threads per bead slot");
    if (!force_block<FT, MODE, FB, LPB>(d, p, cur, MODE == 1 && (fuse == FUSE_CHECK_GATE || fuse == FUSE_GATE))) return;
    if (MODE == 1 && (fuse == FUSE_CHECK || fuse == FUSE_CHECK_GATE)) {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            last_s = atomicAdd(&d.ctr[2], 1ull) == (unsigned long long)(gridDim.x - 1);
        }
        __syncthreads();
        if (last_s) {
            __threadfence();
            if (fuse == FUSE_CHECK_GATE) nl_check_block<CHECK_GATE>(d, 1, p.dt, (cudaGraphConditionalHandle)0);
            else nl_check_block<CHECK_PLAIN>(d, 1, p.dt, (cudaGraphConditionalHandle)0);
            if (threadIdx.x == 0) d.ctr[2] = 0ull;
        }
    }
}

// the replicas whose rebuild overflowed the rows rebuild again at the next
// check (after the rows were reallocated); the others keep their lists
__global__ void k_mark_all(Dev d) {
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < d.R && d.rep[r].active && d.rep[r].rebuild) d.rep[r].first = 1;
}

// Minimum image of a difference of coordinates wrapped into [0, L) (so
// |d| < L) by compare and select: rintf runs on the slow conversion pipe.
// L = 0 (open axis) leaves d unchanged.
__device__ __forceinline__ float min_image_f(float d, float L) {
    const float h = 0.5f * L;
    d = d > h ? d - L : d;
    return d < -h ? d + L : d;
}

// FP32 error bound of a distance d <= ext between FP32 coordinates of
// magnitude <= ext (relative coordinates, or wrapped into [0, L) with L <=
// ext).  Each coordinate is the FP64 value rounded once (<= 2^-24 ext); a
// difference adds one rounding and the minimum-image shift by the rounded
// box length two more (<= 4 * 2^-24 ext per axis); the three squares and
// their sum add <= 3 * 2^-24 relative to d^2.  In distance terms that is
// <= sqrt(3) * 4 * 2^-24 ext + 1.5 * 2^-24 d < 5e-7 ext; the bound used is
// twice that plus an absolute 1e-5.
__host__ __device__ __forceinline__ double band_margin(double ext) { return 1e-5 + 1e-6 * ext; }

// FP32 decision band around a distance threshold T (error bound m)
struct Band {
    float lo, hi;   // squared FP32 distance: below lo -> inside, above hi -> outside
};
__device__ __forceinline__ Band make_band(double T, double m) {
    double a = T - m, b = T + m;
    return Band{a > 0.0 ? __double2float_rd(a * a) : -1.0f, __double2float_ru(b * b)};
}
__device__ __forceinline__ bool in_band(const Band &B, float d2) { return d2 >= B.lo && d2 <= B.hi; }

// ---- cell lists of the flagged replicas ---------------------------------------------
// Two grids per replica.  The near grid holds every bead, with cells of at
// least the largest radius of the terms that act between any two beads
// (Pauli, quasi-adiabatic, PID; each with the pad).  The far grid holds the
// charged beads, with cells of at least the electrostatic radius: only pairs of
// charged beads are kept beyond the near radius.  One grid at the list radius
// would give every bead the candidates of 27 cells of 25 A, ten times as many
// as the two grids do at 1e-3 beads per A^3 and a fifth of the beads charged.
//
// Periodic axes are cut into dims = floor(L / r) cells (wrapped); open axes
// count cells from the bounding-box minimum without bound.  When every axis is
// periodic and the grid fits its bucket budget, a cell IS a bucket; otherwise
// cells are hashed into the budget (chains in open space occupy few of their
// bounding box's cells).  Buckets are visited once each, so collisions only
// add candidates; the exact distance test decides.
enum : int { CG_NEAR = 0, CG_FAR = 1 };
constexpr int CELL_PACK = 1023;   // cell coordinates that fit the packed form
constexpr int CELL_SCAN = 1024;   // buckets per block of the scan
constexpr int CELL_CHARGED = 1 << 31;

__device__ __forceinline__ int cell_coord(const RepDev &rp, int g, int a, double x) {
    if (rp.per[a]) {
        double f = x * rp.box.cell_inv[a];
        f -= floor(f);
        int k = (int)(f * rp.dims[g][a]);
        return k < 0 ? 0 : (k >= rp.dims[g][a] ? rp.dims[g][a] - 1 : k);
    }
    int k = (int)floor((x - rp.lo[a]) * rp.cs[g]);   // cs holds 1 / cell edge on open axes
    return k < 0 ? 0 : k;
}
// bucket of a cell in the pool: the near grids of all replicas first, then the
// far grids, each half the size
__device__ __forceinline__ int cell_bucket(const Dev &d, const RepDev &rp, int g, int cx, int cy, int cz) {
    const int off = g == CG_NEAR ? rp.cell_off : d.ncells_near + rp.cell_off / 2;
    if (!rp.hashed[g]) return off + (cz * rp.dims[g][1] + cy) * rp.dims[g][0] + cx;
    uint32_t h = (uint32_t)cx * 73856093u ^ (uint32_t)cy * 19349663u ^ (uint32_t)cz * 83492791u;
    h = (h ^ (h >> 15)) * 0x9e3779b1u;
    return off + (int)__umulhi(h, (uint32_t)(g == CG_NEAR ? rp.cell_budget : rp.cell_budget / 2));
}
__device__ __forceinline__ bool cell_flagged(const Dev &d, int r) {
    if (r < 0) return false;
    const RepDev &rp = d.rep[r];
    return rp.active && rp.rebuild && !rp.tile;
}
__device__ __forceinline__ int cell_start(const Dev &d, int c) { return d.cell_start[c] + d.cell_base[c / CELL_SCAN]; }
// floats as unsigned integers of the same order
__device__ __forceinline__ unsigned f_key(float x) {
    const unsigned u = __float_as_uint(x);
    return (u >> 31) ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float f_of_key(unsigned k) { return __uint_as_float((k >> 31) ? k & 0x7fffffffu : ~k); }

// Bounding boxes along open axes, over the whole grid (in FP32, rounded
// outwards: no coordinate lies below the minimum, which is the origin of the
// cells and of the FP32 coordinates, and none is larger than the span that
// their error bound is taken from, however far from the origin the replica
// lies); the last block then sets the grids and FP32 bands of the flagged
// replicas.  One block per replica took 138 us for one of 54,744 beads.
// `count`: the launches of the pass, for the statistics.
__global__ void __launch_bounds__(256) k_cells(Dev d, int cur, int count) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    __shared__ int last_s;
    const int r = i < d.N ? d.rep_of[i] : -1;
    const bool on = cell_flagged(d, r) && !(d.rep[r].per[0] && d.rep[r].per[1] && d.rep[r].per[2]);
    const unsigned act = __ballot_sync(0xffffffffu, on);
    if (on) {
        const double4_32a q = d.pos[cur][i];
        const unsigned m = __match_any_sync(act, r);
        const bool lead = (threadIdx.x & 31) == __ffs(m) - 1;
        const double x[3] = {q.x, q.y, q.z};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const unsigned lo = __reduce_min_sync(m, f_key(__double2float_rd(x[a])));
            const unsigned hi = __reduce_max_sync(m, f_key(__double2float_ru(x[a])));
            if (lead) {
                atomicMin(&d.rep[r].lo_key[a], lo);
                atomicMax(&d.rep[r].hi_key[a], hi);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last_s = atomicAdd(&d.ctr[3], 1ull) == (unsigned long long)(gridDim.x - 1);
    }
    __syncthreads();
    if (!last_s) return;
    __threadfence();
    if (threadIdx.x == 0) {
        d.ctr[3] = 0ull;
        atomicAdd(d.ctr, (unsigned long long)count);
    }
    for (int k = threadIdx.x; k < d.R; k += 256) {
        if (!cell_flagged(d, k)) continue;
        RepDev &rp = d.rep[k];
        bool all_per = true;
        double ext = 0.0, span[3];
        for (int a = 0; a < 3; ++a) {
            span[a] = rp.box.cell[a];
            if (!rp.per[a]) {
                all_per = false;
                const float lo = f_of_key(*(volatile unsigned *)&rp.lo_key[a]);
                rp.lo[a] = (double)lo;
                span[a] = (double)f_of_key(*(volatile unsigned *)&rp.hi_key[a]) - (double)lo;
            } else {
                rp.lo[a] = 0.0;
            }
            ext = fmax(ext, span[a]);
        }
        for (int g = 0; g < 2; ++g) {
            const double rr = (g == CG_NEAR ? rp.r_near : rp.r_far) * (1.0 + 1e-9);
            const int bud = g == CG_NEAR ? rp.cell_budget : rp.cell_budget / 2;
            long long total = 1;
            bool packed = true;
            for (int a = 0; a < 3; ++a) {
                int dm = 1;
                if (rp.per[a]) {
                    const double q = floor(rp.box.cell[a] / rr);
                    dm = q < 1.0 ? 1 : (q > 4096.0 ? 4096 : (int)q);
                    packed = packed && dm <= CELL_PACK;
                } else {
                    packed = packed && span[a] / rr < (double)(CELL_PACK - 2);
                }
                rp.dims[g][a] = dm;
                total *= dm;
            }
            rp.cs[g] = 1.0 / rr;
            rp.hashed[g] = !(all_per && total <= bud);
            rp.packed[g] = packed;
        }
        // FP32 error bound of a distance (see band_margin)
        rp.band_m = band_margin(fmax(ext * (1.0 + 1e-6), rp.req_r));
        const double T[5] = {rp.req_r, 1.0 / rp.pauli_min_inv, 1.0 / rp.es_min_inv, 1.0 / rp.qa_min_inv,
                             1.0 / rp.pid_min_inv};
        for (int q = 0; q < 5; ++q) {
            const Band B = make_band(T[q], rp.band_m);
            rp.band_lo[q] = B.lo;
            rp.band_hi[q] = B.hi;
        }
        const Band B = make_band(rp.s_near > 0.0 ? rp.r_near : 0.0, rp.band_m);
        rp.near_lo = B.lo;
        rp.near_hi = B.hi;
        rp.band_mf = __double2float_ru(rp.band_m);
        rp.first = 0;
        rp.rebuilds += 1;
    }
}

// bucket counts of both grids; cell_key keeps a bead's packed cell
// coordinates (or its bucket, where they do not fit), -1 where it is in no cell
__global__ void __launch_bounds__(256) k_cell_count(Dev d, int cur) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= d.N) return;
    const int r = d.rep_of[i];
    const bool on = cell_flagged(d, r);
    int key[2] = {-1, -1};
    if (on) {
        const RepDev &rp = d.rep[r];
        const double4_32a q = d.pos[cur][i];
        for (int g = 0; g < 2; ++g) {
            if (g == CG_FAR && !(rp.far && q.w != 0.0)) continue;
            const int cx = cell_coord(rp, g, 0, q.x), cy = cell_coord(rp, g, 1, q.y), cz = cell_coord(rp, g, 2, q.z);
            const int b = cell_bucket(d, rp, g, cx, cy, cz);
            key[g] = rp.packed[g] ? cx | cy << 10 | cz << 20 : b;
            atomicAdd(&d.cell_cnt[b], 1);
        }
    }
    d.cell_key[i] = key[0];
    d.cell_key[d.N + i] = key[1];
}
// exclusive scan of the bucket counts within blocks of CELL_SCAN; the last
// block to finish scans the blocks' totals into cell_base
__global__ void __launch_bounds__(256) k_cell_scan(Dev d) {
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    __shared__ int ws[8], last_s;
    const int e = blockIdx.x * CELL_SCAN + 4 * t;
    int q[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) q[k] = e + k < d.ncells ? d.cell_cnt[e + k] : 0;
    const int sum = q[0] + q[1] + q[2] + q[3];
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    int before = x - sum;
    for (int k = 0; k < w; ++k) before += ws[k];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (e + k < d.ncells) d.cell_start[e + k] = before;
        before += q[k];
    }
    if (t == 255) d.cell_base[blockIdx.x] = before;
    __syncthreads();
    if (t == 0) {
        __threadfence();
        last_s = atomicAdd(&d.ctr[3], 1ull) == (unsigned long long)(gridDim.x - 1);
    }
    __syncthreads();
    if (!last_s || w != 0) return;
    __threadfence();
    if (t == 0) d.ctr[3] = 0ull;
    int run = 0;
    for (int k0 = 0; k0 < (int)gridDim.x; k0 += 32) {
        const int k = k0 + lane;
        const int p = k < (int)gridDim.x ? *(volatile int *)&d.cell_base[k] : 0;
        int y = p;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) y += u;
        }
        if (k < (int)gridDim.x) d.cell_base[k] = run + y - p;
        run += __shfl_sync(0xffffffffu, y, 31);
    }
    if (lane == 0) d.cell_base[gridDim.x] = run;
}
__device__ __forceinline__ int cell_bucket_of(const Dev &d, const RepDev &rp, int g, int key) {
    return rp.packed[g] ? cell_bucket(d, rp, g, key & 1023, (key >> 10) & 1023, (key >> 20) & 1023) : key;
}
// the sort leaves every count at zero, for the next build
__global__ void __launch_bounds__(256) k_cell_scatter(Dev d) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= d.N) return;
    for (int g = 0; g < 2; ++g) {
        const int key = d.cell_key[(size_t)g * d.N + i];
        if (key == -1) continue;
        const int b = cell_bucket_of(d, d.rep[d.rep_of[i]], g, key);
        d.cell_items[cell_start(d, b) + atomicSub(&d.cell_cnt[b], 1) - 1] = i;
    }
}
// slots of a bucket
__device__ __forceinline__ int cell_slots(const Dev &d) { return d.cell_base[(d.ncells + CELL_SCAN - 1) / CELL_SCAN]; }
__device__ __forceinline__ int2 cell_range(const Dev &d, int b) {
    return make_int2(cell_start(d, b), b + 1 < d.ncells ? cell_start(d, b + 1) : cell_slots(d));
}
// one thread per slot: the bead's rank among its bucket's is its place there
// (a deterministic order), with its FP32 coordinates, wrapped into [0, L) or
// taken from the bounding-box minimum
__global__ void __launch_bounds__(256) k_cell_finish(Dev d, int cur) {
    const int k = blockIdx.x * 256 + threadIdx.x;
    if (k >= cell_slots(d)) return;
    const int i = d.cell_items[k];
    const RepDev &rp = d.rep[d.rep_of[i]];
    // the near slots come first
    const int g = k < cell_start(d, d.ncells_near) ? CG_NEAR : CG_FAR;
    const int2 s = cell_range(d, cell_bucket_of(d, rp, g, d.cell_key[(size_t)g * d.N + i]));
    int rank = 0;
    for (int u = s.x; u < s.y; ++u) rank += d.cell_items[u] < i;
    const double4_32a q = d.pos[cur][i];
    const double x[3] = {q.x, q.y, q.z};
    float f[3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
        f[a] = (float)(rp.per[a] ? x[a] - rp.box.cell[a] * floor(x[a] * rp.box.cell_inv[a]) : x[a] - rp.lo[a]);
    d.cell_pos[s.x + rank] = make_float4(f[0], f[1], f[2], __int_as_float(q.w != 0.0 ? i | CELL_CHARGED : i));
}

// ---- Verlet rows of the cell build (legacy_update.cpp:16-62 + the update_*
// filters), one warp per bead i, beads in bucket order ------------------------------
// A pair is decided in FP32 when its FP32 distance is outside the bands of
// the replica (k_cells: the list radius, r_excl + pad, 2D + pad, the QA
// formation radius + pad, each widened by the FP32 error bound), and by the
// exact FP64 test inside them.  The candidates of the neighbouring buckets are
// taken 32 at a time by the lanes: the row is compacted by ballot, and the
// bead's latency chain is a few rounds deep instead of one candidate deep.
// The near grid gives every pair within the near radius, all its flags with it;
// the far grid then, for a charged bead, the pairs beyond that radius.
// Buckets are visited z, then y, then x offset (first occurrence of each
// bucket).  Quasi-adiabatic partners are ranked by j within the warp at the
// end, so the free-pair source list is ordered as update_free_pairs
// (free_pair.cpp:9-19) walks it.
// Go-list membership of a native contact of length nd (r < T = 2 nd + pad,
// go.cpp:11-22): by the FP32 squared distance d2 outside a band around T
// (directed rounding, widened by the narrowing error of T and by mf, the
// error bound of the FP32 distance), by the reference's test inside it
__device__ __forceinline__ bool go_listed(const RepDev &rp, const BoxD &bx, float mf, double nd, float d2,
                                          double4_32a pi, const double4_32a &pj) {
    const double T = __dadd_rn(__dmul_rn(2.0, nd), rp.pad);
    const float Tf = narrow_f(T);
    const float mm = __fmaf_ru(Tf, 1.2e-7f, mf);
    const float blo = __fsub_rd(Tf, mm), bhi = __fadd_ru(Tf, mm);
    const Band B{blo > 0.0f ? __fmul_rd(blo, blo) : -1.0f, __fmul_ru(bhi, bhi)};
    if (in_band(B, d2)) return dist_exact(bx, pi, pj) < T;
    return d2 < B.lo;
}
// entry k of the natives [n0, n1) of the warp's bead: its list flag, and its
// place in the bead's Go list, which keeps the order of the natives
__device__ __forceinline__ void go_append(const Dev &d, int k, int n0, int n1, bool on, int j, double nd, int &ngo) {
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (k < n1) d.nat_on[k] = on;
    if (on) {
        const int at = n0 + ngo + __popc(m & ((1u << (threadIdx.x & 31)) - 1u));
        d.act_j[at] = j;
        d.act_d[at] = nd;
    }
    ngo += __popc(m);
}
// the Go list of beads [b, b + n) from the list flags (after a restore)
__global__ void k_go_lists(Dev d, int b, int n) {
    const int i = b + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= b + n) return;
    const int n0 = d.nat_start[i], n1 = d.nat_end[i];
    int at = n0;
    for (int k = n0; k < n1; ++k)
        if (d.nat_on[k]) {
            d.act_j[at] = d.nat_j[k];
            d.act_d[at++] = d.nat_d[k];
        }
    d.go_cnt[i] = at - n0;
}

// One bead's partners put in ascending order by the warp that collected them:
// a bitonic sort of 32 U register entries (distinct beads, padded with the
// largest int).  Ranking every entry against every other took two thirds of
// k_nl_cells' instructions (3470 a bead at about 60 partners).
template <int U> __device__ __noinline__ void sort_row(int32_t *row, int m, int lane) {
    static_assert(32 * U <= QA_TMP_CAP, "a row holds the padded entries' slots");
    int v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = u * 32 + lane < m ? row[u * 32 + lane] : INT_MAX;
#pragma unroll
    for (int k = 2; k <= 32 * U; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j; j >>= 1) {
            if (j >= 32) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int w = u ^ (j >> 5);
                    if (w < u) continue;
                    const int lo = min(v[u], v[w]), hi = max(v[u], v[w]);
                    const bool up = ((u * 32) & k) == 0;
                    v[u] = up ? lo : hi;
                    v[w] = up ? hi : lo;
                }
            } else {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int o = __shfl_xor_sync(0xffffffffu, v[u], j);
                    const bool up = ((u * 32 + lane) & k) == 0;
                    v[u] = up == ((lane & j) == 0) ? min(v[u], o) : max(v[u], o);
                }
            }
        }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (u * 32 + lane < m) row[u * 32 + lane] = v[u];
}

constexpr int NC_WARPS = 8;
__global__ void __launch_bounds__(NC_WARPS * 32, 4) k_nl_cells(Dev d, TermP p, int cur) {
    const int lane = threadIdx.x & 31;
    const int slot = blockIdx.x * NC_WARPS + (threadIdx.x >> 5);
    if (slot >= cell_start(d, d.ncells_near)) return;   // warp-uniform: the near slots
    const float4 me = d.cell_pos[slot];
    const int i = __float_as_int(me.w) & ~CELL_CHARGED;
    const bool charged = __float_as_int(me.w) < 0;
    const RepDev &rp = d.rep[d.rep_of[i]];
    const double4_32a *pos = d.pos[cur];
    const double4_32a pi = pos[i];
    const int ci = d.chain[i], si = d.seq[i];
    const int n0 = d.nat_start[i], n1 = d.nat_end[i];
    const unsigned FULL = 0xffffffffu, lt = (1u << lane) - 1u;
    const bool periodic = rp.per_any != 0;

    // Go list: update_go_contacts, go.cpp:11-22 (lanes over the natives)
    int ngo = 0;
    if (n0 < n1) {
        const PairGeo<float> geo(rp.box, periodic, pi);
        for (int k0 = n0; k0 < n1; k0 += 32) {
            const int k = k0 + lane;
            bool on = false;
            int j = 0;
            double nd = 0.0;
            if (k < n1) {
                j = d.nat_j[k];
                nd = d.nat_d[k];
                const double4_32a pj = pos[j];
                const V3<float> e = geo.to(pj);
                on = go_listed(rp, rp.box, rp.band_mf, nd, e.x * e.x + e.y * e.y + e.z * e.z, pi, pj);
            }
            go_append(d, k, n0, n1, on, j, nd, ngo);
        }
    }
    if (lane == 0) d.go_cnt[i] = ngo;

    const float Lx = narrow_f(rp.box.cell[0]), Ly = narrow_f(rp.box.cell[1]), Lz = narrow_f(rp.box.cell[2]);
    const Band Breq{rp.band_lo[0], rp.band_hi[0]}, Bpa{rp.band_lo[1], rp.band_hi[1]};
    const Band Bes{rp.band_lo[2], rp.band_hi[2]}, Bqa{rp.band_lo[3], rp.band_hi[3]};
    const Band Bpid{rp.band_lo[4], rp.band_hi[4]}, Bnear{rp.near_lo, rp.near_hi};
    const bool pauli_on = p.on[XMD_TERM_PAULI] != 0;
    // PID bundles join beads that both have their chain neighbours
    const bool pid_on = p.on[XMD_TERM_PID] != 0 && (d.bflags[i] & (BF_PREV | BF_NEXT)) == (BF_PREV | BF_NEXT);
    const bool go_on = p.on[XMD_TERM_GO] != 0;
    const bool es_on = charged && (p.on[XMD_TERM_CONST_ES] || p.on[XMD_TERM_REL_ES]);
    const bool qa_on = d.qa_on && p.on[XMD_TERM_QA];
    const int nref = qa_on ? min(d.qa.ref_cnt[i], QA_REF_CAP) : 0;
    const int nnat = n1 - n0;
    const int my_nat = lane < nnat ? d.nat_j[n0 + lane] : -1;
    // disulfide list (update_nat_ssbonds, native_ss.cpp:8-19) and partners
    const bool ss_on = p.on[XMD_TERM_NAT_SS] != 0;
    const int ss0 = d.ss_start[i], ss1 = d.ss_end[i];
    if (ss_on)
        for (int k = ss0 + lane; k < ss1; k += 32)
            d.ss_on[k] = dist2_exact(rp.box, pi, pos[d.ss_j[k]]) < rp.s_ss;
    const int nss = ss_on ? ss1 - ss0 : 0;
    const int my_ss = lane < nss ? d.ss_j[ss0 + lane] : -1;
    int my_qa = -1;
    if (lane < nref) {
        const int s = d.qa.ref[(size_t)lane * d.N + i];
        my_qa = d.qa.ct_i1[s] == i ? d.qa.ct_i2[s] : d.qa.ct_i1[s];
    }
    const int cap = d.nl_cap;
    int cnt = 0, tcnt = 0;
    // candidates within reach (one in six of those in the buckets), in order;
    // the tests behind the distance run on 32 of them at a time
    __shared__ int2 s_queue[NC_WARPS][64];
    int2 *queue = s_queue[threadIdx.x >> 5];
    for (int g = 0; g < 2; ++g) {
        int qn = 0;
        if (g == CG_NEAR ? rp.s_near <= 0.0 : !(es_on && rp.far)) continue;
        // neighbouring buckets: lane l < 27 takes offsets (l % 3, l / 3 % 3, l / 9) - 1,
        // the first lane of each bucket its range of slots
        int key = -1;
        if (lane < 27) {
            int cc[3];
            if (rp.packed[g]) {
                const int v = d.cell_key[(size_t)g * d.N + i];
                cc[0] = v & 1023; cc[1] = (v >> 10) & 1023; cc[2] = (v >> 20) & 1023;
            } else {
                cc[0] = cell_coord(rp, g, 0, pi.x);
                cc[1] = cell_coord(rp, g, 1, pi.y);
                cc[2] = cell_coord(rp, g, 2, pi.z);
            }
            const int off[3] = {lane % 3 - 1, (lane / 3) % 3 - 1, lane / 9 - 1};
            bool ok = true;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                int k = cc[a] + off[a];
                if (rp.per[a]) {
                    const int dm = rp.dims[g][a];
                    k = k < 0 ? k + dm : (k >= dm ? k - dm : k);
                } else if (k < 0) {
                    ok = false;
                }
                cc[a] = k;
            }
            if (ok) key = cell_bucket(d, rp, g, cc[0], cc[1], cc[2]);
        }
        const unsigned same = __match_any_sync(FULL, key);
        int q0 = 0, csz = 0;
        if (key >= 0 && (same & lt) == 0u) {
            const int2 s = cell_range(d, key);
            q0 = s.x;
            csz = s.y - s.x;
        }
        // the buckets' candidates as one sequence, taken 32 at a time: lane l
        // takes entry c = base + l, which lies in the bucket of the last lane
        // whose exclusive prefix of bucket sizes is <= c
        int pre = csz;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, pre, o);
            if (lane >= o) pre += y;
        }
        const int total = __shfl_sync(FULL, pre, 31);
        pre -= csz;
        q0 -= pre;
        const float reach = g == CG_NEAR ? Bnear.hi : fminf(Bes.hi, Breq.hi);
        for (int base = 0; base < total; base += 32) {
            const int c = base + lane;
            int lo = 0;
#pragma unroll
            for (int step = 16; step; step >>= 1) {
                const int pm = __shfl_sync(FULL, pre, lo + step);
                if (pm <= c) lo += step;
            }
            const int q = __shfl_sync(FULL, q0, lo) + c;
            bool in = false;
            int jw = 0;
            float dj = 0.0f;
            if (c < total) {
                const float4 f = d.cell_pos[q];
                jw = __float_as_int(f.w);
                float ddx = f.x - me.x, ddy = f.y - me.y, ddz = f.z - me.z;
                if (periodic) {
                    ddx = min_image_f(ddx, Lx);
                    ddy = min_image_f(ddy, Ly);
                    ddz = min_image_f(ddz, Lz);
                }
                dj = ddx * ddx + ddy * ddy + ddz * ddz;
                in = (jw & ~CELL_CHARGED) != i && dj <= reach;
            }
            const unsigned im = __ballot_sync(FULL, in);
            if (in) queue[qn + __popc(im & lt)] = make_int2(jw, __float_as_int(dj));
            qn += __popc(im);
            const bool last = base + 32 >= total;
            while (qn >= 32 || (last && qn)) {
                __syncwarp();
                int flags = 0;
                bool qa_free = false;
                int j = -1;
                if (lane < qn) {
                    const int2 e = queue[lane];
                    j = e.x & ~CELL_CHARGED;
                    const bool es_pair = es_on && e.x < 0;
                    const float d2 = __int_as_float(e.y);
                    const int cj = d.chain[j], sj = d.seq[j];
                    const int df = si > sj ? si - sj : sj - si;
                    if (!(ci == cj && df < 3)) {
                        bool in_req, pa, es, qa, pd, near;
                        if (in_band(Breq, d2) || in_band(Bnear, d2) || (pauli_on && in_band(Bpa, d2)) ||
                            (es_pair && in_band(Bes, d2)) || (qa_on && in_band(Bqa, d2)) ||
                            (pid_on && in_band(Bpid, d2))) {
                            const double s2 = periodic ? dist2_exact(rp.box, pi, pos[j]) : dist2_open(pi, pos[j]);
                            in_req = s2 < rp.s_req;
                            near = s2 < rp.s_near;
                            pa = s2 < rp.s_pa;
                            es = s2 < rp.s_es;
                            qa = s2 < rp.s_qa;
                            pd = s2 < rp.s_pid;
                        } else {
                            in_req = d2 < Breq.lo;
                            near = d2 < Bnear.lo;
                            pa = d2 < Bpa.lo;
                            es = d2 < Bes.lo;
                            qa = d2 < Bqa.lo;
                            pd = d2 < Bpid.lo;
                        }
                        if (in_req && near == (g == CG_NEAR)) {
                            if (pauli_on && pa) flags |= NL_PAULI;
                            if (es_pair && es) flags |= NL_ES;
                            if (pid_on && pd && (d.bflags[j] & (BF_PREV | BF_NEXT)) == (BF_PREV | BF_NEXT))
                                flags |= NL_PID;
                            qa_free = qa_on && j > i && qa;
                        }
                    }
                }
                // a native contact leaves every list (natives leave only with
                // native contacts enabled, main.cpp:504-530); a pair in contact
                // is no free pair.  The bead's natives and contact partners are
                // held one per lane and broadcast.
                if (go_on && __any_sync(FULL, flags != 0 || qa_free)) {
                    if (nnat <= 32) {
                        for (int k = 0; k < nnat; ++k)
                            if (__shfl_sync(FULL, my_nat, k) == j) { flags = 0; qa_free = false; }
                    } else {
                        for (int k = n0; k < n1; ++k)
                            if (d.nat_j[k] == j) { flags = 0; qa_free = false; }
                    }
                }
                if (qa_on && __any_sync(FULL, qa_free))
                    for (int k = 0; k < nref; ++k)
                        if (__shfl_sync(FULL, my_qa, k) == j) qa_free = false;
                // a native disulfide is in no non-native list (main.cpp:579-580)
                if (nss && __any_sync(FULL, flags != 0 || qa_free)) {
                    if (nss <= 32) {
                        for (int k = 0; k < nss; ++k)
                            if (__shfl_sync(FULL, my_ss, k) == j) { flags = 0; qa_free = false; }
                    } else {
                        for (int k = ss0; k < ss1; ++k)
                            if (d.ss_j[k] == j) { flags = 0; qa_free = false; }
                    }
                }
                const unsigned km = __ballot_sync(FULL, flags != 0);
                if (flags) {
                    const int at = cnt + __popc(km & lt);
                    if (at < cap) d.nl_row[(size_t)at * d.N + i] = j | flags;
                }
                cnt += __popc(km);
                if (qa_on) {
                    const unsigned qm = __ballot_sync(FULL, qa_free);
                    if (qa_free) {
                        const int at = tcnt + __popc(qm & lt);
                        if (at < QA_TMP_CAP) d.qa.tmp[(size_t)i * QA_TMP_CAP + at] = j;
                    }
                    tcnt += __popc(qm);
                }
                // what is left (fewer than 32) moves to the front
                const int2 left = queue[32 + lane];
                __syncwarp();
                queue[lane] = left;
                __syncwarp();
                qn = max(qn - 32, 0);
            }
        }
    }
    if (qa_on && tcnt > 1) {
        const int m = min(tcnt, QA_TMP_CAP);
        int32_t *row = d.qa.tmp + (size_t)i * QA_TMP_CAP;
        __syncwarp();
        if (m <= 32) sort_row<1>(row, m, lane);
        else if (m <= 64) sort_row<2>(row, m, lane);
        else if (m <= 128) sort_row<4>(row, m, lane);
        else sort_row<8>(row, m, lane);
    }
    if (lane == 0) {
        atomicMax(&d.ctr[1], (unsigned long long)cnt);   // longest row needed
        if (cnt > cap) {
            atomicOr(d.status, ST_CAPACITY);
            cnt = cap;
        }
        d.nl_cnt[i] = cnt;
        d.orig[i] = pi;
        if (qa_on) {
            if (tcnt > QA_TMP_CAP) atomicOr(d.status, ST_CAPACITY);
            d.qa.tmp_cnt[i] = min(tcnt, QA_TMP_CAP);
        }
    }
}

// ---- Verlet build for replicas of at most TILE_MAX beads ---------------------------
// A block takes chunks of TL_CH beads i from the work list of the last skin
// check (the chunks of every flagged replica); for each it holds the whole replica in
// shared memory (FP32 coordinates relative to the replica, chain and sequence
// index) and each warp scans every bead j of the replica for one bead i at a
// time, lane k taking j = j0 + k.  A pair is decided in FP32 when its FP32
// distance is farther than the error margin m from every threshold (the list
// radius, r_excl + pad, 2D + pad, the QA formation radius + pad); otherwise the
// exact FP64 test decides it.  The margin (band_margin) bounds the FP32 error
// of a distance between coordinates of magnitude <= ext, so both paths keep
// exactly the same pairs.
// Rows come out ordered by j (ballot compaction in lane order).
constexpr int TL_CH = 8;       // rows per chunk: one per warp (a pass of a few replicas spreads over more blocks)
constexpr int TL_THREADS = 256;
constexpr int TL_WARPS = TL_THREADS / 32;
constexpr int TILE_MAX = 4096;

// dynamic shared memory of a tile block for a replica of n beads: the box of
// each group of 32 consecutive beads (lo, hi), then the FP32 coordinates, then
// chain and sequence indices
__host__ __device__ constexpr size_t tile_bytes(int n) {
    return 2 * sizeof(float4) * (size_t)((n + 31) / 32) + (sizeof(float4) + sizeof(int2)) * (size_t)n;
}

// FP32 coordinate of the pre-filter: wrapped into [0, L) on periodic axes,
// else relative to the replica's first bead (from split positions: the FP64
// difference to within 2^-46, then rounded to FP32, with no FP64 instruction)
__device__ __forceinline__ float tl_rel(const RepDev &rp, int a, double x, F2 ref) {
    if (rp.per[a]) return (float)(x - rp.box.cell[a] * floor(x * rp.box.cell_inv[a]));
    return ff_diff(ref, split_d(x)).h;
}



__device__ __forceinline__ void tl_chunk(const Dev &d, const TermP &p, int cur, const int2 chk) {
    const int r = chk.x;
    if (r < 0) return;   // free chunk slot
    RepDev &rp = d.rep[r];
    if (!rp.active || !rp.rebuild || !rp.tile) return;
    extern __shared__ float4 tl_smem[];
    const int b = rp.begin, n = rp.n;
    const int ng = (n + 31) / 32;
    float4 *gbox = tl_smem;
    float4 *sq = gbox + 2 * ng;
    int2 *scs = (int2 *)(sq + n);
    __shared__ float ext_s[TL_WARPS];
    const double4_32a *pos = d.pos[cur];
    const BoxD bx = rp.box;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const P2 p0 = split_p(pos[b]);

    float ext = 0.0f;
    // two loops on a block-uniform flag, so the open-box loop carries no
    // FP64 work (a select between the two forms would execute both)
    if ((rp.per[0] | rp.per[1] | rp.per[2]) == 0) {
        for (int k = t; k < n; k += TL_THREADS) {
            const double4_32a q = pos[b + k];
            const float x = ff_diff(p0.x, split_d(q.x)).h, y = ff_diff(p0.y, split_d(q.y)).h,
                        z = ff_diff(p0.z, split_d(q.z)).h;
            sq[k] = make_float4(x, y, z, narrow_f(q.w));
            scs[k] = make_int2(d.chain[b + k], d.seq[b + k]);
            ext = fmaxf(ext, fmaxf(fabsf(x), fmaxf(fabsf(y), fabsf(z))));
        }
    } else {
        for (int k = t; k < n; k += TL_THREADS) {
            const double4_32a q = pos[b + k];
            const float x = tl_rel(rp, 0, q.x, p0.x), y = tl_rel(rp, 1, q.y, p0.y), z = tl_rel(rp, 2, q.z, p0.z);
            sq[k] = make_float4(x, y, z, narrow_f(q.w));
            scs[k] = make_int2(d.chain[b + k], d.seq[b + k]);
            ext = fmaxf(ext, fmaxf(fabsf(x), fmaxf(fabsf(y), fabsf(z))));
        }
    }
    for (int o = 16; o; o >>= 1) ext = fmaxf(ext, __shfl_xor_sync(0xffffffffu, ext, o));
    if (lane == 0) ext_s[w] = ext;
    __syncthreads();
    ext = 0.0f;
    for (int q = 0; q < TL_WARPS; ++q) ext = fmaxf(ext, ext_s[q]);
    // decision bands of the chunk, formed once (FP64 work off the scan)
    // (one thread per band: the reciprocals are FP64 divisions)
    __shared__ Band bands_s[5];
    __shared__ float mf_s;
    if (t < 5) {
        double exd = fmax((double)ext, rp.req_r);
        for (int a = 0; a < 3; ++a) exd = fmax(exd, bx.cell[a]);
        const double m = band_margin(exd);
        const double inv = t == 1 ? rp.pauli_min_inv : t == 2 ? rp.es_min_inv : t == 3 ? rp.qa_min_inv
                                                                                       : rp.pid_min_inv;
        bands_s[t] = make_band(t == 0 ? rp.req_r : 1.0 / inv, m);
        if (t == 0) mf_s = __double2float_ru(m);
    }
    // bounding box of each group of 32 beads j (one warp per group)
    for (int g = w; g < ng; g += TL_WARPS) {
        const float4 q = sq[min(g * 32 + lane, n - 1)];
        float lx = q.x, ly = q.y, lz = q.z, hx = q.x, hy = q.y, hz = q.z;
        for (int o = 16; o; o >>= 1) {
            lx = fminf(lx, __shfl_xor_sync(0xffffffffu, lx, o));
            ly = fminf(ly, __shfl_xor_sync(0xffffffffu, ly, o));
            lz = fminf(lz, __shfl_xor_sync(0xffffffffu, lz, o));
            hx = fmaxf(hx, __shfl_xor_sync(0xffffffffu, hx, o));
            hy = fmaxf(hy, __shfl_xor_sync(0xffffffffu, hy, o));
            hz = fmaxf(hz, __shfl_xor_sync(0xffffffffu, hz, o));
        }
        if (lane == 0) {
            gbox[2 * g] = make_float4(lx, ly, lz, 0.0f);
            gbox[2 * g + 1] = make_float4(hx, hy, hz, 0.0f);
        }
    }
    __syncthreads();
    const float mf = mf_s;

    const bool pauli_on = p.on[XMD_TERM_PAULI] != 0;
    const bool go_on = p.on[XMD_TERM_GO] != 0;
    const bool es_on = (p.on[XMD_TERM_CONST_ES] || p.on[XMD_TERM_REL_ES]);
    const bool qa_on = d.qa_on && p.on[XMD_TERM_QA];
    const bool ss_on = p.on[XMD_TERM_NAT_SS] != 0;
    const Band Breq = bands_s[0], Bpa = bands_s[1], Bes = bands_s[2], Bqa = bands_s[3], Bpid = bands_s[4];
    const bool pid_term = p.on[XMD_TERM_PID] != 0;
    const float Lx = narrow_f(bx.cell[0]), Ly = narrow_f(bx.cell[1]), Lz = narrow_f(bx.cell[2]);
    const bool periodic = (rp.per[0] | rp.per[1] | rp.per[2]) != 0;
    const int cap = d.nl_cap;
    const unsigned lt = (1u << lane) - 1u;
    const float skip2 = Breq.hi * 1.0001f;

    if (t == 0 && chk.y == b) {
        rp.first = 0;
        rp.rebuilds += 1;
    }
    const int i_end = min(chk.y + TL_CH, b + n);
    for (int i = chk.y + w; i < i_end; i += TL_WARPS) {
        const int li = i - b;
        const float4 qi = sq[li];
        const int2 ci = scs[li];
        const double4_32a pi = pos[i];
        const int n0 = d.nat_start[i], n1 = d.nat_end[i];
        // PID bundles join beads that both have their chain neighbours
        const bool pid_on = pid_term && (d.bflags[i] & (BF_PREV | BF_NEXT)) == (BF_PREV | BF_NEXT);

        // Go list: update_go_contacts, go.cpp:11-22
        int ngo = 0;
        for (int k0 = n0; k0 < n1; k0 += 32) {
            const int k = k0 + lane;
            bool on = false;
            int j = 0;
            double nd = 0.0;
            if (k < n1) {
                j = d.nat_j[k];
                nd = d.nat_d[k];
                const float4 qj = sq[j - b];
                float dx = qj.x - qi.x, dy = qj.y - qi.y, dz = qj.z - qi.z;
                if (periodic) {
                    dx = min_image_f(dx, Lx);
                    dy = min_image_f(dy, Ly);
                    dz = min_image_f(dz, Lz);
                }
                on = go_listed(rp, bx, mf, nd, dx * dx + dy * dy + dz * dz, pi, pos[j]);
            }
            go_append(d, k, n0, n1, on, j, nd, ngo);
        }
        if (lane == 0) d.go_cnt[i] = ngo;

        // disulfide list: update_nat_ssbonds, native_ss.cpp:8-19 (exact test;
        // a bead has at most a few disulfides)
        const int ss0 = d.ss_start[i], ss1 = d.ss_end[i];
        if (ss_on)
            for (int k = ss0 + lane; k < ss1; k += 32) {
                const double4_32a pj = pos[d.ss_j[k]];
                d.ss_on[k] = (periodic ? dist2_exact(bx, pi, pj) : dist2_open(pi, pj)) < rp.s_ss;
            }
        const int nss = ss_on ? ss1 - ss0 : 0;
        const int my_ss = lane < nss ? d.ss_j[ss0 + lane] : -1;

        int nref = 0;
        if (qa_on) nref = min(d.qa.ref_cnt[i], QA_REF_CAP);
        // the row's natives and contact partners, one per lane (broadcast by
        // shuffle in the exclusion checks)
        const int nnat = n1 - n0;
        const int my_nat = lane < nnat ? d.nat_j[n0 + lane] : -1;
        int my_qa = -1;
        if (lane < nref) {
            const int s = d.qa.ref[(size_t)lane * d.N + i];
            my_qa = d.qa.ct_i1[s] == i ? d.qa.ct_i2[s] : d.qa.ct_i1[s];
        }
        int cnt = 0, tcnt = 0;
        for (int j0 = 0; j0 < n; j0 += 32) {
            if (!periodic) {
                // a group whose box is beyond the list radius holds no pair
                // (FP32 rounding is monotone, so the box distance never exceeds
                // a member's distance; the factor covers contraction order)
                const float4 lo = gbox[2 * (j0 >> 5)], hi = gbox[2 * (j0 >> 5) + 1];
                const float gx = fmaxf(fmaxf(lo.x - qi.x, qi.x - hi.x), 0.0f);
                const float gy = fmaxf(fmaxf(lo.y - qi.y, qi.y - hi.y), 0.0f);
                const float gz = fmaxf(fmaxf(lo.z - qi.z, qi.z - hi.z), 0.0f);
                if (gx * gx + gy * gy + gz * gz > skip2) continue;
            }
            const int lj = j0 + lane;
            int flags = 0;
            bool qa_free = false;
            if (lj < n && lj != li) {
                const float4 qj = sq[lj];
                float dx = qj.x - qi.x, dy = qj.y - qi.y, dz = qj.z - qi.z;
                if (periodic) {
                    dx = min_image_f(dx, Lx);
                    dy = min_image_f(dy, Ly);
                    dz = min_image_f(dz, Lz);
                }
                const float d2 = dx * dx + dy * dy + dz * dz;
                const int2 cj = scs[lj];
                const int df = ci.y > cj.y ? ci.y - cj.y : cj.y - ci.y;
                if (d2 <= Breq.hi && !(ci.x == cj.x && df < 3)) {
                    bool in_req, pa, es, qa, pd;
                    if (in_band(Breq, d2) || (pauli_on && in_band(Bpa, d2)) || (es_on && in_band(Bes, d2)) ||
                        (qa_on && in_band(Bqa, d2)) || (pid_on && in_band(Bpid, d2))) {
                        const double s2 = periodic ? dist2_exact(bx, pi, pos[b + lj]) : dist2_open(pi, pos[b + lj]);
                        in_req = s2 < rp.s_req;
                        pa = s2 < rp.s_pa;
                        es = s2 < rp.s_es;
                        qa = s2 < rp.s_qa;
                        pd = s2 < rp.s_pid;
                    } else {
                        in_req = d2 < Breq.lo;
                        pa = d2 < Bpa.lo;
                        es = d2 < Bes.lo;
                        qa = d2 < Bqa.lo;
                        pd = d2 < Bpid.lo;
                    }
                    if (in_req) {
                        if (pauli_on && pa) flags |= NL_PAULI;
                        if (es_on && es && qi.w * qj.w != 0.0f) flags |= NL_ES;
                        if (pid_on && pd && (d.bflags[b + lj] & (BF_PREV | BF_NEXT)) == (BF_PREV | BF_NEXT))
                            flags |= NL_PID;
                        qa_free = qa_on && lj > li && qa;
                    }
                }
            }
            // natives leave the list only with native contacts enabled
            // (main.cpp:504-530); the loop is warp-uniform
            if (go_on && __any_sync(0xffffffffu, flags != 0 || qa_free)) {
                if (nnat <= 32) {
                    for (int k = 0; k < nnat; ++k)
                        if (__shfl_sync(0xffffffffu, my_nat, k) == b + lj) { flags = 0; qa_free = false; }
                } else {
                    for (int k = n0; k < n1; ++k)
                        if (d.nat_j[k] == b + lj) { flags = 0; qa_free = false; }
                }
            }
            if (qa_on && __any_sync(0xffffffffu, qa_free))
                for (int k = 0; k < nref; ++k)
                    if (__shfl_sync(0xffffffffu, my_qa, k) == b + lj) qa_free = false;
            // a native disulfide is in no non-native list (legacy_update's
            // merge against all_nat_ss, main.cpp:579-580)
            if (nss && __any_sync(0xffffffffu, flags != 0 || qa_free)) {
                if (nss <= 32) {
                    for (int k = 0; k < nss; ++k)
                        if (__shfl_sync(0xffffffffu, my_ss, k) == b + lj) { flags = 0; qa_free = false; }
                } else {
                    for (int k = ss0; k < ss1; ++k)
                        if (d.ss_j[k] == b + lj) { flags = 0; qa_free = false; }
                }
            }
            const unsigned km = __ballot_sync(0xffffffffu, flags != 0);
            if (flags) {
                const int at = cnt + __popc(km & lt);
                if (at < cap) d.nl_row[(size_t)at * d.N + i] = (b + lj) | flags;
            }
            cnt += __popc(km);
            if (qa_on) {
                const unsigned qm = __ballot_sync(0xffffffffu, qa_free);
                if (qa_free) {
                    const int at = tcnt + __popc(qm & lt);
                    if (at < QA_TMP_CAP) d.qa.tmp[(size_t)i * QA_TMP_CAP + at] = b + lj;
                }
                tcnt += __popc(qm);
            }
        }
        if (lane == 0) {
            atomicMax(&d.ctr[1], (unsigned long long)cnt);
            if (cnt > cap) {
                atomicOr(d.status, ST_CAPACITY);
                cnt = cap;
            }
            d.nl_cnt[i] = cnt;
            d.orig[i] = pi;
            if (qa_on) {
                if (tcnt > QA_TMP_CAP) atomicOr(d.status, ST_CAPACITY);
                d.qa.tmp_cnt[i] = min(tcnt, QA_TMP_CAP);
            }
        }
    }
}

// `count`: the launches of a pass that has no cell build (0: counted elsewhere;
// launches that run every step, with or without work, where they are issued)
__global__ void __launch_bounds__(TL_THREADS, 4) k_nl_tile(Dev d, TermP p, int cur, int count) {
    step_order();
    const int nw = *d.nwork;
    if (count && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(d.ctr, (unsigned long long)count);
    for (int w = blockIdx.x; w < nw; w += gridDim.x) {
        tl_chunk(d, p, cur, d.chunks[d.work[w]]);
        __syncthreads();   // the next chunk overwrites the shared tile
    }
}

// =================================================================== host ==

// the step kernel of a precision, mode and launch shape (beads per block and
// threads per bead, the shapes the autotuner chooses from); the evaluation
// pass has one shape
constexpr int EVAL_FB = 64, EVAL_LPB = 4;
// The limit belongs to the kernel, not to a context: always the largest any
// context uses, so that a later context does not lower it for an earlier one.
static void allow_smem(const void *kernel, size_t most) {
    CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
}
static size_t force_smem(bool mixed, int mode, int fb, bool qa) {
    if (mode == 0) fb = EVAL_FB;
#define XMD_SM(B) (mixed ? step_smem<float, B>(qa) : step_smem<double, B>(qa))
    return fb == 32 ? XMD_SM(32) : fb == 64 ? XMD_SM(64) : XMD_SM(128);
#undef XMD_SM
}
static int force_blocks(int n, int fb) { return (n + fb - 6) / (fb - 5); }   // step_beads
static void *force_kernel(bool mixed, int mode, int fb, int lpb) {
#define XMD_FK(M, B, L) (mixed ? (void *)k_force<float, M, B, L> : (void *)k_force<double, M, B, L>)
    if (mode == 0) return XMD_FK(0, EVAL_FB, EVAL_LPB);
    switch (fb * 8 + lpb) {   // (eight threads per slot: Engine::force_shape)
    case 32 * 8 + 1: return XMD_FK(1, 32, 1);
    case 32 * 8 + 2: return XMD_FK(1, 32, 2);
    case 32 * 8 + 4: return XMD_FK(1, 32, 4);
    case 32 * 8 + 8: return XMD_FK(1, 32, 8);
    case 64 * 8 + 1: return XMD_FK(1, 64, 1);
    case 64 * 8 + 2: return XMD_FK(1, 64, 2);
    case 64 * 8 + 4: return XMD_FK(1, 64, 4);
    case 128 * 8 + 1: return XMD_FK(1, 128, 1);
    case 128 * 8 + 2: return XMD_FK(1, 128, 2);
    default: return XMD_FK(1, 128, 4);
    }
#undef XMD_FK
}

// The step kernel's block as it runs: slots and threads per slot.  With 32-slot
// blocks so few that a block's own latency is the kernel's time (mixed: all
// resident at once, four per SM; FP64: one per SM, beyond which the FP64 pipe
// binds), eight threads per slot instead of four: the pair entries go to twice
// the warps.  us per MD step, four -> eight: 61 native chains mixed 26.8 -> 21.5,
// 16 x 500 mixed 20.0 -> 17.2, 67 short chains with contacts FP64 52 -> 47;
// 16 x 500 FP64 (297 blocks) 39 -> 44.
Engine::ForceShape Engine::force_shape() const {
    const bool mixed = params.precision == XMD_PREC_MIXED;
    if (tune.fb == 32 && tune.lpb == 4 && force_blocks(d.N, 32) <= (mixed ? 4 : 1) * tile_sms) return ForceShape{32, 8};
    return ForceShape{tune.fb, tune.lpb};
}
// The shape where none was set: 32-slot blocks up to 16 per SM (two waves at
// four threads per slot), where more and smaller blocks keep the SMs evenly
// loaded; beyond that 64-slot blocks, whose halo is half as large (5 of 64
// slots, not of 32).  us per MD step, 32 / 64 slots: 8,000 beads mixed 17.2 /
// 22.0 and FP64 35.1 / 42.7, 54,744 beads mixed 35.4 / 35.9, 66,007 beads mixed
// 44.0 / 42.0; FP64 hardly minds there (141.8 / 143.7), so the line lies where
// mixed turns.
void Engine::default_shape() {
    if (!tuned) tune.fb = force_blocks(d.N, 32) <= 16 * tile_sms ? 32 : 64;
}

void Engine::launch_force(int mode, int c) {
    if (tp.ext_on) {
        if (mode == 0) k_ext<0><<<(d.N + 255) / 256, 256, 0, stream>>>(d, tp, c);
        else k_ext<1><<<(d.N + 255) / 256, 256, 0, stream>>>(d, tp, c);
    }
    if (tp.on[XMD_TERM_PID]) {
        if (mode == 0) k_pid<0><<<(d.N + 127) / 128, 128, 0, stream>>>(d, tp, c);
        else k_pid<1><<<(d.N + 127) / 128, 128, 0, stream>>>(d, tp, c);
    }
    const ForceShape fs = mode == 0 ? ForceShape{EVAL_FB, EVAL_LPB} : force_shape();
    const int fb = fs.fb, lpb = fs.lpb;
    const int nb = force_blocks(d.N, fb);
    int fuse = FUSE_NONE;
    void *args[] = {&d, &tp, &c, &fuse};
    const bool mixed = params.precision == XMD_PREC_MIXED;
    void *fk = force_kernel(mixed, mode, fb, lpb);
    const size_t smem = force_smem(mixed, mode, fb, d.qa_on);
    if (smem > 48 * 1024) allow_smem(fk, force_smem(mixed, mode, fb, true));
    CK(cudaLaunchKernel(fk, dim3(nb), dim3(fb * lpb), args, smem, stream));
}

void Engine::split_positions() {
    if (params.precision != XMD_PREC_MIXED && !d.qa_on) return;
    // a context that was FP64 until now allocates them here (an allocation
    // enqueues the array's clearing on the step stream)
    for (auto &x : d.spl)
        if (!x) x = (float4 *)dalloc(2 * sizeof(float4) * (size_t)d.N);
    k_split<<<(d.N + 255) / 256, 256, 0, stream>>>(d, cur);
    ++launches;
}

Engine::Engine(const xmd_params &p) : params(p) {
    int ndev = 0;
    CK(cudaGetDeviceCount(&ndev));
    if (ndev < 1) throw std::runtime_error("no CUDA device");
    device = p.device;
    if (device < 0 || device >= ndev) throw std::invalid_argument("engine: device out of range");
    use_device();
    CK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    CK(cudaStreamCreateWithFlags(&ustream, cudaStreamNonBlocking));
    CK(cudaEventCreateWithFlags(&ev_staged, cudaEventDisableTiming));
    CK(cudaEventCreateWithFlags(&ev_removed, cudaEventDisableTiming));
    CK(cudaMallocHost(&h_any, sizeof(int) * 16 + sizeof(double) * XMD_NUM_TERMS));
    for (auto &e : down_ev) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    ring.s = stream;
    uring.s = ustream;
}

char *Engine::HostRing::take(size_t bytes) {
    bytes = (bytes + 15) & ~(size_t)15;
    if (bytes > HALF) throw std::logic_error("engine: copy larger than its staging memory");
    if (!h) {
        CK(cudaMallocHost(&h, 2 * HALF));
        for (auto &e : ev) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    if (off + bytes > HALF) {
        CK(cudaEventRecord(ev[cur], s));
        cur ^= 1;
        CK(cudaEventSynchronize(ev[cur]));
        off = 0;
    }
    char *p = h + cur * HALF + off;
    off += bytes;
    return p;
}

void Engine::HostRing::up(void *dst, const void *src, size_t bytes) {
    for (size_t o = 0; o < bytes; o += HALF) {
        const size_t m = std::min(HALF, bytes - o);
        char *p = take(m);
        std::memcpy(p, (const char *)src + o, m);
        CK(cudaMemcpyAsync((char *)dst + o, p, m, cudaMemcpyHostToDevice, s));
    }
}

Engine::HostRing::~HostRing() {
    if (h) cudaFreeHost(h);
    for (auto &e : ev)
        if (e) cudaEventDestroy(e);
}

void Engine::fetch_words() {
    CK(cudaMemcpyAsync(h_any, d.any_rebuild, sizeof(int) * 16, cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
}

void Engine::down(void *dst, const void *src, size_t bytes) {
    constexpr size_t PIECE = HostRing::HALF / 2 + 16;   // two pieces never share a half
    char *p[2] = {nullptr, nullptr};
    size_t len[2] = {0, 0}, at = 0;
    for (size_t o = 0, k = 0; o < bytes + PIECE; o += PIECE, ++k) {
        if (o < bytes) {
            len[k & 1] = std::min(PIECE, bytes - o);
            p[k & 1] = ring.take(len[k & 1]);
            CK(cudaMemcpyAsync(p[k & 1], (const char *)src + o, len[k & 1], cudaMemcpyDeviceToHost, stream));
            CK(cudaEventRecord(down_ev[k & 1], stream));
        }
        if (k && at < bytes) {
            const int q = (k - 1) & 1;
            CK(cudaEventSynchronize(down_ev[q]));
            std::memcpy((char *)dst + at, p[q], len[q]);
            at += len[q];
        }
    }
}

Engine::~Engine() {
    cudaSetDevice(device);
    for (auto &kv : graphs) {
        if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
        if (kv.second.graph) cudaGraphDestroy(kv.second.graph);
    }
    for (auto e : ev_force) cudaEventDestroy(e);
    for (auto e : ev_rebuild) cudaEventDestroy(e);
    release();
    if (h_any) cudaFreeHost(h_any);
    for (auto e : down_ev)
        if (e) cudaEventDestroy(e);
    if (ev_staged) cudaEventDestroy(ev_staged);
    if (ev_removed) cudaEventDestroy(ev_removed);
    if (ustream) cudaStreamDestroy(ustream);
    if (stream) cudaStreamDestroy(stream);
}

void *Engine::dalloc(size_t bytes) {
    void *p = nullptr;
    CK(cudaMalloc(&p, bytes < 16 ? 16 : bytes));
    CK(cudaMemsetAsync(p, 0, bytes < 16 ? 16 : bytes, stream));
    allocs.push_back(p);
    alloc_bytes += bytes < 16 ? 16 : bytes;
    return p;
}

void Engine::release() {
    for (void *p : allocs) cudaFree(p);
    allocs.clear();
    alloc_bytes = 0;
    d = Dev{};
    finalized = false;
}

int Engine::add_replica(int n, const int32_t *chain, const int32_t *seq, const uint8_t *atype,
                        const double cell[3], double temperature, uint64_t seed) {
    if (finalized && !dynamic)
        throw std::invalid_argument("replicas must be added before the first eval/step (or reserve capacity)");
    if (n <= 0 || n > NL_MASK) throw std::invalid_argument("bead count out of range");
    if (!chain || !seq || !atype) throw std::invalid_argument("null topology array");
    RepHost r;
    r.n = n;
    r.chain.assign(chain, chain + n);
    r.seq.assign(seq, seq + n);
    r.atype.assign(atype, atype + n);
    for (int i = 0; i < n; ++i)
        if (atype[i] >= XMD_NUM_AA) throw std::invalid_argument("atype out of range (0..19)");
    for (int a = 0; a < 3; ++a) {
        r.cell[a] = cell ? cell[a] : 0.0;
        if (r.cell[a] < 0 || !std::isfinite(r.cell[a])) throw std::invalid_argument("bad cell");
    }
    r.temperature = temperature > 0 ? temperature : params.temperature;
    r.seed = seed;
    const double nan = std::nan("");
    r.teth_r0.assign(n, nan);
    r.ang_t0.assign(n, nan);
    r.dih_p0.assign(n, nan);
    r.chir_f.assign(n, nan);
    r.chir_n.assign(n, nan);
    r.hang_t.assign(n, -1);
    r.hdih_t.assign(n, -1);
    if (dynamic) {
        // reuse a free slot; the replica is placed at the next eval/step
        for (int k = 0; k < (int)reps.size(); ++k)
            if (!reps[k].in_use) {
                reps[k] = std::move(r);
                return k;
            }
        if ((int)reps.size() >= cap.reps) throw std::length_error("engine: every reserved replica slot is taken");
    }
    reps.push_back(std::move(r));
    return (int)reps.size() - 1;
}

static void check_rep(const std::vector<RepHost> &reps, int rep) {
    if (rep < 0 || rep >= (int)reps.size() || !reps[rep].in_use)
        throw std::invalid_argument("replica id out of range");
}

void Engine::reserve(int beads, int replicas, int natives) {
    if (finalized) throw std::logic_error("reserve must precede the first eval/step");
    if (params.on[XMD_TERM_QA]) throw std::invalid_argument("reserve: the quasi-adiabatic term needs a static context");
    if (beads < 1 || replicas < 1 || natives < 0) throw std::invalid_argument("reserve: bad capacity");
    int nb = 0;
    for (auto &r : reps) nb += r.n;
    if (nb > beads || (int)reps.size() > replicas) throw std::invalid_argument("reserve: replicas already exceed it");
    dynamic = true;
    cap = Caps{};
    cap.beads = beads;
    cap.reps = replicas;
    cap.nat = natives;
    cap.ss = natives;   // disulfide entries share the native budget
    // bucket pool for replicas above the tile limit; chunk slots for the rest
    cap.cells = params.nl_build == XMD_NL_BUILD_TILE ? 0 : std::max(64, 2 * beads);
    cap.chunks = params.nl_build == XMD_NL_BUILD_CELL ? 0 : beads / TL_CH + replicas;
    finalize();
}

void Engine::remove_replica(int rep) {
    check_rep(reps, rep);
    if (!dynamic) throw std::logic_error("remove_replica needs a context with reserved capacity");
    RepHost &r = reps[rep];
    if (r.placed) {
        use_device();
        const int b = r.begin, n = r.n;
        CK(cudaStreamSynchronize(stream));
        CK(cudaMemsetAsync(d.rep_of + b, 0xff, sizeof(int32_t) * n, stream));
        CK(cudaMemsetAsync(d.bflags + b, 0, sizeof(uint32_t) * n, stream));
        CK(cudaMemsetAsync(d.nl_cnt + b, 0, sizeof(int32_t) * n, stream));
        CK(cudaMemsetAsync(d.go_cnt + b, 0, sizeof(int32_t) * n, stream));
        if (r.nat_len) CK(cudaMemsetAsync(d.nat_on + r.nat_off, 0, r.nat_len, stream));
        if (r.chunk_len) CK(cudaMemsetAsync(d.chunks + r.chunk_off, 0xff, sizeof(int2) * r.chunk_len, stream));
        CK(cudaMemsetAsync(d.rep + rep, 0, sizeof(RepDev), stream));
        CK(cudaStreamSynchronize(stream));
        if (r.cell_len) --live_cell;
        for (int i = 0; i < n; ++i) owner_h[b + i] = -1;
        a_beads.release(b, n);
        a_nat.release(r.nat_off, r.nat_len);
        a_ss.release(r.ss_off, r.ss_len);
        CK(cudaMemsetAsync(d.ss_start + b, 0, sizeof(int32_t) * n, stream));
        CK(cudaMemsetAsync(d.ss_end + b, 0, sizeof(int32_t) * n, stream));
        a_cells.release(r.cell_off, r.cell_len);
        a_chunks.release(r.chunk_off, r.chunk_len);
        a_afm.release(r.afm_off, r.afm_len);
        // staged uploads into these ranges wait for the clears above
        CK(cudaEventRecord(ev_removed, stream));
    } else if (r.staged) {
        // staged, never activated: its uploads are ordered before any later
        // staging on the side stream, so its ranges can be reused at once
        for (size_t q = 0; q < staged_reps.size(); ++q)
            if (staged_reps[q].k == rep) {
                staged_reps.erase(staged_reps.begin() + (long)q);
                break;
            }
        a_beads.release(r.begin, r.n);
        a_nat.release(r.nat_off, r.nat_len);
        a_ss.release(r.ss_off, r.ss_len);
        a_cells.release(r.cell_off, r.cell_len);
        a_chunks.release(r.chunk_off, r.chunk_len);
        a_afm.release(r.afm_off, r.afm_len);
    }
    r = RepHost{};
    r.in_use = false;
}

void Engine::stage(int rep) {
    check_rep(reps, rep);
    if (!dynamic) throw std::logic_error("stage needs a context with reserved capacity");
    ready_alloc();
    RepHost &r = reps[rep];
    if (r.placed || r.staged) return;
    if (!r.have_state) throw std::logic_error("set_state must precede placement");
    use_device();
    Staged st;
    place(rep, &st);
    staged_reps.push_back(std::move(st));
}

void Engine::activate_staged() {
    if (staged_reps.empty()) return;
    use_device();
    CK(cudaEventRecord(ev_staged, ustream));
    CK(cudaStreamWaitEvent(stream, ev_staged, 0));
    for (Staged &st : staged_reps) {
        RepHost &r = reps[st.k];
        ring.up(d.rep_of + r.begin, st.rep_of.data(), sizeof(int32_t) * r.n);
        ring.up(d.rep + st.k, &st.rd, sizeof(RepDev));
        for (int i = 0; i < r.n; ++i) owner_h[r.begin + i] = st.k;
        r.staged = false;
        r.placed = true;
        if (r.cell_len) ++live_cell;
    }
    staged_reps.clear();
}

void Engine::step_async(int nsteps) {
    use_device();
    ready();
    if (!params.langevin_on) throw std::invalid_argument("langevin: enabled is false; nothing integrates");
    ensure_nl();
    split_positions();
    int s = 0;
    if (!timing && use_graphs) {
        const int gsteps = tune.graph_steps;
        // launches per step of each graph form: the step kernel, plus the
        // quasi-adiabatic kernels with that term, the external-force and PID
        // kernels, and the plain form's row-build node or the IF form's
        // separate check (gated QA graphs take the decision in the
        // re-freeing kernel); rebuild kernels of IF nodes and of the host's
        // rebuilds are counted per pass in stats()
        const int64_t extra = (tp.ext_on ? 1 : 0) + (tp.on[XMD_TERM_PID] ? 1 : 0);
        const int64_t per_plain = 2 + extra, per_gated = (d.qa_on ? 5 : 1) + extra,
                      per_cond = (d.qa_on ? 6 : 2) + extra;
        // graphs of graph_steps steps, and the rest in graphs of the largest
        // powers of two that fit
        auto chunk = [&](int left) {
            if (left >= gsteps) return gsteps;
            int l = 1;
            while (2 * l <= left) l *= 2;
            return l;
        };
        if (gated_graphs()) {
            // each graph runs until a check flags a replica (or its steps are
            // done); the host then rebuilds and goes on from the steps taken.
            // While rebuilds come every few steps (a relaxing start) the
            // halted steps would be launches for nothing: graphs with IF
            // rebuild nodes run instead for a while.  The gate is open
            // outside the gated graphs (per-launch steps read it).
            struct Open {
                Engine *e;
                ~Open() { cudaMemsetAsync(e->d.gate, 0, sizeof(int) * 3, e->stream); }
            } open_gate{this};
            while (s < nsteps) {
                const int len = chunk(nsteps - s);
                if (cond_graphs_left > 0) {
                    CK(cudaGraphLaunch(graph_for(cur, false, len), stream));
                    launches += per_cond * len;
                    md_steps += len;
                    s += len;
                    cur ^= len & 1;
                    --cond_graphs_left;
                    continue;
                }
                h_any[0] = 0; h_any[1] = 0; h_any[2] = 0; h_any[3] = len;
                CK(cudaMemcpyAsync(d.any_rebuild, h_any, sizeof(int) * 4, cudaMemcpyHostToDevice, stream));
                CK(cudaGraphLaunch(graph_for(cur, true, len), stream));
                CK(cudaMemcpyAsync(h_any, d.any_rebuild, sizeof(int) * 4, cudaMemcpyDeviceToHost, stream));
                CK(cudaStreamSynchronize(stream));
                const int done = h_any[2];
                if (done < 1 || done > len) throw std::logic_error("engine: graph step count out of range");
                CK(cudaMemsetAsync(d.gate, 0, sizeof(int) * 3, stream));   // open for what follows
                launches += per_gated * len;
                md_steps += done;
                s += done;
                cur ^= done & 1;
                if (h_any[0]) {
                    launch_rebuild();
                    if (done < len / 4) cond_graphs_left = 8;
                }
            }
        } else {
            const int64_t per = plain_rebuild() ? per_plain : per_cond;
            while (s < nsteps) {
                const int len = chunk(nsteps - s);
                CK(cudaGraphLaunch(graph_for(cur, false, len), stream));
                launches += per * len;
                md_steps += len;
                s += len;
                cur ^= len & 1;
            }
        }
    }
    for (; s < nsteps; ++s) {
        launch_force_step();
        cur ^= 1;
        k_nl_check<<<1, 1024, 0, stream>>>(d, 1, params.dt, (cudaGraphConditionalHandle)0, 0);
        ++launches;
        ++md_steps;
        CK(cudaMemcpyAsync(h_any, d.any_rebuild, sizeof(int), cudaMemcpyDeviceToHost, stream));
        CK(cudaStreamSynchronize(stream));
        if (*h_any) launch_rebuild();
    }
}

void Engine::step_wait() {
    use_device();
    check_status("step");
    if (auto_grow) grow_rows(0.6);
}

void Engine::set_steps(int rep, long long nsteps) {
    check_rep(reps, rep);
    if (params.on[XMD_TERM_QA]) throw std::invalid_argument("per-replica step budgets exclude the quasi-adiabatic term");
    reps[rep].steps_left = nsteps < 0 ? -1 : nsteps;
    if (reps[rep].placed) {
        use_device();
        long long v = reps[rep].steps_left;
        CK(cudaMemcpyAsync((char *)(d.rep + rep) + offsetof(RepDev, steps_left), &v, sizeof v,
                           cudaMemcpyHostToDevice, stream));
        CK(cudaStreamSynchronize(stream));
    }
}

void Engine::place_now(int rep) {
    check_rep(reps, rep);
    ready_alloc();
    if (!reps[rep].placed) {
        if (!reps[rep].have_state) throw std::logic_error("set_state must precede placement");
        use_device();
        place(rep);
    }
}

void Engine::steps_left(long long *out) {
    use_device();
    std::vector<RepDev> rd(std::max(1, d.R));
    if (finalized) {
        CK(cudaMemcpyAsync(rd.data(), d.rep, sizeof(RepDev) * d.R, cudaMemcpyDeviceToHost, stream));
        CK(cudaStreamSynchronize(stream));
    }
    for (int k = 0; k < (int)reps.size(); ++k)
        out[k] = !reps[k].in_use ? -2
                 : (reps[k].placed ? (rd[k].fault ? -3 : rd[k].steps_left) : reps[k].steps_left);
}
static bool consecutive(const RepHost &r, int a, int b) {
    return a >= 0 && b < r.n && b == a + 1 && r.chain[a] == r.chain[b] && r.seq[b] == r.seq[a] + 1;
}

void Engine::set_tethers(int rep, int n, const int32_t *i1, const int32_t *i2, const double *dd) {
    check_rep(reps, rep);
    if (reps[rep].placed) throw std::invalid_argument("topology is fixed once the replica is on the device");
    RepHost &r = reps[rep];
    std::fill(r.teth_r0.begin(), r.teth_r0.end(), std::nan(""));
    for (int k = 0; k < n; ++k) {
        int a = std::min(i1[k], i2[k]), b = std::max(i1[k], i2[k]);
        if (!consecutive(r, a, b)) throw std::invalid_argument("tether is not a bond between consecutive beads of a chain");
        if (!std::isnan(r.teth_r0[a])) throw std::invalid_argument("duplicate tether");
        // tether.length.value_or(def_length), main.cpp:409-413
        r.teth_r0[a] = (dd && dd[k] > 0) ? dd[k] : params.tether_def_length;
    }
}
void Engine::set_angles(int rep, int n, const int32_t *i1, const int32_t *i2, const int32_t *i3,
                        const double *th) {
    check_rep(reps, rep);
    if (reps[rep].placed) throw std::invalid_argument("topology is fixed once the replica is on the device");
    RepHost &r = reps[rep];
    std::fill(r.ang_t0.begin(), r.ang_t0.end(), std::nan(""));
    for (int k = 0; k < n; ++k) {
        if (!consecutive(r, i1[k], i2[k]) || !consecutive(r, i2[k], i3[k]))
            throw std::invalid_argument("angle must be (i-1, i, i+1) of one chain");
        if (!std::isnan(r.ang_t0[i2[k]])) throw std::invalid_argument("duplicate angle");
        if (r.hang_t[i2[k]] >= 0) throw std::invalid_argument("angle is already heuristic");
        if (!std::isfinite(th[k])) throw std::invalid_argument("non-finite native angle");
        r.ang_t0[i2[k]] = th[k];
    }
}
void Engine::set_dihedrals(int rep, int n, const int32_t *i1, const int32_t *i2, const int32_t *i3,
                           const int32_t *i4, const double *ph) {
    check_rep(reps, rep);
    if (reps[rep].placed) throw std::invalid_argument("topology is fixed once the replica is on the device");
    RepHost &r = reps[rep];
    std::fill(r.dih_p0.begin(), r.dih_p0.end(), std::nan(""));
    for (int k = 0; k < n; ++k) {
        if (!consecutive(r, i1[k], i2[k]) || !consecutive(r, i2[k], i3[k]) || !consecutive(r, i3[k], i4[k]))
            throw std::invalid_argument("dihedral must be (i-1, i, i+1, i+2) of one chain");
        if (!std::isnan(r.dih_p0[i2[k]])) throw std::invalid_argument("duplicate dihedral");
        if (r.hdih_t[i2[k]] >= 0) throw std::invalid_argument("dihedral is already heuristic");
        if (!std::isfinite(ph[k])) throw std::invalid_argument("non-finite native dihedral");
        r.dih_p0[i2[k]] = ph[k];
    }
}
void Engine::set_native(int rep, int n, const int32_t *i1, const int32_t *i2, const double *dd) {
    check_rep(reps, rep);
    if (reps[rep].placed) throw std::invalid_argument("topology is fixed once the replica is on the device");
    RepHost &r = reps[rep];
    std::vector<std::tuple<int, int, double>> v;
    for (int k = 0; k < n; ++k) {
        int a = std::min(i1[k], i2[k]), b = std::max(i1[k], i2[k]);
        if (a < 0 || b >= r.n || a == b) throw std::invalid_argument("native contact index out of range");
        if (!(dd[k] > 0)) throw std::invalid_argument("native distance must be positive");
        v.emplace_back(a, b, dd[k]);
    }
    std::sort(v.begin(), v.end());
    for (size_t k = 1; k < v.size(); ++k)
        if (std::get<0>(v[k]) == std::get<0>(v[k - 1]) && std::get<1>(v[k]) == std::get<1>(v[k - 1]))
            throw std::invalid_argument("duplicate native contact");
    r.nat_i1.clear(); r.nat_i2.clear(); r.nat_d.clear();
    for (auto &[a, b, x] : v) { r.nat_i1.push_back(a); r.nat_i2.push_back(b); r.nat_d.push_back(x); }
}

void Engine::set_chirals(int rep, int n, const int32_t *i1, const int32_t *i2, const int32_t *i3,
                         const int32_t *i4, const double *f, const double *c) {
    check_rep(reps, rep);
    if (reps[rep].placed) throw std::invalid_argument("topology is fixed once the replica is on the device");
    RepHost &r = reps[rep];
    std::fill(r.chir_f.begin(), r.chir_f.end(), std::nan(""));
    std::fill(r.chir_n.begin(), r.chir_n.end(), std::nan(""));
    for (int k = 0; k < n; ++k) {
        if (!consecutive(r, i1[k], i2[k]) || !consecutive(r, i2[k], i3[k]) || !consecutive(r, i3[k], i4[k]))
            throw std::invalid_argument("chiral quad must be (i-1, i, i+1, i+2) of one chain");
        if (!std::isnan(r.chir_f[i2[k]])) throw std::invalid_argument("duplicate chiral quad");
        if (!std::isfinite(f[k]) || !std::isfinite(c[k])) throw std::invalid_argument("non-finite chiral parameter");
        r.chir_f[i2[k]] = f[k];
        r.chir_n[i2[k]] = c[k];
    }
}
// heur_ang_type / heur_dih_type: G = 0, P = 1, any other residue = 2,
// type = 3 t1 + t2 (angle/heurestic.cpp:9-15, dihedral/heurestic.cpp:8-14)
static int8_t heur_type(uint8_t a, uint8_t b) {
    auto cls = [](uint8_t x) { return x == 7 ? 0 : (x == 14 ? 1 : 2); };   // GLY, PRO of amino_acid.h:10-13
    return (int8_t)(3 * cls(a) + cls(b));
}
void Engine::set_heuristic_angles(int rep, int n, const int32_t *i1, const int32_t *i2, const int32_t *i3) {
    check_rep(reps, rep);
    if (reps[rep].placed) throw std::invalid_argument("topology is fixed once the replica is on the device");
    RepHost &r = reps[rep];
    std::fill(r.hang_t.begin(), r.hang_t.end(), (int8_t)-1);
    for (int k = 0; k < n; ++k) {
        if (!consecutive(r, i1[k], i2[k]) || !consecutive(r, i2[k], i3[k]))
            throw std::invalid_argument("heuristic angle must be (i-1, i, i+1) of one chain");
        if (r.hang_t[i2[k]] >= 0) throw std::invalid_argument("duplicate heuristic angle");
        if (!std::isnan(r.ang_t0[i2[k]])) throw std::invalid_argument("angle is already native");
        r.hang_t[i2[k]] = heur_type(r.atype[i1[k]], r.atype[i2[k]]);
    }
}
void Engine::set_heuristic_dihedrals(int rep, int n, const int32_t *i1, const int32_t *i2, const int32_t *i3,
                                     const int32_t *i4) {
    check_rep(reps, rep);
    if (reps[rep].placed) throw std::invalid_argument("topology is fixed once the replica is on the device");
    RepHost &r = reps[rep];
    std::fill(r.hdih_t.begin(), r.hdih_t.end(), (int8_t)-1);
    for (int k = 0; k < n; ++k) {
        if (!consecutive(r, i1[k], i2[k]) || !consecutive(r, i2[k], i3[k]) || !consecutive(r, i3[k], i4[k]))
            throw std::invalid_argument("heuristic dihedral must be (i-1, i, i+1, i+2) of one chain");
        if (r.hdih_t[i2[k]] >= 0) throw std::invalid_argument("duplicate heuristic dihedral");
        if (!std::isnan(r.dih_p0[i2[k]])) throw std::invalid_argument("dihedral is already native");
        r.hdih_t[i2[k]] = heur_type(r.atype[i2[k]], r.atype[i3[k]]);
    }
}
void Engine::set_velocity_afm(int rep, int n, const int32_t *bead, const double *orig, const double *vel) {
    check_rep(reps, rep);
    if (reps[rep].placed) throw std::invalid_argument("topology is fixed once the replica is on the device");
    if (dynamic) throw std::invalid_argument("AFM tips need a static context");
    RepHost &r = reps[rep];
    std::vector<int32_t> seen;
    for (int k = 0; k < n; ++k) {
        if (bead[k] < 0 || bead[k] >= r.n) throw std::invalid_argument("AFM tip bead out of range");
        if (std::find(seen.begin(), seen.end(), bead[k]) != seen.end())
            throw std::invalid_argument("one velocity AFM tip per bead");
        seen.push_back(bead[k]);
        for (int a = 0; a < 3; ++a)
            if (!std::isfinite(vel[3 * k + a]) || std::isinf(orig[3 * k + a]))
                throw std::invalid_argument("non-finite AFM tip");
    }
    r.vafm_i.assign(bead, bead + n);
    r.vafm_o.assign(orig, orig + 3 * n);
    r.vafm_v.assign(vel, vel + 3 * n);
}
void Engine::set_force_afm(int rep, int n, const int32_t *bead, const double *F) {
    check_rep(reps, rep);
    if (reps[rep].placed) throw std::invalid_argument("topology is fixed once the replica is on the device");
    if (dynamic) throw std::invalid_argument("AFM tips need a static context");
    RepHost &r = reps[rep];
    for (int k = 0; k < n; ++k) {
        if (bead[k] < 0 || bead[k] >= r.n) throw std::invalid_argument("AFM tip bead out of range");
        for (int a = 0; a < 3; ++a)
            if (!std::isfinite(F[3 * k + a])) throw std::invalid_argument("non-finite AFM force");
    }
    r.fafm_i.assign(bead, bead + n);
    r.fafm_F.assign(F, F + 3 * n);
}
void Engine::set_walls(int kind, int n, const double *origin, const double *normal) {
    if (kind != 0 && kind != 1) throw std::invalid_argument("wall kind must be 0 (solid) or 1 (LJ attractive)");
    if (n < 0 || n > XMD_MAX_WALLS) throw std::invalid_argument("at most XMD_MAX_WALLS planes per wall kind");
    if (finalized) throw std::invalid_argument("walls are set before the first replica is placed");
    std::vector<double> w;
    for (int k = 0; k < n; ++k) {
        for (int a = 0; a < 3; ++a)
            if (!std::isfinite(origin[3 * k + a]) || !std::isfinite(normal[3 * k + a]))
                throw std::invalid_argument("non-finite wall plane");
        for (int a = 0; a < 3; ++a) w.push_back(origin[3 * k + a]);
        for (int a = 0; a < 3; ++a) w.push_back(normal[3 * k + a]);
    }
    walls[kind] = w;
}
// beads of replica r pulled by some AFM tip, in order
static std::vector<int> afm_beads(const RepHost &r) {
    std::vector<int> v(r.vafm_i.begin(), r.vafm_i.end());
    v.insert(v.end(), r.fafm_i.begin(), r.fafm_i.end());
    std::sort(v.begin(), v.end());
    v.erase(std::unique(v.begin(), v.end()), v.end());
    return v;
}
void Engine::set_ssbonds(int rep, int n, const int32_t *i1, const int32_t *i2) {
    check_rep(reps, rep);
    if (reps[rep].placed) throw std::invalid_argument("topology is fixed once the replica is on the device");
    RepHost &r = reps[rep];
    std::vector<std::pair<int, int>> v;
    for (int k = 0; k < n; ++k) {
        int a = std::min(i1[k], i2[k]), b = std::max(i1[k], i2[k]);
        if (a < 0 || b >= r.n || a == b) throw std::invalid_argument("disulfide index out of range");
        v.emplace_back(a, b);
    }
    std::sort(v.begin(), v.end());
    if (std::adjacent_find(v.begin(), v.end()) != v.end()) throw std::invalid_argument("duplicate disulfide");
    r.ss_i1.clear(); r.ss_i2.clear();
    for (auto &[a, b] : v) { r.ss_i1.push_back(a); r.ss_i2.push_back(b); }
}

void Engine::derive_rep(int ri, RepDev &rd) {
    const RepHost &r = reps[ri];
    const xmd_params &p = params;
    std::memset(&rd, 0, sizeof rd);
    for (int a = 0; a < 3; ++a) {
        rd.box.cell[a] = r.cell[a];
        rd.box.cell_inv[a] = r.cell[a] != 0.0 ? 1.0 / r.cell[a] : 0.0;   // box.h:12-22
        rd.per[a] = r.cell[a] != 0.0;
        rd.per_any |= rd.per[a];
        // the length as h + l, both truncated as split_d's
        auto leading = [](double x) {
            uint64_t u;
            std::memcpy(&u, &x, 8);
            u &= ~0x1fffffffull;
            std::memcpy(&x, &u, 8);
            return x;
        };
        const double h = leading(r.cell[a]);
        rd.Lh[a] = (float)h;
        rd.Ll[a] = (float)leading(r.cell[a] - h);
        rd.Li[a] = (float)rd.box.cell_inv[a];
    }
    // max_cutoff: main.cpp:500, 545-551, 628-630, 642-644, 742-746
    double mc = 0.0;
    if (p.on[XMD_TERM_PAULI]) mc = std::max(mc, p.pauli_r_excl);
    if (p.on[XMD_TERM_NAT_SS]) mc = std::max(mc, 2.0 * p.nat_ss_dist);   // harmonic::cutoff, main.cpp:596-597
    if (p.on[XMD_TERM_GO]) for (double x : r.nat_d) mc = std::max(mc, 2.0 * x);
    if (p.on[XMD_TERM_CONST_ES]) mc = std::max(mc, 2.0 * p.const_es_screen_dist);
    if (p.on[XMD_TERM_REL_ES]) mc = std::max(mc, 2.0 * p.rel_es_screen_dist);
    // max req_min_dist over contact types (main.cpp:742-746), also the
    // intended max_formation_min_dist of update_free_pairs
    double max_form = std::max(p.lj_bb_r_min, p.lj_bs_r_min);
    for (int k = 0; k < XMD_NUM_SS; ++k) max_form = std::max(max_form, p.ss_r_max[k]);
    if (p.on[XMD_TERM_QA]) mc = std::max(mc, max_form);
    // PID bundles: the largest LJ-variant cutoff (lj::cutoff = 2 r_min,
    // sink_lj::cutoff = 2 r_max), main.cpp:801-810
    double pid_cut = std::max(2.0 * p.lj_bb_r_min, 2.0 * p.lj_bs_r_min);
    for (int k = 0; k < XMD_NUM_SS; ++k) pid_cut = std::max(pid_cut, 2.0 * p.ss_r_max[k]);
    if (p.on[XMD_TERM_PID]) mc = std::max(mc, pid_cut);
    if (p.nl_cutoff > 0.0) mc = p.nl_cutoff;
    rd.pad = p.nl_skin > 0.0 ? p.nl_skin : p.pad_factor * mc;   // legacy_update.cpp:7-8
    rd.req_r = mc + rd.pad;
    double es_cut = p.on[XMD_TERM_CONST_ES] ? 2.0 * p.const_es_screen_dist : 2.0 * p.rel_es_screen_dist;
    rd.es_min_inv = 1.0 / (es_cut + rd.pad);                      // es_pair.cpp:9
    rd.pauli_min_inv = 1.0 / (p.pauli_r_excl + rd.pad);           // pauli.cpp:12-13
    rd.qa_min_inv = 1.0 / (max_form + rd.pad);                     // free_pair.cpp:9-10
    rd.pid_min_inv = 1.0 / (pid_cut + rd.pad);                     // pid/bundle.cpp:9-12
    rd.s_req = sq_below(rd.req_r);
    rd.s_pa = sq_below(inv_above(rd.pauli_min_inv));
    rd.s_es = sq_below(inv_above(rd.es_min_inv));
    rd.s_qa = sq_below(inv_above(rd.qa_min_inv));
    rd.s_pid = sq_below(inv_above(rd.pid_min_inv));
    // the near grid's radius: the largest of the terms that act between any
    // two beads; the far grid's: the electrostatic one
    auto near_term = [&](double radius, double s) {
        rd.r_near = std::max(rd.r_near, std::min(radius, rd.req_r));
        rd.s_near = std::max(rd.s_near, std::min(s, rd.s_req));
    };
    if (p.on[XMD_TERM_PAULI]) near_term(1.0 / rd.pauli_min_inv, rd.s_pa);
    if (p.on[XMD_TERM_QA]) near_term(1.0 / rd.qa_min_inv, rd.s_qa);
    if (p.on[XMD_TERM_PID]) near_term(1.0 / rd.pid_min_inv, rd.s_pid);
    if (rd.r_near <= 0.0) rd.r_near = rd.req_r > 0.0 ? rd.req_r : 1.0;
    rd.far = (p.on[XMD_TERM_CONST_ES] || p.on[XMD_TERM_REL_ES]) && rd.req_r > 0.0;
    rd.r_far = rd.far ? std::min(1.0 / rd.es_min_inv, rd.req_r) : 1.0;
    rd.s_ss = sq_below(2.0 * p.nat_ss_dist + rd.pad);   // update_nat_ssbonds, native_ss.cpp:15
    rd.noise_sd = std::sqrt(2.0 * 1.0 * r.temperature) * std::sqrt(p.gamma_factor) * 1.0;
    rd.begin = r.begin;
    rd.n = r.n;
    rd.first = 1;
}

// Capacities: exact totals of the replicas added so far (static contexts), or
// the reservation (dynamic contexts, where replicas come and go between steps).
void Engine::finalize() {
    if (finalized) return;
    if (!dynamic) {
        if (reps.empty()) throw std::logic_error("no replica added");
        for (auto &r : reps)
            if (!r.have_state) throw std::logic_error("set_state must be called for every replica");
        cap = Caps{};
        cap.reps = (int)reps.size();
        for (auto &r : reps) {
            cap.beads += r.n;
            cap.nat += 2 * (int)r.nat_i1.size();
            cap.ss += 2 * (int)r.ss_i1.size();
            cap.afm += (int)afm_beads(r).size();
            const bool tile = params.nl_build == XMD_NL_BUILD_TILE ||
                              (params.nl_build == XMD_NL_BUILD_AUTO && r.n <= TILE_MAX);
            if (tile) cap.chunks += (r.n + TL_CH - 1) / TL_CH;
            else cap.cells += std::max(64, 2 * r.n);
            if (params.on[XMD_TERM_QA]) {
                cap.fp += r.n * QA_FP_PER_BEAD + 256;
                cap.qab += (r.n + QA_BCHUNK - 1) / QA_BCHUNK;
                cap.ct += r.n * QA_CT_PER_BEAD + 256;
            }
        }
    }
    allocate();
    finalized = true;
    place_pending();
}

// every device array at capacity; slots start empty (rep_of = -1)
void Engine::allocate() {
    const xmd_params &p = params;
    const int N = cap.beads, R = cap.reps;
    if (N > NL_MASK) throw std::invalid_argument("the context holds more beads than a Verlet entry can index");
    nl_cap = p.nl_capacity > 0 ? p.nl_capacity : 64;
    auto_grow = p.nl_grow != 0;
    d.N = N;
    d.R = R;
    d.nl_cap = nl_cap;
    // near grids, then the far grids at half their size
    const size_t cells = (size_t)std::max(1, cap.cells) / 2 * 3 + 3;
    const size_t NN = (size_t)std::max(1, cap.nat);
    d.pos[0] = (double4_32a *)dalloc(sizeof(double4_32a) * N);
    d.pos[1] = (double4_32a *)dalloc(sizeof(double4_32a) * N);
    // nothing else reads split positions (a later change of the precision:
    // split_positions)
    if (p.precision == XMD_PREC_MIXED || p.on[XMD_TERM_QA])
        for (auto &x : d.spl) x = (float4 *)dalloc(2 * sizeof(float4) * N);
    d.yh = (double *)dalloc(sizeof(double) * 15 * (size_t)N);
    d.orig = (double4_32a *)dalloc(sizeof(double4_32a) * N);
    d.F = (double *)dalloc(sizeof(double) * 3 * (size_t)N);
    d.Vrep = (double *)dalloc(sizeof(double) * XMD_NUM_TERMS * R);
    d.rep_of = (int32_t *)dalloc(sizeof(int32_t) * N);
    CK(cudaMemsetAsync(d.rep_of, 0xff, sizeof(int32_t) * N, stream));
    d.bflags = (uint32_t *)dalloc(sizeof(uint32_t) * N);
    d.chain = (int32_t *)dalloc(sizeof(int32_t) * N);
    d.seq = (int32_t *)dalloc(sizeof(int32_t) * N);
    d.atype = (uint8_t *)dalloc(N);
    d.teth_r0 = (double *)dalloc(sizeof(double) * N);
    d.ang_t0 = (double *)dalloc(sizeof(double) * N);
    d.dih_p0 = (double *)dalloc(sizeof(double) * N);
    d.dih_cs = (double2 *)dalloc(sizeof(double2) * N);
    d.bond_f = (float4 *)dalloc(sizeof(float4) * N);
    d.nat_start = (int32_t *)dalloc(sizeof(int32_t) * N);
    d.nat_end = (int32_t *)dalloc(sizeof(int32_t) * N);
    d.nat_j = (int32_t *)dalloc(sizeof(int32_t) * NN);
    d.nat_d = (double *)dalloc(sizeof(double) * NN);
    d.nat_on = (uint8_t *)dalloc(NN);
    d.act_j = (int32_t *)dalloc(sizeof(int32_t) * NN);
    d.act_d = (double *)dalloc(sizeof(double) * NN);
    d.go_cnt = (int32_t *)dalloc(sizeof(int32_t) * N);
    {
        const size_t SS = (size_t)std::max(1, cap.ss);
        d.ss_start = (int32_t *)dalloc(sizeof(int32_t) * N);
        d.ss_end = (int32_t *)dalloc(sizeof(int32_t) * N);
        CK(cudaMemsetAsync(d.ss_start, 0, sizeof(int32_t) * N, stream));
        CK(cudaMemsetAsync(d.ss_end, 0, sizeof(int32_t) * N, stream));
        d.ss_j = (int32_t *)dalloc(sizeof(int32_t) * SS);
        d.ss_on = (uint8_t *)dalloc(SS);
        CK(cudaMemsetAsync(d.ss_on, 0, SS, stream));
        if (p.on[XMD_TERM_CHIR]) {
            d.chir = (double2 *)dalloc(sizeof(double2) * N);
            d.chir_f32 = (float2 *)dalloc(sizeof(float2) * N);
        }
        d.afm = (AfmTip *)dalloc(sizeof(AfmTip) * (size_t)std::max(1, cap.afm));
        // wall planes, and the state of every (bead, LJ attractive wall) pair
        double wt[2 * XMD_MAX_WALLS * 6] = {0};
        for (int kind = 0; kind < 2; ++kind)
            for (size_t q = 0; q < walls[kind].size(); ++q) wt[kind * XMD_MAX_WALLS * 6 + q] = walls[kind][q];
        d.wall = (double *)dalloc(sizeof(wt));
        CK(cudaMemcpyAsync(d.wall, wt, sizeof(wt), cudaMemcpyHostToDevice, stream));
        const size_t nlj = walls[1].size() / 6;
        d.ljw = (LjWallState *)dalloc(sizeof(LjWallState) * std::max<size_t>(1, nlj * N));
        CK(cudaMemsetAsync(d.ljw, 0, sizeof(LjWallState) * std::max<size_t>(1, nlj * N), stream));
        CK(cudaStreamSynchronize(stream));
    }
    {
        // heuristic coefficient tables: constants of the context
        double *ha = (double *)dalloc(sizeof(double) * 9 * 7);
        double *hd = (double *)dalloc(sizeof(double) * 9 * 6);
        float *hdf = (float *)dalloc(sizeof(float) * 9 * 6);
        float tf[9 * 6];
        for (int k = 0; k < 9 * 6; ++k) tf[k] = (float)(&params.heur_dih_coeffs[0][0])[k];
        CK(cudaMemcpyAsync(ha, &params.heur_ang_coeffs[0][0], sizeof(double) * 9 * 7, cudaMemcpyHostToDevice, stream));
        CK(cudaMemcpyAsync(hd, &params.heur_dih_coeffs[0][0], sizeof(double) * 9 * 6, cudaMemcpyHostToDevice, stream));
        CK(cudaMemcpyAsync(hdf, tf, sizeof(float) * 9 * 6, cudaMemcpyHostToDevice, stream));
        CK(cudaStreamSynchronize(stream));
        d.heur_ang = ha; d.heur_dih = hd; d.heur_dih_f = hdf;
        // radius_of: c is the middle of interval j of 128 in [1, 2), halved in
        // the upper half, 1 beside 1
        double2 lt[128];
        for (int j = 0; j < 128; ++j) {
            const double mid = 1.0 + (j + 0.5) / 128.0;
            const double inv = j == 0 || j == 127 ? 1.0 : 1.0 / (j < 64 ? mid : 0.5 * mid);
            lt[j] = make_double2(inv, (double)-logl((long double)inv));
        }
        double2 *ltd = (double2 *)dalloc(sizeof lt);
        CK(cudaMemcpyAsync(ltd, lt, sizeof lt, cudaMemcpyHostToDevice, stream));
        CK(cudaStreamSynchronize(stream));
        d.logt = ltd;
    }
    d.nl_row = (int32_t *)dalloc(sizeof(int32_t) * (size_t)nl_cap * N);
    d.nl_cnt = (int32_t *)dalloc(sizeof(int32_t) * N);
    d.cell_cnt = (int32_t *)dalloc(sizeof(int32_t) * cells);
    d.cell_start = (int32_t *)dalloc(sizeof(int32_t) * cells);
    d.ncells = (int)cells;
    d.ncells_near = (int)cells / 3 * 2;
    d.cell_base = (int32_t *)dalloc(sizeof(int32_t) * ((cells + CELL_SCAN - 1) / CELL_SCAN + 1));
    // both grids' slots, where some replica may use them
    const size_t slots = cap.cells > 0 ? 2 * (size_t)N : 1;
    d.cell_items = (int32_t *)dalloc(sizeof(int32_t) * slots);
    d.cell_key = (int32_t *)dalloc(sizeof(int32_t) * slots);
    d.cell_pos = (float4 *)dalloc(sizeof(float4) * slots);
    d.rng = (uint64_t *)dalloc(sizeof(uint64_t) * N);
    d.jump = (uint64_t *)dalloc(sizeof(uint64_t) * JUMP_WORDS * R);
    d.rep = (RepDev *)dalloc(sizeof(RepDev) * R);
    d.any_rebuild = (int *)dalloc(sizeof(int) * 16);   // one block: the host reads it with one copy
    d.gate = d.any_rebuild + 1;
    d.status = d.any_rebuild + 4;
    d.ctr = (unsigned long long *)(d.any_rebuild + 8);
    // jumps of the generator by 4 2^l draws (bead i starts 4 i draws after the
    // seed), as nibble tables: entry [q][v] = XOR of the columns 4q + b for
    // the bits b of v
    rng_levels = 1;
    while (N >> rng_levels) ++rng_levels;
    rng_pow = (uint64_t *)dalloc(sizeof(uint64_t) * JUMP_WORDS * rng_levels);
    std::vector<uint64_t> jt((size_t)JUMP_WORDS * rng_levels);
    GF2 jm = gf2_jump(4);
    for (int l = 0; l < rng_levels; ++l) {
        for (int q = 0; q < 16; ++q)
            for (int v = 0; v < 16; ++v) {
                uint64_t e = 0;
                for (int bb = 0; bb < 4; ++bb)
                    if ((v >> bb) & 1) e ^= jm[4 * q + bb];
                jt[(size_t)JUMP_WORDS * l + 16 * q + v] = e;
            }
        jm = gf2_mul(jm, jm);
    }
    ring.up(rng_pow, jt.data(), sizeof(uint64_t) * jt.size());
    if (dynamic) uring.take(0);   // both rings exist before the first step
    d.nchunks = std::max(1, cap.chunks);
    d.chunks = (int2 *)dalloc(sizeof(int2) * d.nchunks);
    d.work = (int *)dalloc(sizeof(int) * d.nchunks);
    d.nwork = (int *)dalloc(sizeof(int));
    CK(cudaMemsetAsync(d.nwork, 0, sizeof(int), stream));
    CK(cudaMemsetAsync(d.chunks, 0xff, sizeof(int2) * d.nchunks, stream));
    owner_h.assign(N, -1);
    a_beads.init(N);
    a_nat.init(cap.nat);
    a_ss.init(cap.ss);
    if (cap.afm > AFM_MAX_TIPS) throw std::length_error("engine: more AFM-pulled beads than the tip table holds");
    a_afm.init(cap.afm);
    a_cells.init(cap.cells);
    a_chunks.init(cap.chunks);
    a_fp.init(cap.fp);
    a_ct.init(cap.ct);
    any_tile = cap.chunks > 0;
    live_cell = 0;
    tile_smem = 0;
    for (auto &r : reps)
        if (r.in_use && r.n <= TILE_MAX) tile_smem = std::max(tile_smem, tile_bytes(r.n));
    if (dynamic) tile_smem = tile_bytes(std::min(TILE_MAX, cap.beads));
    if (tile_smem > 48 * 1024)
        allow_smem((const void *)k_nl_tile, tile_bytes(TILE_MAX));
    {
        // the tile build runs as many blocks as are resident at once (or the
        // tuned number per SM); they take the work list's chunks in turn
        int sms = 0, per_sm = 0;
        CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_nl_tile, TL_THREADS, tile_smem));
        tile_sms = std::max(1, sms);
        tile_max_per_sm = std::max(1, per_sm);
        const int k = tune.tile_per_sm > 0 ? std::min(tune.tile_per_sm, tile_max_per_sm) : tile_max_per_sm;
        tile_grid = std::max(1, std::min(d.nchunks, tile_sms * k));
    }
    default_shape();

    // term parameters
    std::memset(&tp, 0, sizeof tp);
    for (int k = 0; k < XMD_NUM_TERMS; ++k) tp.on[k] = p.on[k];
    tp.dt = p.dt;
    tp.dt_inv = 1.0 / p.dt;
    tp.dt2_half = p.dt * p.dt / 2.0;
    tp.gamma_factor = p.gamma_factor;
    tp.tether_H1 = p.tether_H1; tp.tether_H2 = p.tether_H2;
    tp.nat_ang_k = p.nat_ang_k; tp.cnd_CDA = p.cnd_CDA; tp.cnd_CDB = p.cnd_CDB; tp.snd_CDH = p.snd_CDH;
    tp.go_depth = p.go_depth;
    tp.pauli_r_excl = p.pauli_r_excl; tp.pauli_depth = p.pauli_depth;
    if (p.on[XMD_TERM_CONST_ES]) {      // main.cpp:619-631
        tp.es_Vf = 1.0 / (4.0 * M_PI * p.const_es_permittivity);
        tp.es_sdi = 1.0 / p.const_es_screen_dist;
        tp.es_rel = 0;
    } else {                            // main.cpp:633-645
        tp.es_Vf = 1.0 / (4.0 * M_PI * p.rel_es_factor);
        tp.es_sdi = 1.0 / p.rel_es_screen_dist;
        tp.es_rel = 1;
    }
    if (p.on[XMD_TERM_CONST_ES] && p.on[XMD_TERM_REL_ES])
        throw std::invalid_argument("const ES and relative ES cannot both be enabled in this engine");
    tp.qa_cycle = p.qa_phase_duration;
    tp.qa_cycle_inv = 1.0 / p.qa_phase_duration;
    tp.qa_factor = p.qa_breaking_factor * (double)powf(2.0f, -1.0f / 6.0f);   // main.cpp:719-723
    tp.lj_bb_r_min = p.lj_bb_r_min; tp.lj_bb_depth = p.lj_bb_depth;
    tp.lj_bs_r_min = p.lj_bs_r_min; tp.lj_bs_depth = p.lj_bs_depth;
    tp.ss_sinking = p.ss_sinking;
    tp.chir_e_chi = p.chir_e_chi;
    tp.nat_ss_H1 = p.nat_ss_H1;
    tp.nat_ss_dist = p.nat_ss_dist;
    tp.vel_afm_H1 = p.vel_afm_H1;
    tp.vel_afm_H2 = p.vel_afm_H2;
    tp.ext_on = (cap.afm > 0 && (p.on[XMD_TERM_VEL_AFM] || p.on[XMD_TERM_FORCE_AFM])) ||
                (p.on[XMD_TERM_SOLID_WALL] && !walls[0].empty()) || (p.on[XMD_TERM_LJ_WALL] && !walls[1].empty());
    if (tp.ext_on) d.fext = (double *)dalloc(sizeof(double) * 3 * N);
    tp.n_solid = p.on[XMD_TERM_SOLID_WALL] ? (int)walls[0].size() / 6 : 0;
    tp.n_ljw = p.on[XMD_TERM_LJ_WALL] ? (int)walls[1].size() / 6 : 0;
    tp.solid_eps = p.solid_wall_depth;
    tp.solid_cutoff = p.solid_wall_cutoff;
    tp.ljw_min_dist = p.lj_wall_min_dist;
    tp.ljw_factor = p.lj_wall_breaking_factor * std::pow(2.0, -1.0 / 6.0);   // main.cpp:842
    tp.ljw_cycle = p.lj_wall_phase_duration;
    tp.ljw_cycle_inv = 1.0 / p.lj_wall_phase_duration;
    tp.ljw_depth = p.lj_wall_depth;
    tp.pid_lambda = p.pid_lambda;
    for (int k = 0; k < 4; ++k) {
        tp.pid_bbp[k] = p.pid_bbp[k];
        tp.pid_bbm[k] = p.pid_bbm[k];
    }
    tp.pid_ss[0] = p.pid_ss[0];
    tp.pid_ss[1] = p.pid_ss[1];
    if (p.on[XMD_TERM_PID]) {
        // bundle forces per bead, and the side-chain LJ table by pair type
        // (lj_variants.cpp:59-62: sink_lj(depth, r_min = bb r_min when
        // sinking else r_max, r_max))
        d.pid_f = (double *)dalloc(sizeof(double) * 9 * (size_t)N);
        std::vector<double> sd(XMD_NUM_SS), smin(XMD_NUM_SS), smax(XMD_NUM_SS);
        for (int k = 0; k < XMD_NUM_SS; ++k) {
            sd[k] = p.ss_depth[k];
            smax[k] = p.ss_r_max[k];
            smin[k] = p.ss_sinking ? p.lj_bb_r_min : p.ss_r_max[k];
        }
        double *t_sd = (double *)dalloc(sizeof(double) * XMD_NUM_SS);
        double *t_smin = (double *)dalloc(sizeof(double) * XMD_NUM_SS);
        double *t_smax = (double *)dalloc(sizeof(double) * XMD_NUM_SS);
        CK(cudaMemcpyAsync(t_sd, sd.data(), sizeof(double) * XMD_NUM_SS, cudaMemcpyHostToDevice, stream));
        CK(cudaMemcpyAsync(t_smin, smin.data(), sizeof(double) * XMD_NUM_SS, cudaMemcpyHostToDevice, stream));
        CK(cudaMemcpyAsync(t_smax, smax.data(), sizeof(double) * XMD_NUM_SS, cudaMemcpyHostToDevice, stream));
        d.pid_sd = t_sd;
        d.pid_smin = t_smin;
        d.pid_smax = t_smax;
        CK(cudaStreamSynchronize(stream));
    }
    tp.f = TermP::F32{(float)tp.tether_H1, (float)tp.tether_H2, (float)tp.nat_ang_k, (float)tp.cnd_CDA,
                      (float)tp.cnd_CDB, (float)tp.snd_CDH, (float)tp.go_depth, (float)tp.pauli_r_excl,
                      (float)tp.pauli_depth, (float)tp.es_Vf, (float)tp.es_sdi, (float)tp.chir_e_chi,
                      (float)tp.nat_ss_H1, (float)tp.nat_ss_dist};
    if (p.on[XMD_TERM_QA]) {
        // quasi-adiabatic state (tables of main.cpp:681-700, lj_variants.cpp:59-62)
        d.qa_on = 1;
        QaDev &q = d.qa;
        q.nh = (float4 *)dalloc(2 * sizeof(float4) * (size_t)N);
        q.sync = (int32_t *)dalloc(sizeof(int32_t) * N);
        q.ref_cnt = (int32_t *)dalloc(sizeof(int32_t) * N);
        q.ref = (int32_t *)dalloc(sizeof(int32_t) * QA_REF_CAP * (size_t)N);
        q.tmp_cnt = (int32_t *)dalloc(sizeof(int32_t) * N);
        q.tmp = (int32_t *)dalloc(sizeof(int32_t) * QA_TMP_CAP * (size_t)N);
        q.tmp_off = (int32_t *)dalloc(sizeof(int32_t) * N);
        q.nbchunk = std::max(1, cap.qab);
        q.bchunk = (int2 *)dalloc(sizeof(int2) * q.nbchunk);
        CK(cudaMemsetAsync(q.bchunk, 0, sizeof(int2) * q.nbchunk, stream));
        q.bcsum = (int32_t *)dalloc(sizeof(int32_t) * q.nbchunk);
        qa_bchunk_next = 0;
        const int fp_total = std::max(1, cap.fp), ct_total = std::max(1, cap.ct);
        q.fp_total = fp_total;
        q.ct_total = ct_total;
        q.fp_i1 = (int32_t *)dalloc(sizeof(int32_t) * fp_total);
        q.fp_i2 = (int32_t *)dalloc(sizeof(int32_t) * fp_total);
        q.fp_rep = (int32_t *)dalloc(sizeof(int32_t) * fp_total);
        q.fp_vac = (uint8_t *)dalloc(fp_total);
        q.cand_type = (int32_t *)dalloc(sizeof(int32_t) * fp_total);
        q.cand_d1 = (int32_t *)dalloc(sizeof(int32_t) * fp_total);
        q.cand_d2 = (int32_t *)dalloc(sizeof(int32_t) * fp_total);
        const int nsift = (fp_total + QA_SIFT - 1) / QA_SIFT;
        q.cand_list = (int32_t *)dalloc(sizeof(int32_t) * (size_t)nsift * QA_SIFT);
        q.cand_blk = (int32_t *)dalloc(sizeof(int32_t) * nsift);
        CK(cudaMemsetAsync(q.cand_blk, 0, sizeof(int32_t) * nsift, stream));
        q.ct_i1 = (int32_t *)dalloc(sizeof(int32_t) * ct_total);
        q.ct_i2 = (int32_t *)dalloc(sizeof(int32_t) * ct_total);
        q.ct_type = (int32_t *)dalloc(sizeof(int32_t) * ct_total);
        q.ct_d1 = (int32_t *)dalloc(sizeof(int32_t) * ct_total);
        q.ct_d2 = (int32_t *)dalloc(sizeof(int32_t) * ct_total);
        q.ct_status = (uint8_t *)dalloc(ct_total);
        q.ct_vac = (uint8_t *)dalloc(ct_total);
        q.ct_rm = (uint8_t *)dalloc(ct_total);
        CK(cudaMemsetAsync(q.ct_rm, 0, ct_total, stream));
        q.ct_rep = (int32_t *)dalloc(sizeof(int32_t) * ct_total);
        CK(cudaMemsetAsync(q.ct_rep, 0xff, sizeof(int32_t) * ct_total, stream));
        q.ct_ref = (double *)dalloc(sizeof(double) * ct_total);
        std::vector<double> req(4 + XMD_NUM_SS, 0.0), sd(XMD_NUM_SS), smin(XMD_NUM_SS), smax(XMD_NUM_SS);
        req[1] = p.lj_bb_r_min;
        req[2] = req[3] = p.lj_bs_r_min;
        for (int a1 = 0; a1 < XMD_NUM_AA; ++a1)
            for (int a2 = 0; a2 < XMD_NUM_AA; ++a2)
                req[4 + a1 + XMD_NUM_AA * a2] = p.ss_r_max[a1 * XMD_NUM_AA + a2];
        for (int k = 0; k < XMD_NUM_SS; ++k) {
            sd[k] = p.ss_depth[k];
            smax[k] = p.ss_r_max[k];
            smin[k] = p.ss_sinking ? p.lj_bb_r_min : p.ss_r_max[k];
        }
        double *t_req = (double *)dalloc(sizeof(double) * req.size());
        double *t_sd = (double *)dalloc(sizeof(double) * XMD_NUM_SS);
        double *t_smin = (double *)dalloc(sizeof(double) * XMD_NUM_SS);
        double *t_smax = (double *)dalloc(sizeof(double) * XMD_NUM_SS);
        int32_t *t_pt = (int32_t *)dalloc(sizeof(int32_t) * XMD_NUM_AA);
        CK(cudaMemcpyAsync(t_req, req.data(), sizeof(double) * req.size(), cudaMemcpyHostToDevice, stream));
        CK(cudaMemcpyAsync(t_sd, sd.data(), sizeof(double) * XMD_NUM_SS, cudaMemcpyHostToDevice, stream));
        CK(cudaMemcpyAsync(t_smin, smin.data(), sizeof(double) * XMD_NUM_SS, cudaMemcpyHostToDevice, stream));
        CK(cudaMemcpyAsync(t_smax, smax.data(), sizeof(double) * XMD_NUM_SS, cudaMemcpyHostToDevice, stream));
        CK(cudaMemcpyAsync(t_pt, p.polarization, sizeof(int32_t) * XMD_NUM_AA, cudaMemcpyHostToDevice, stream));
        q.req_min_dist = t_req;
        q.ss_depth = t_sd;
        q.ss_rmin = t_smin;
        q.ss_rmax = t_smax;
        q.ptype = t_pt;
        q.min_cos_hr = p.qa_min_cos_hr;
        q.min_cos_hh = p.qa_min_cos_hh;
        q.max_cos_nr = p.qa_max_cos_nr;
        double rmax = 0.0;
        for (double v : req) rmax = std::max(rmax, v);
        const double w = rmax * (1.0 + 1e-9);
        q.req_out2 = w * w;
        q.req_out2_f = (float)(q.req_out2 * (1.0 + 1e-4));
        q.min_cos_hr_f = (float)q.min_cos_hr;
        q.min_cos_hh_f = (float)q.min_cos_hh;
        q.max_cos_nr_f = (float)q.max_cos_nr;
    }
    CK(cudaStreamSynchronize(stream));
}

void Engine::ready() {
    finalize();
    place_pending();
}
void Engine::ready_alloc() {
    if (!finalized) finalize();
}

void Engine::place_pending() {
    for (int k = 0; k < (int)reps.size(); ++k)
        if (reps[k].in_use && !reps[k].placed && !reps[k].staged) {
            if (!reps[k].have_state) throw std::logic_error("set_state must be called for every replica");
            place(k);
        }
}

// the jump table of replica slot k: 4 n draws, the bits of n applied in turn
__global__ void k_jump(Dev d, int k, const uint64_t *__restrict__ pw, unsigned n) {
    const int t = threadIdx.x;
    uint64_t x = (uint64_t)(t & 15) << (4 * (t >> 4));
    for (int l = 0; n >> l; ++l)
        if ((n >> l) & 1u) x = gf2_apply_nib(pw + (size_t)JUMP_WORDS * l, x);
    d.jump[(size_t)JUMP_WORDS * k + t] = x;
}

// static data, lists and state of replica slot k onto the device.  With st
// (staged placement) every upload goes on the side stream, after the last
// removal's clears, and the activation data (bead owners, the
// replica record) is kept in st for activate_staged().
void Engine::place(int k, Staged *st) {
    const xmd_params &p = params;
    cudaStream_t us = st ? ustream : stream;
    HostRing &ring_ = st ? uring : ring;
    if (st) CK(cudaStreamWaitEvent(ustream, ev_removed, 0));
    RepHost &r = reps[k];
    const int n = r.n;
    const bool tile = p.nl_build == XMD_NL_BUILD_TILE || (p.nl_build == XMD_NL_BUILD_AUTO && n <= TILE_MAX);
    if (tile && n > TILE_MAX)
        throw std::invalid_argument("engine: nl build 'tile' takes replicas of at most " +
                                    std::to_string(TILE_MAX) + " beads");
    const int nnat = 2 * (int)r.nat_i1.size();
    const int nss = 2 * (int)r.ss_i1.size();
    const int nchunk = tile ? (n + TL_CH - 1) / TL_CH : 0;
    const int ncell = tile ? 0 : std::max(64, 2 * n);
    const bool qa = p.on[XMD_TERM_QA] != 0;
    const int nfp = qa ? n * QA_FP_PER_BEAD + 256 : 0, nct = qa ? n * QA_CT_PER_BEAD + 256 : 0;
    // device ranges (all or nothing)
    int b = a_beads.alloc(n), no = a_nat.alloc(nnat), co = a_cells.alloc(ncell), ho = a_chunks.alloc(nchunk);
    const std::vector<int> afm_b = afm_beads(r);
    const int nafm = (int)afm_b.size();
    int fo = a_fp.alloc(nfp), to = a_ct.alloc(nct), so = a_ss.alloc(nss), ao = a_afm.alloc(nafm);
    if (b < 0 || no < 0 || co < 0 || ho < 0 || fo < 0 || to < 0 || so < 0 || ao < 0) {
        if (ao >= 0) a_afm.release(ao, nafm);
        if (so >= 0) a_ss.release(so, nss);
        if (b >= 0) a_beads.release(b, n);
        if (no >= 0) a_nat.release(no, nnat);
        if (co >= 0) a_cells.release(co, ncell);
        if (ho >= 0) a_chunks.release(ho, nchunk);
        if (fo >= 0) a_fp.release(fo, nfp);
        if (to >= 0) a_ct.release(to, nct);
        throw std::length_error("engine: the reserved capacity has no room for this replica");
    }
    r.begin = b;
    r.nat_off = no; r.nat_len = nnat;
    r.ss_off = so; r.ss_len = nss;
    r.cell_off = co; r.cell_len = ncell;
    r.chunk_off = ho; r.chunk_len = nchunk;
    r.fp_off = fo; r.fp_len = nfp;
    r.ct_off = to; r.ct_len = nct;
    r.afm_off = ao; r.afm_len = nafm;

    // per-bead static data; chain ids are local (pairs never cross replicas)
    std::vector<int32_t> rep_of(n, k), seq(r.seq), chain(r.chain), ns(n), ne(n);
    std::vector<uint32_t> bfl(n, 0);
    std::vector<double> tr(n, 0.0), ar(n, 0.0), dr(n, 0.0);
    for (int i = 0; i < n; ++i) {
        uint32_t f = 0;
        if (!std::isnan(r.teth_r0[i])) { f |= BF_TETH; tr[i] = r.teth_r0[i]; }
        if (!std::isnan(r.ang_t0[i])) { f |= BF_ANG; ar[i] = r.ang_t0[i]; }
        if (!std::isnan(r.dih_p0[i])) { f |= BF_DIH; dr[i] = r.dih_p0[i]; }
        if (!std::isnan(r.chir_f[i])) f |= BF_CHIR;
        if (r.hang_t[i] >= 0) f |= BF_HANG | ((uint32_t)r.hang_t[i] << BF_HANG_SHIFT);
        if (r.hdih_t[i] >= 0) f |= BF_HDIH | ((uint32_t)r.hdih_t[i] << BF_HDIH_SHIFT);
        {
            auto it = std::lower_bound(afm_b.begin(), afm_b.end(), i);
            if (it != afm_b.end() && *it == i)
                f |= BF_AFM | ((uint32_t)(ao + (int)(it - afm_b.begin())) << BF_AFM_SHIFT);
        }
        if (i > 0 && consecutive(r, i - 1, i)) f |= BF_PREV;
        if (i + 1 < r.n && consecutive(r, i, i + 1)) f |= BF_NEXT;
        bfl[i] = f;
    }
    // natives of each bead (both directions), ordered by partner: a CSR
    // segment of the replica
    std::vector<std::vector<std::pair<int, double>>> nat(n);
    for (size_t q = 0; q < r.nat_i1.size(); ++q) {
        nat[r.nat_i1[q]].push_back({b + r.nat_i2[q], r.nat_d[q]});
        nat[r.nat_i2[q]].push_back({b + r.nat_i1[q], r.nat_d[q]});
    }
    std::vector<int32_t> nj;
    std::vector<double> nd;
    for (int i = 0; i < n; ++i) {
        std::sort(nat[i].begin(), nat[i].end());
        ns[i] = no + (int)nj.size();
        for (auto &e : nat[i]) { nj.push_back(e.first); nd.push_back(e.second); }
        ne[i] = no + (int)nj.size();
    }
    // (the ring has taken the data when a call returns)
    auto up = [&](void *dst, const void *src, size_t bytes_) { ring_.up(dst, src, bytes_); };
    if (st) st->rep_of = rep_of;
    else up(d.rep_of + b, rep_of.data(), sizeof(int32_t) * n);
    up(d.chain + b, chain.data(), sizeof(int32_t) * n);
    up(d.seq + b, seq.data(), sizeof(int32_t) * n);
    up(d.atype + b, r.atype.data(), n);
    up(d.bflags + b, bfl.data(), sizeof(uint32_t) * n);
    up(d.teth_r0 + b, tr.data(), sizeof(double) * n);
    up(d.ang_t0 + b, ar.data(), sizeof(double) * n);
    up(d.dih_p0 + b, dr.data(), sizeof(double) * n);
    {
        std::vector<double2> ch(n);
        std::vector<float2> chf(n);
        for (int i = 0; i < n; ++i) {
            const bool on = !std::isnan(r.chir_f[i]);
            ch[i] = make_double2(on ? r.chir_f[i] : 0.0, on ? r.chir_n[i] : 0.0);
            chf[i] = make_float2((float)ch[i].x, (float)ch[i].y);
        }
        if (d.chir) {
            up(d.chir + b, ch.data(), sizeof(double2) * n);
            up(d.chir_f32 + b, chf.data(), sizeof(float2) * n);
        }
        // disulfide partners per bead, both directions, ordered by partner
        std::vector<std::vector<int>> sp(n);
        for (size_t q = 0; q < r.ss_i1.size(); ++q) {
            sp[r.ss_i1[q]].push_back(b + r.ss_i2[q]);
            sp[r.ss_i2[q]].push_back(b + r.ss_i1[q]);
        }
        std::vector<int32_t> sst(n), sse(n), sj;
        for (int i = 0; i < n; ++i) {
            std::sort(sp[i].begin(), sp[i].end());
            sst[i] = so + (int)sj.size();
            for (int x : sp[i]) sj.push_back(x);
            sse[i] = so + (int)sj.size();
        }
        up(d.ss_start + b, sst.data(), sizeof(int32_t) * n);
        up(d.ss_end + b, sse.data(), sizeof(int32_t) * n);
        up(d.ss_j + so, sj.data(), sizeof(int32_t) * sj.size());
        if (nss) CK(cudaMemsetAsync(d.ss_on + so, 0, nss, us));
    }
    std::vector<float4> bf(n);
    std::vector<double2> dcs(n);
    for (int i = 0; i < n; ++i) {
        dcs[i] = make_double2(std::cos(dr[i]), std::sin(dr[i]));
        bf[i] = make_float4((float)tr[i], (float)ar[i], (float)dr[i], 0.0f);
    }
    up(d.dih_cs + b, dcs.data(), sizeof(double2) * n);
    up(d.bond_f + b, bf.data(), sizeof(float4) * n);
    up(d.nat_start + b, ns.data(), sizeof(int32_t) * n);
    up(d.nat_end + b, ne.data(), sizeof(int32_t) * n);
    up(d.nat_j + no, nj.data(), sizeof(int32_t) * nj.size());
    up(d.nat_d + no, nd.data(), sizeof(double) * nd.size());
    CK(cudaMemsetAsync(d.nat_on + no, 0, nnat, us));
    CK(cudaMemsetAsync(d.nl_cnt + b, 0, sizeof(int32_t) * n, us));
    CK(cudaMemsetAsync(d.go_cnt + b, 0, sizeof(int32_t) * n, us));
    std::vector<int2> ch(nchunk);
    for (int c = 0; c < nchunk; ++c) ch[c] = make_int2(k, b + c * TL_CH);
    up(d.chunks + ho, ch.data(), sizeof(int2) * nchunk);

    RepDev rd;
    derive_rep(k, rd);
    rd.cell_off = co;
    rd.cell_budget = ncell;
    rd.tile = tile;
    rd.fault = 0;
    rd.chunk_off = tile ? ho : 0;
    rd.nchunk = nchunk;
    rd.active = 1;
    rd.steps_left = r.steps_left;
    rd.afm = nafm > 0;
    if (nafm) {
        // the tips of each pulled bead; a velocity tip's origin defaults to
        // the bead's position when placed (main.cpp:884)
        std::vector<AfmTip> tips(nafm);
        for (auto &tp : tips) tp = AfmTip{0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        auto slot = [&](int i) { return (int)(std::lower_bound(afm_b.begin(), afm_b.end(), i) - afm_b.begin()); };
        for (size_t q = 0; q < r.vafm_i.size(); ++q) {
            const int i = r.vafm_i[q];
            AfmTip &tp = tips[slot(i)];
            const double *o = &r.vafm_o[3 * q], *v = &r.vafm_v[3 * q];
            tp.ox = std::isnan(o[0]) ? r.r[3 * i] : o[0];
            tp.oy = std::isnan(o[1]) ? r.r[3 * i + 1] : o[1];
            tp.oz = std::isnan(o[2]) ? r.r[3 * i + 2] : o[2];
            tp.vx = v[0]; tp.vy = v[1]; tp.vz = v[2];
            tp.has_vel = 1;
        }
        for (size_t q = 0; q < r.fafm_i.size(); ++q) {
            AfmTip &tp = tips[slot(r.fafm_i[q])];
            tp.fx += r.fafm_F[3 * q]; tp.fy += r.fafm_F[3 * q + 1]; tp.fz += r.fafm_F[3 * q + 2];
        }
        up(d.afm + ao, tips.data(), sizeof(AfmTip) * nafm);
    }
    if (qa) {
        rd.fp_off = fo;
        rd.fp_cap = nfp;
        rd.ct_off = to;
        rd.ct_cap = nct;
        std::vector<int32_t> fprep(nfp, k), sy(n);
        up(d.qa.fp_rep + fo, fprep.data(), sizeof(int32_t) * nfp);
        std::vector<int32_t> ctrep(nct, k);
        up(d.qa.ct_rep + to, ctrep.data(), sizeof(int32_t) * nct);
        const int nbc = (n + QA_BCHUNK - 1) / QA_BCHUNK;
        if (qa_bchunk_next + nbc > d.qa.nbchunk) throw std::logic_error("engine: QA chunk table full");
        std::vector<int2> bch(nbc);
        for (int c = 0; c < nbc; ++c) bch[c] = make_int2(k, b + c * QA_BCHUNK);
        up(d.qa.bchunk + qa_bchunk_next, bch.data(), sizeof(int2) * nbc);
        rd.qa_bchunk_off = qa_bchunk_next;
        rd.qa_nbchunk = nbc;
        qa_bchunk_next += nbc;
        // valences start at the residue limits (intended main.cpp:662-672)
        for (int i = 0; i < n; ++i) {
            const int32_t *lim = p.limits[r.atype[i]];
            sy[i] = (lim[0] & 0xff) | ((lim[1] & 0xff) << 8) | ((lim[2] & 0xff) << 16) | ((lim[3] & 0xff) << 24);
        }
        up(d.qa.sync + b, sy.data(), sizeof(int32_t) * n);
        CK(cudaMemsetAsync(d.qa.ref_cnt + b, 0, sizeof(int32_t) * n, us));
    }
    if (!st) up(d.rep + k, &rd, sizeof(RepDev));
    k_jump<<<1, JUMP_WORDS, 0, us>>>(d, k, rng_pow, (unsigned)n);
    if (st) {
        // the state (upload_state's data) on the side stream too; the record
        // starts as upload_state leaves it: t = 0, first list build pending
        upload_state_data(k, ring_, false);
        rd.t = 0.0;
        rd.first = 1;
        rd.maxdisp = 0;
        rd.fault = 0;
        st->k = k;
        st->rd = rd;
        r.staged = true;
        return;
    }
    for (int i = 0; i < n; ++i) owner_h[b + i] = k;
    r.placed = true;
    if (r.cell_len) ++live_cell;
    upload_state(k);
}

// A replica's state from the host: positions, history (y1 = v dt, y2..y5 = 0)
// and generator states of beads i0 .. i0 + m of replica slot k, read from
// pinned memory (r, then v), a block's rows in one sweep.  The generator of
// bead i is the seed 4 i draws on, by the bits of i (the host's chain over the
// beads and 18 pageable copies took 0.96 ms for 54744 beads).  With `record`
// the slot starts over: t = 0, first list build pending; a new state thaws a
// frozen replica.
struct ChargeP { double q[XMD_NUM_AA]; };
constexpr int ST_TB = 256, ST_PIECE = 16384;   // beads per block, per piece of staging memory
__global__ void __launch_bounds__(ST_TB) k_set_state(Dev d, int cur, int k, int b, int i0, int m,
                                                     const double *__restrict__ in, ChargeP c, double dt,
                                                     uint64_t seed, const uint64_t *__restrict__ pw, int record,
                                                     long long steps_left) {
    __shared__ double s_in[6 * ST_TB];
    const int t = threadIdx.x, base = blockIdx.x * ST_TB, cnt = min(ST_TB, m - base);
    for (int q = t; q < 3 * cnt; q += ST_TB) {
        s_in[q] = in[3 * (size_t)base + q];
        s_in[3 * ST_TB + q] = in[3 * (size_t)(m + base) + q];
    }
    __syncthreads();
    if (t < cnt) {
        const int i = i0 + base + t;
        const size_t g = (size_t)b + i, N = d.N;
        const double *x = s_in + 3 * t, *v = x + 3 * ST_TB;
        d.pos[cur][g] = make_double4_32a(x[0], x[1], x[2], c.q[d.atype[g]]);
        for (int a = 0; a < 15; ++a) d.yh[a * N + g] = a < 3 ? __dmul_rn(v[a], dt) : 0.0;
        uint64_t s = seed;
        for (int l = 0; i >> l; ++l)
            if ((i >> l) & 1) s = gf2_apply_nib(pw + (size_t)JUMP_WORDS * l, s);
        d.rng[g] = s;
    }
    if (record && blockIdx.x == 0 && t == 0) {
        RepDev &rp = d.rep[k];
        rp.t = 0.0;
        rp.first = 1;
        rp.maxdisp = 0;
        if (rp.fault) {
            rp.fault = 0;
            rp.steps_left = steps_left;
        }
    }
}
// positions, velocities (y1 / dt) and time the other way
__global__ void __launch_bounds__(ST_TB) k_get_state(Dev d, int cur, int k, int b, int i0, int m, double dt_inv,
                                                     double *__restrict__ out, double *__restrict__ t_out) {
    __shared__ double s_out[6 * ST_TB];
    const int t = threadIdx.x, base = blockIdx.x * ST_TB, cnt = min(ST_TB, m - base);
    if (t < cnt) {
        const size_t g = (size_t)b + i0 + base + t, N = d.N;
        const double4_32a p = d.pos[cur][g];
        double *x = s_out + 3 * t, *v = x + 3 * ST_TB;
        x[0] = p.x; x[1] = p.y; x[2] = p.z;
        for (int a = 0; a < 3; ++a) v[a] = __dmul_rn(d.yh[a * N + g], dt_inv);
    }
    __syncthreads();
    for (int q = t; q < 3 * cnt; q += ST_TB) {
        out[3 * (size_t)base + q] = s_out[q];
        out[3 * (size_t)(m + base) + q] = s_out[3 * ST_TB + q];
    }
    if (blockIdx.x == 0 && t == 0) *t_out = d.rep[k].t;
}

void Engine::upload_state_data(int k, HostRing &up, bool record) {
    const RepHost &r = reps[k];
    ChargeP c;
    for (int a = 0; a < XMD_NUM_AA; ++a) c.q[a] = params.charge[a];
    for (int i0 = 0; i0 < r.n; i0 += ST_PIECE) {
        const int m = std::min(ST_PIECE, r.n - i0);
        double *in = (double *)up.take(sizeof(double) * 6 * m);
        std::memcpy(in, r.r.data() + 3 * (size_t)i0, sizeof(double) * 3 * m);
        std::memcpy(in + 3 * (size_t)m, r.v.data() + 3 * (size_t)i0, sizeof(double) * 3 * m);
        k_set_state<<<(m + ST_TB - 1) / ST_TB, ST_TB, 0, up.s>>>(d, cur, k, r.begin, i0, m, in, c, params.dt, r.seed,
                                                                 rng_pow, record && i0 == 0, r.steps_left);
        CK(cudaGetLastError());
    }
}

void Engine::upload_state(int k) { upload_state_data(k, ring, true); }

// (no early way out: the test vectorises)
static bool all_finite(const double *x, size_t n) {
    const uint64_t EXP = 0x7ffull << 52;
    uint64_t bad = 0;
    for (size_t k = 0; k < n; ++k) {
        uint64_t u;
        std::memcpy(&u, x + k, 8);
        bad |= (uint64_t)((u & EXP) == EXP);
    }
    return bad == 0;
}

void Engine::set_state(int rep, const double *r, const double *v) {
    check_rep(reps, rep);
    if (!r) throw std::invalid_argument("null positions");
    RepHost &h = reps[rep];
    h.r.assign(r, r + 3 * (size_t)h.n);
    if (v) h.v.assign(v, v + 3 * (size_t)h.n);
    else h.v.assign(3 * (size_t)h.n, 0.0);
    if (!all_finite(h.r.data(), h.r.size())) throw std::invalid_argument("non-finite position");
    h.have_state = true;
    if (h.placed) upload_state(rep);
}

void Engine::set_history(int rep, const double *y, double t, uint64_t rngs) {
    check_rep(reps, rep);
    ready();
    RepHost &h = reps[rep];
    int n = h.n, b = h.begin;
    size_t n3 = 3 * (size_t)n;
    std::vector<double4_32a> pos(n);
    for (int i = 0; i < n; ++i)
        pos[i] = make_double4_32a(y[3 * i], y[3 * i + 1], y[3 * i + 2], params.charge[h.atype[i]]);
    CK(cudaMemcpyAsync(d.pos[cur] + b, pos.data(), sizeof(double4_32a) * n, cudaMemcpyHostToDevice, stream));
    std::vector<double> col(n);
    for (int ord = 1; ord < 6; ++ord)
        for (int a = 0; a < 3; ++a) {
            for (int i = 0; i < n; ++i) col[i] = y[ord * n3 + 3 * i + a];
            CK(cudaMemcpyAsync(d.yh + (size_t)((ord - 1) * 3 + a) * d.N + b, col.data(), sizeof(double) * n,
                               cudaMemcpyHostToDevice, stream));
        }
    std::vector<uint64_t> st(n);
    uint64_t s = rngs;
    for (int i = 0; i < n; ++i) {
        st[i] = s;
        for (int q = 0; q < 4; ++q) s = xs_step(s);
    }
    CK(cudaMemcpyAsync(d.rng + b, st.data(), sizeof(uint64_t) * n, cudaMemcpyHostToDevice, stream));
    RepDev rd;
    CK(cudaMemcpyAsync(&rd, d.rep + rep, sizeof(RepDev), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    rd.t = t;
    rd.first = 1;
    rd.maxdisp = 0;
    if (rd.fault) {   // a new state thaws a frozen replica
        rd.fault = 0;
        rd.steps_left = reps[rep].steps_left;
    }
    CK(cudaMemcpyAsync(d.rep + rep, &rd, sizeof(RepDev), cudaMemcpyHostToDevice, stream));
    CK(cudaStreamSynchronize(stream));
}

void Engine::get_state(int rep, double *r, double *v, double *t) {
    check_rep(reps, rep);
    ready();
    const RepHost &h = reps[rep];
    const double dt_inv = 1.0 / params.dt;
    // pieces of staging memory (more than half a half each, so that a piece
    // waits only for one already handed over), the last copied out while the
    // next is filled
    static_assert(2 * (48 * ST_PIECE + 8) > HostRing::HALF && 48 * ST_PIECE + 8 <= HostRing::HALF, "pieces");
    double *p[2] = {nullptr, nullptr};
    for (int i0 = 0, c = 0; i0 < h.n + ST_PIECE; i0 += ST_PIECE, ++c) {
        if (i0 < h.n) {
            const int m = std::min(ST_PIECE, h.n - i0);
            p[c & 1] = (double *)ring.take(sizeof(double) * (6 * (size_t)m + 1));
            k_get_state<<<(m + ST_TB - 1) / ST_TB, ST_TB, 0, stream>>>(d, cur, rep, h.begin, i0, m, dt_inv, p[c & 1],
                                                                       p[c & 1] + 6 * (size_t)m);
            CK(cudaGetLastError());
            CK(cudaEventRecord(down_ev[c & 1], stream));
        }
        if (c && i0 - ST_PIECE < h.n) {
            const int j0 = i0 - ST_PIECE, m = std::min(ST_PIECE, h.n - j0);
            const double *q = p[(c - 1) & 1];
            CK(cudaEventSynchronize(down_ev[(c - 1) & 1]));
            if (r) std::memcpy(r + 3 * (size_t)j0, q, sizeof(double) * 3 * m);
            if (v) std::memcpy(v + 3 * (size_t)j0, q + 3 * (size_t)m, sizeof(double) * 3 * m);
            if (t) *t = q[6 * (size_t)m];
        }
    }
}
// ---- snapshots: the replica's whole mutable device state -----------------------
// The reference's store (include/xmd/store/store.h; main.cpp's make_saved
// items) keeps positions, the Gear history, time, the pair lists and the QA
// sets, but not the generator (a make_temp), so a resumed run draws new
// noise.  A snapshot here holds everything a step reads and writes:
// positions, Gear history, time, per-bead generators, skin origins, the
// Verlet rows, native and disulfide activity, and the quasi-adiabatic state
// (sync, contacts with their slots, free pairs).  Restoring it continues
// the run bit for bit.  It is taken and restored in place: the replica must
// sit at the same slots of a context built the same way (same parameters,
// the same systems added in the same order); the header checks this.

namespace {
struct SnapHeader {
    char magic[8];
    uint32_t version, precision;
    int32_t rep, n, begin, nl_cap;
    int32_t nat_off, nat_len, ss_off, ss_len;
    int32_t qa_on, fp_off, fp_len, ct_off, ct_len;
    int32_t pad_;
    uint64_t topo;
};
constexpr uint32_t SNAP_VERSION = 1;
constexpr char SNAP_MAGIC[8] = {'X', 'M', 'D', 'S', 'N', 'A', 'P', '1'};
struct SnapRep {   // the mutable scalars of RepDev
    double t;
    int32_t first, rebuild, fault, fp_n, ct_n, pad_;
    long long steps_left;
    unsigned long long maxdisp, rebuilds;
};

uint64_t fnv(uint64_t h, const void *p, size_t bytes) {
    const unsigned char *c = (const unsigned char *)p;
    for (size_t k = 0; k < bytes; ++k) h = (h ^ c[k]) * 1099511628211ull;
    return h;
}
}  // namespace

uint64_t Engine::topo_hash(int rep) const {
    const RepHost &r = reps[rep];
    uint64_t h = 1469598103934665603ull;
    h = fnv(h, r.chain.data(), r.chain.size() * sizeof(int32_t));
    h = fnv(h, r.seq.data(), r.seq.size() * sizeof(int32_t));
    h = fnv(h, r.atype.data(), r.atype.size());
    h = fnv(h, r.nat_i1.data(), r.nat_i1.size() * sizeof(int32_t));
    h = fnv(h, r.nat_i2.data(), r.nat_i2.size() * sizeof(int32_t));
    h = fnv(h, r.ss_i1.data(), r.ss_i1.size() * sizeof(int32_t));
    h = fnv(h, r.ss_i2.data(), r.ss_i2.size() * sizeof(int32_t));
    return h;
}

size_t Engine::snapshot_io(int rep, unsigned char *buf, size_t bytes, bool save, int cap_rows) {
    check_rep(reps, rep);
    ready();
    RepHost &h = reps[rep];
    const int n = h.n, b = h.begin;
    const size_t N = (size_t)d.N;
    SnapHeader hd{};
    std::memcpy(hd.magic, SNAP_MAGIC, 8);
    hd.version = SNAP_VERSION;
    hd.precision = (uint32_t)params.precision;
    hd.rep = rep; hd.n = n; hd.begin = b; hd.nl_cap = 0;   // the row capacity may differ (below)
    hd.nat_off = h.nat_off; hd.nat_len = h.nat_len; hd.ss_off = h.ss_off; hd.ss_len = h.ss_len;
    hd.qa_on = d.qa_on; hd.fp_off = h.fp_off; hd.fp_len = h.fp_len; hd.ct_off = h.ct_off; hd.ct_len = h.ct_len;
    // the topology, and the wall planes the saved LJ attractive wall states
    // refer to
    hd.topo = fnv(fnv(topo_hash(rep), walls[0].data(), walls[0].size() * sizeof(double)), walls[1].data(),
                  walls[1].size() * sizeof(double));
    hd.pad_ = (int32_t)(walls[1].size() / 6);   // LJ attractive walls (their pair states are saved)
    size_t off = 0;
    auto host = [&](void *p, size_t nb) {
        if (buf && off + nb <= bytes) {
            if (save) std::memcpy(buf + off, p, nb);
            else std::memcpy(p, buf + off, nb);
        }
        off += nb;
    };
    auto dev = [&](void *p, size_t nb) {
        if (buf && nb && off + nb <= bytes)
            CK(cudaMemcpyAsync(save ? (void *)(buf + off) : p, save ? p : (const void *)(buf + off), nb,
                               save ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, stream));
        off += nb;
    };
    // rows [k][N] of a per-bead array: the replica's n entries of each row
    auto rows = [&](void *base, size_t elem, int nrows) {
        for (int k = 0; k < nrows; ++k) dev((char *)base + ((size_t)k * N + b) * elem, elem * n);
    };
    if (!save) {
        if (!buf || bytes < sizeof(SnapHeader)) throw std::invalid_argument("snapshot too short");
        SnapHeader got;
        std::memcpy(&got, buf, sizeof got);
        if (std::memcmp(got.magic, SNAP_MAGIC, 8) != 0 || got.version != SNAP_VERSION)
            throw std::invalid_argument("not a snapshot of this format");
        if (std::memcmp(&got, &hd, sizeof hd) != 0)
            throw std::invalid_argument("snapshot of another replica layout (precision, replica sizes or order, "
                                        "topology or wall planes differ)");
        // the whole snapshot must be there before anything of the replica
        // is overwritten: a short buffer leaves the replica as it was
        int32_t scap;
        if (bytes < sizeof(SnapHeader) + sizeof scap) throw std::invalid_argument("snapshot truncated");
        std::memcpy(&scap, buf + sizeof(SnapHeader), sizeof scap);
        if (scap <= 0 || scap > (1 << 20)) throw std::invalid_argument("snapshot: bad row capacity");
        if (bytes < snapshot_io(rep, nullptr, 0, true, scap)) throw std::invalid_argument("snapshot truncated");
    }
    host(&hd, sizeof hd);
    // Verlet row capacity of the snapshot; a restore grows this context's rows
    // to it (capacity does not change the trajectory)
    int32_t cap = cap_rows >= 0 ? cap_rows : nl_cap;
    host(&cap, sizeof cap);
    if (buf && !save) {
        if (cap <= 0 || cap > (1 << 20)) throw std::invalid_argument("snapshot: bad row capacity");
        if (cap > nl_cap) resize_rows(cap);
    }
    CK(cudaStreamSynchronize(stream));
    RepDev rd;
    CK(cudaMemcpy(&rd, d.rep + rep, sizeof(RepDev), cudaMemcpyDeviceToHost));
    SnapRep sr{rd.t, rd.first, rd.rebuild, rd.fault, rd.fp_n, rd.ct_n, 0, rd.steps_left, rd.maxdisp, rd.rebuilds};
    host(&sr, sizeof sr);
    dev(d.pos[cur] + b, sizeof(double4_32a) * n);
    rows(d.yh, sizeof(double), 15);
    dev(d.orig + b, sizeof(double4_32a) * n);
    dev(d.rng + b, sizeof(uint64_t) * n);
    dev(d.nl_cnt + b, sizeof(int32_t) * n);
    rows(d.nl_row, sizeof(int32_t), cap);
    dev(d.nat_on + h.nat_off, h.nat_len);
    dev(d.ss_on + h.ss_off, h.ss_len);
    for (int w = 0; w < hd.pad_; ++w) dev(d.ljw + (size_t)w * N + b, sizeof(LjWallState) * n);
    if (d.qa_on) {
        rows(d.qa.sync, sizeof(int32_t), 1);
        rows(d.qa.ref_cnt, sizeof(int32_t), 1);
        rows(d.qa.ref, sizeof(int32_t), QA_REF_CAP);
        const int fo = h.fp_off, fl = h.fp_len, co = h.ct_off, cl = h.ct_len;
        dev(d.qa.fp_i1 + fo, sizeof(int32_t) * fl);
        dev(d.qa.fp_i2 + fo, sizeof(int32_t) * fl);
        dev(d.qa.fp_rep + fo, sizeof(int32_t) * fl);
        dev(d.qa.fp_vac + fo, fl);
        dev(d.qa.ct_i1 + co, sizeof(int32_t) * cl);
        dev(d.qa.ct_i2 + co, sizeof(int32_t) * cl);
        dev(d.qa.ct_type + co, sizeof(int32_t) * cl);
        dev(d.qa.ct_d1 + co, sizeof(int32_t) * cl);
        dev(d.qa.ct_d2 + co, sizeof(int32_t) * cl);
        dev(d.qa.ct_status + co, cl);
        dev(d.qa.ct_vac + co, cl);
        dev(d.qa.ct_rm + co, cl);
        dev(d.qa.ct_rep + co, sizeof(int32_t) * cl);
        dev(d.qa.ct_ref + co, sizeof(double) * cl);
    }
    CK(cudaStreamSynchronize(stream));
    if (buf && !save) {
        if (off > bytes) throw std::invalid_argument("snapshot truncated");
        rd.t = sr.t; rd.first = sr.first; rd.rebuild = sr.rebuild; rd.fault = sr.fault;
        rd.fp_n = sr.fp_n; rd.ct_n = sr.ct_n; rd.steps_left = sr.steps_left;
        rd.maxdisp = sr.maxdisp; rd.rebuilds = sr.rebuilds;
        CK(cudaMemcpy(d.rep + rep, &rd, sizeof(RepDev), cudaMemcpyHostToDevice));
        k_go_lists<<<(n + 127) / 128, 128, 0, stream>>>(d, b, n);
        h.steps_left = sr.steps_left;
    }
    return off;
}
size_t Engine::snapshot_size(int rep) { return snapshot_io(rep, nullptr, 0, true); }
void Engine::snapshot(int rep, void *buf, size_t bytes) {
    if (bytes < snapshot_size(rep)) throw std::invalid_argument("snapshot buffer too small");
    snapshot_io(rep, (unsigned char *)buf, bytes, true);
}
void Engine::restore(int rep, const void *buf, size_t bytes) {
    snapshot_io(rep, (unsigned char *)const_cast<void *>(buf), bytes, false);
}

void Engine::get_history(int rep, double *y, double *t, uint64_t *rngs) {
    check_rep(reps, rep);
    ready();
    const RepHost &h = reps[rep];
    int n = h.n, b = h.begin;
    size_t n3 = 3 * (size_t)n;
    std::vector<double4_32a> pos(n);
    CK(cudaMemcpyAsync(pos.data(), d.pos[cur] + b, sizeof(double4_32a) * n, cudaMemcpyDeviceToHost, stream));
    std::vector<double> col(15 * (size_t)n);
    for (int k = 0; k < 15; ++k)
        CK(cudaMemcpyAsync(col.data() + (size_t)k * n, d.yh + (size_t)k * d.N + b, sizeof(double) * n,
                           cudaMemcpyDeviceToHost, stream));
    uint64_t s0 = 0;
    CK(cudaMemcpyAsync(&s0, d.rng + b, sizeof(uint64_t), cudaMemcpyDeviceToHost, stream));
    RepDev rd;
    CK(cudaMemcpyAsync(&rd, d.rep + rep, sizeof(RepDev), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    if (y) {
        for (int i = 0; i < n; ++i) { y[3 * i] = pos[i].x; y[3 * i + 1] = pos[i].y; y[3 * i + 2] = pos[i].z; }
        for (int ord = 1; ord < 6; ++ord)
            for (int a = 0; a < 3; ++a)
                for (int i = 0; i < n; ++i)
                    y[ord * n3 + 3 * i + a] = col[(size_t)((ord - 1) * 3 + a) * n + i];
    }
    if (t) *t = rd.t;
    if (rngs) *rngs = s0;
}

void Engine::use_device() const { CK(cudaSetDevice(device)); }

void Engine::record(std::vector<cudaEvent_t> &pool, size_t &n) {
    if (n >= pool.size()) {
        cudaEvent_t e;
        CK(cudaEventCreate(&e));
        pool.push_back(e);
    }
    CK(cudaEventRecord(pool[n++], stream));
}

void Engine::launch_rebuild() {
    if (timing) record(ev_rebuild, n_ev_rebuild);
    if (live_cell) {
        const int gb = (d.N + 255) / 256;
        k_cells<<<gb, 256, 0, stream>>>(d, cur, pass_launches(true));
        k_cell_count<<<gb, 256, 0, stream>>>(d, cur);
        k_cell_scan<<<(d.ncells + CELL_SCAN - 1) / CELL_SCAN, 256, 0, stream>>>(d);
        k_cell_scatter<<<gb, 256, 0, stream>>>(d);
        k_cell_finish<<<2 * gb, 256, 0, stream>>>(d, cur);
        k_nl_cells<<<(d.N + NC_WARPS - 1) / NC_WARPS, NC_WARPS * 32, 0, stream>>>(d, tp, cur);
    }
    if (any_tile) k_nl_tile<<<tile_grid, TL_THREADS, tile_smem, stream>>>(d, tp, cur, live_cell ? 0 : pass_launches(false));
    if (d.qa_on) {
        k_qa_fp_scan<<<d.qa.nbchunk, QA_BCHUNK, 0, stream>>>(d);
        k_qa_fp_fill<<<dim3(d.qa.nbchunk, QA_FG), 256, 0, stream>>>(d);
        k_qa_compact<<<d.R, 1024, 0, stream>>>(d);
    }
    if (timing) record(ev_rebuild, n_ev_rebuild);
}

// Grow the Verlet rows when the longest row needed (recorded by the builds)
// reaches `frac` of the capacity.  Returns true when the rows were
// reallocated (lists must then be rebuilt; captured graphs are dropped).
bool Engine::grow_rows(double frac) {
    const unsigned long long need = ((const unsigned long long *)(h_any + 8))[1];
    if ((double)need < frac * nl_cap) return false;
    resize_rows((int)(2 * need + 16));
    return true;
}

// Reallocate the Verlet rows with ncap slots per bead, keeping the rows held.
void Engine::resize_rows(int ncap) {
    int32_t *rows = nullptr;
    CK(cudaMalloc(&rows, sizeof(int32_t) * (size_t)ncap * d.N));
    // rows are slot-major ([k][N]), so the current lists keep their place:
    // growing for headroom leaves them valid without a rebuild
    CK(cudaMemcpyAsync(rows, d.nl_row, sizeof(int32_t) * (size_t)std::min(nl_cap, ncap) * d.N,
                       cudaMemcpyDeviceToDevice, stream));
    CK(cudaStreamSynchronize(stream));
    for (auto &a : allocs)
        if (a == (void *)d.nl_row) {
            CK(cudaFree(a));
            a = rows;
        }
    alloc_bytes += sizeof(int32_t) * (size_t)d.N * ncap;
    alloc_bytes -= std::max<size_t>(16, sizeof(int32_t) * (size_t)nl_cap * d.N);
    d.nl_row = rows;
    d.nl_cap = nl_cap = ncap;
    drop_graphs();
}

void Engine::set_tuning(const Tune &t) {
    if (t.fb != 32 && t.fb != 64 && t.fb != 128)
        throw std::invalid_argument("tuning: step-kernel block size must be 32, 64 or 128 beads");
    if (t.lpb != 1 && t.lpb != 2 && t.lpb != 4)
        throw std::invalid_argument("tuning: threads per bead must be 1, 2 or 4");
    if (t.graph_steps != 8 && t.graph_steps != 16 && t.graph_steps != 32 && t.graph_steps != 64)
        throw std::invalid_argument("tuning: steps per graph must be 8, 16, 32 or 64");
    if (t.tile_per_sm < 0) throw std::invalid_argument("tuning: tile blocks per SM must be >= 0");
    tune = t;
    tuned = true;
    if (finalized) {
        const int k = tune.tile_per_sm > 0 ? std::min(tune.tile_per_sm, tile_max_per_sm) : tile_max_per_sm;
        tile_grid = std::max(1, std::min(d.nchunks, tile_sms * k));
        drop_graphs();
    }
}

// The autotuner.  Every candidate launch shape (step-kernel block size,
// resident tile-build blocks per SM, steps per graph) runs on a fresh clone of
// this context: the same replicas from the same starting state, so each is
// timed on the same trajectory (the trajectory does not depend on the shape).
// A candidate's time is CUDA-event time per step over `steps` graph steps
// after one warm-up graph (which builds the first lists and captures the
// graph).  This context's device state is not touched.
Engine::Tune Engine::autotune(int steps, double *ms_out) {
    if (dynamic) throw std::logic_error("autotune needs a static context (replicas added before the first step)");
    int live = 0;
    for (auto &r : reps) live += r.in_use ? 1 : 0;
    if (!live) throw std::logic_error("autotune: the context has no replica");
    for (auto &r : reps)
        if (r.in_use && !r.have_state) throw std::logic_error("autotune: set_state must be called for every replica");
    steps = std::max(32, (steps + 31) / 32 * 32);
    // two stages: the step kernel's shape (beads per block x threads per
    // bead) at 16 steps per graph, then graph length and tile residency with
    // the best step-kernel shape
    Tune best = tune;
    double best_ms = 1e300;
    auto trial = [&](const Tune &cand) {
        Engine c(params);
        for (auto &r : reps)
            if (r.in_use) {
                RepHost h = r;
                h.placed = false;
                c.reps.push_back(std::move(h));
            }
        c.tune = cand;
        c.use_device();
        c.ready();
        c.set_tuning(cand);
        c.step(cand.graph_steps);   // first lists, graph capture
        c.sync();
        cudaEvent_t e0, e1;
        CK(cudaEventCreate(&e0));
        CK(cudaEventCreate(&e1));
        CK(cudaEventRecord(e0, c.stream));
        c.step(steps);
        CK(cudaEventRecord(e1, c.stream));
        CK(cudaEventSynchronize(e1));
        float ms = 0.0f;
        CK(cudaEventElapsedTime(&ms, e0, e1));
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        const double per = (double)ms / steps;
        if (per < best_ms) {
            best_ms = per;
            best = cand;
        }
    };
    for (int fb : {32, 64, 128})
        for (int lpb : {1, 2, 4}) trial(Tune{fb, 0, 16, lpb});
    const Tune kshape = best;
    for (int gs : {8, 16, 32, 64})
        for (int tps : {0, 2})
            if (gs != 16 || tps != 0) trial(Tune{kshape.fb, tps, gs, kshape.lpb});
    use_device();
    set_tuning(best);
    if (ms_out) *ms_out = best_ms;
    return best;
}

void Engine::drop_graphs() {
    for (auto &kv : graphs) {
        if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
        if (kv.second.graph) cudaGraphDestroy(kv.second.graph);
    }
    graphs.clear();
}

void Engine::ensure_nl() {
    for (int attempt = 0; attempt < 3; ++attempt) {
        k_nl_check<<<1, 1024, 0, stream>>>(d, 0, 0.0, (cudaGraphConditionalHandle)0, 0);
        ++launches;
        fetch_words();
        if (h_any[0]) {
            launch_rebuild();
            fetch_words();
        }
        const int st = h_any[4];
        if (!(st & ST_CAPACITY) || !auto_grow) {
            if (auto_grow) grow_rows(0.6);   // keep headroom for the run ahead
            return;
        }
        // rows overflowed at this rebuild: grow, clear the flag, rebuild all
        if (!grow_rows(0.0)) return;
        CK(cudaMemsetAsync(d.status, 0, sizeof(int), stream));
        k_mark_all<<<(d.R + 255) / 256, 256, 0, stream>>>(d);
    }
}

void Engine::launch_force_step() {
    if (timing) record(ev_force, n_ev_force);
    launch_force(1, cur);
    if (timing) record(ev_force, n_ev_force);
    launches += 1 + (tp.ext_on ? 1 : 0) + (tp.on[XMD_TERM_PID] ? 1 : 0);
    if (d.qa_on) {
        // sift + acceptance + transitions at this step's positions (qa.cpp:20-31)
        k_qa_sift<<<sift_grid(), QA_SIFT, 0, stream>>>(d, tp, cur);
        k_qa_step<<<d.R, 1024, 0, stream>>>(d, tp, cur);
        k_qa_trans<<<trans_grid(), QA_TG, 0, stream>>>(d, tp, cur);
        k_qa_refree<<<d.R, 1024, 0, stream>>>(d, 0.0, 0);
        launches += 4;
    }
}

// One graph runs `len` steps (tune.graph_steps, or a power of two for the
// rest of a call).  IF form: per step a force+integrate node, a skin check
// that sets a conditional handle on the device, and an IF node whose body
// rebuilds the lists of the flagged replicas (cells, then rows).  Plain form
// (the rebuild is the row build alone: no cell-path replica, no
// quasi-adiabatic term): the step kernel takes the decision and a row-build
// node follows, which returns at once when the work list is empty (an IF
// node costs more per step than that empty launch).  Gated form (`gated`):
// no rebuild node; the check halts the graph's remaining steps and the host
// rebuilds.  A graph of odd length leaves the position double buffer
// swapped.
cudaGraphExec_t Engine::graph_for(int start_cur, bool gated, int len) {
    const bool plain = plain_rebuild();
    const int mix = params.precision == XMD_PREC_MIXED ? 1 : 0;
    const int key = (((len * 2 + mix) * 2 + (gated ? 1 : 0)) * 2 + start_cur) * 2 + (plain ? 1 : 0);
    GraphSet &gs = graphs[key];
    if (gs.exec) return gs.exec;
    cudaGraph_t g;
    CK(cudaGraphCreate(&g, 0));
    const bool mixed = params.precision == XMD_PREC_MIXED;
    const ForceShape fs = force_shape();
    const int nb = force_blocks(d.N, fs.fb);
    void *fk = force_kernel(mixed, 1, fs.fb, fs.lpb);
    const size_t fsmem = force_smem(mixed, 1, fs.fb, d.qa_on);
    if (fsmem > 48 * 1024) allow_smem(fk, force_smem(mixed, 1, fs.fb, true));
    // a chain of nodes.  Between two kernels the edge is programmatic: the
    // second is launched while the first one's last blocks run and waits in
    // step_order(); a conditional node takes and gives full edges.
    cudaGraphNode_t prev = nullptr;
    bool prev_kernel = false;
    auto add = [&](const void *func, int grid, int block, size_t smem, void **args) {
        cudaKernelNodeParams kp{};
        kp.func = const_cast<void *>(func);
        kp.gridDim = dim3((unsigned)grid);
        kp.blockDim = dim3((unsigned)block);
        kp.sharedMemBytes = (unsigned)smem;
        kp.kernelParams = args;
        cudaGraphNode_t nn;
        CK(cudaGraphAddKernelNode(&nn, g, nullptr, 0, &kp));
        if (prev) {
            cudaGraphEdgeData ed{};
            if (prev_kernel) {
                ed.from_port = cudaGraphKernelNodePortProgrammatic;
                ed.type = cudaGraphDependencyTypeProgrammatic;
            }
            CK(cudaGraphAddDependencies(g, &prev, &nn, &ed, 1));
        }
        prev = nn;
        prev_kernel = true;
    };
    double dt = params.dt;
    // without the quasi-adiabatic term the step kernel takes the skin
    // decision itself (its last block) where no IF node needs it; with it,
    // the re-freeing kernel does in gated graphs
    const int fuse = d.qa_on ? (gated ? FUSE_GATE : FUSE_NONE) : plain ? FUSE_CHECK
                     : gated ? FUSE_CHECK_GATE : FUSE_NONE;
    int zero = 0;
    for (int s = 0; s < len; ++s) {
        int c = start_cur ^ (s & 1), cn = c ^ 1;
        int adv = 1, setc = gated ? CHECK_GATE : CHECK_COND;
        cudaGraphConditionalHandle h = 0;
        if (!plain && !gated) CK(cudaGraphConditionalHandleCreate(&h, g, 0, 0));
        int ff = fuse, rcheck = gated ? 1 : 0;   // the re-freeing's last block takes the skin decision
        void *sargs[] = {&d, &tp, &c};
        void *fargs[] = {&d, &tp, &c, &ff};
        void *dargs[] = {&d, &dt, &rcheck};
        if (tp.ext_on) add((void *)k_ext<1>, (d.N + 255) / 256, 256, 0, sargs);   // AFM, walls
        if (tp.on[XMD_TERM_PID]) add((void *)k_pid<1>, (d.N + 127) / 128, 128, 0, sargs);
        add(fk, nb, fs.fb * fs.lpb, fsmem, fargs);
        if (d.qa_on) {
            add((void *)k_qa_sift, sift_grid(), QA_SIFT, 0, sargs);
            add((void *)k_qa_step, d.R, 1024, 0, sargs);
            add((void *)k_qa_trans, trans_grid(), QA_TG, 0, sargs);
            add((void *)k_qa_refree, d.R, 1024, 0, dargs);
        }
        if (fuse != FUSE_CHECK && fuse != FUSE_CHECK_GATE && !(d.qa_on && gated)) {
            void *cargs[] = {&d, &adv, &dt, &h, &setc};
            add((void *)k_nl_check, 1, 1024, 0, cargs);
        }
        if (gated) continue;   // the host rebuilds after a halt
        if (plain) {
            void *targs[] = {&d, &tp, &cn, &zero};
            add((void *)k_nl_tile, tile_grid, TL_THREADS, tile_smem, targs);
            continue;
        }
        cudaGraphNodeParams cp{};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = h;
        cp.conditional.type = cudaGraphCondTypeIf;
        cp.conditional.size = 1;
        cudaGraphNode_t ncond;
        CK(cudaGraphAddNode(&ncond, g, &prev, nullptr, 1, &cp));
        add_rebuild_nodes(cp.conditional.phGraph_out[0], cn);
        prev = ncond;
        prev_kernel = false;
    }
    CK(cudaGraphInstantiate(&gs.exec, g, 0));
    gs.graph = g;
    return gs.exec;
}

// the list rebuild as a chain of kernel nodes (body of the rebuild IF node)
void Engine::add_rebuild_nodes(cudaGraph_t body, int cn) {
    cudaGraphNode_t last = nullptr;
    auto add = [&](cudaKernelNodeParams &kp) {
        cudaGraphNode_t nn;
        CK(cudaGraphAddKernelNode(&nn, body, last ? &last : nullptr, last ? 1 : 0, &kp));
        last = nn;
    };
    void *a1[] = {&d, &cn};
    void *a2[] = {&d, &tp, &cn};
    void *a3[] = {&d};
    const bool cells = cap.cells > 0;
    int in_cells = pass_launches(cells), in_tile = cells ? 0 : in_cells;
    void *ac[] = {&d, &cn, &in_cells};
    void *a4[] = {&d, &tp, &cn, &in_tile};
    // (by the context's capacity, not by what is placed now: the graph is kept
    // while replicas come and go, and a kernel without a flagged replica returns)
    if (cells) {
        cudaKernelNodeParams k1{}, k2{}, kc{}, ks{}, kx{}, kf{};
        k1.func = (void *)k_cells;
        const unsigned gb = (unsigned)((d.N + 255) / 256);
        k1.gridDim = dim3(gb);
        k1.blockDim = dim3(256);
        k1.kernelParams = ac;
        add(k1);
        kc.func = (void *)k_cell_count;
        kc.gridDim = dim3(gb);
        kc.blockDim = dim3(256);
        kc.kernelParams = a1;
        add(kc);
        ks.func = (void *)k_cell_scan;
        ks.gridDim = dim3((unsigned)((d.ncells + CELL_SCAN - 1) / CELL_SCAN));
        ks.blockDim = dim3(256);
        ks.kernelParams = a3;
        add(ks);
        kx.func = (void *)k_cell_scatter;
        kx.gridDim = dim3(gb);
        kx.blockDim = dim3(256);
        kx.kernelParams = a3;
        add(kx);
        kf.func = (void *)k_cell_finish;
        kf.gridDim = dim3(2 * gb);
        kf.blockDim = dim3(256);
        kf.kernelParams = a1;
        add(kf);
        k2.func = (void *)k_nl_cells;
        k2.gridDim = dim3((d.N + NC_WARPS - 1) / NC_WARPS);
        k2.blockDim = dim3(NC_WARPS * 32);
        k2.kernelParams = a2;
        add(k2);
    }
    if (any_tile) {
        cudaKernelNodeParams kt{};
        kt.func = (void *)k_nl_tile;
        kt.gridDim = dim3(tile_grid);
        kt.blockDim = dim3(TL_THREADS);
        kt.sharedMemBytes = (unsigned)tile_smem;
        kt.kernelParams = a4;
        add(kt);
    }
    if (d.qa_on) {
        cudaKernelNodeParams k3{}, k5{}, k6{};
        k3.func = (void *)k_qa_fp_scan;
        k3.gridDim = dim3(d.qa.nbchunk);
        k3.blockDim = dim3(QA_BCHUNK);
        k3.kernelParams = a3;
        add(k3);
        k5.func = (void *)k_qa_fp_fill;
        k5.gridDim = dim3(d.qa.nbchunk, QA_FG);
        k5.blockDim = dim3(256);
        k5.kernelParams = a3;
        add(k5);
        k6.func = (void *)k_qa_compact;
        k6.gridDim = dim3(d.R);
        k6.blockDim = dim3(1024);
        k6.kernelParams = a3;
        add(k6);
    }
}

void Engine::check_status(const char *where) {
    fetch_words();
    const int st = h_any[4];
    CK(cudaGetLastError());
    if (st & ST_CAPACITY)
        throw std::length_error(std::string(where) + ": Verlet row capacity exceeded (raise `engine: nl capacity`)");
    if (st & ST_NONFINITE) {
        // reported once: the faulted replicas are frozen (a new state thaws
        // them); the other replicas of the context go on
        const int keep = st & ~ST_NONFINITE;
        CK(cudaMemcpyAsync(d.status, &keep, sizeof(int), cudaMemcpyHostToDevice, stream));
        CK(cudaStreamSynchronize(stream));
        if (!isolate_faults) throw std::domain_error(std::string(where) + ": non-finite force");
    }
}

void Engine::eval_forces(int rep, double *F, double *V) {
    check_rep(reps, rep);
    ready();
    ensure_nl();
    split_positions();
    CK(cudaMemsetAsync(d.Vrep, 0, sizeof(double) * XMD_NUM_TERMS * d.R, stream));
    launch_force(0, cur);
    const RepHost &h = reps[rep];
    std::vector<double> Ft;
    double *Fh = F;
    if (!Fh) {
        Ft.resize(3 * (size_t)h.n);
        Fh = Ft.data();
    }
    double *Vh = (double *)(h_any + 16);
    if (V) CK(cudaMemcpyAsync(Vh, d.Vrep + (size_t)rep * XMD_NUM_TERMS, sizeof(double) * XMD_NUM_TERMS,
                              cudaMemcpyDeviceToHost, stream));
    down(Fh, d.F + 3 * (size_t)h.begin, sizeof(double) * 3 * h.n);
    if (V) std::memcpy(V, Vh, sizeof(double) * XMD_NUM_TERMS);
    // only this replica's forces decide: a replica frozen by a non-finite
    // force does not fail the evaluation of the others
    const bool iso = isolate_faults;
    isolate_faults = true;
    try {
        check_status("eval_forces");
    } catch (...) {
        isolate_faults = iso;
        throw;
    }
    isolate_faults = iso;
    if (!all_finite(Fh, 3 * (size_t)h.n)) throw std::domain_error("eval_forces: non-finite force");
}

void Engine::step(int nsteps) {
    step_async(nsteps);
    // rows keep their contents when they grow: no list needs rebuilding, so
    // no replica's trajectory depends on another's row lengths
    step_wait();
}

// ---- packed host-buffer path ----------------------------------------------------
__global__ void k_unpack_history(Dev d, const double *__restrict__ y, int cur) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.N) return;
    const size_t n3 = 3 * (size_t)d.N;
    double4_32a p = d.pos[cur][i];
    p.x = y[3 * (size_t)i];
    p.y = y[3 * (size_t)i + 1];
    p.z = y[3 * (size_t)i + 2];
    d.pos[cur][i] = p;
    for (int ord = 1; ord < 6; ++ord)
        for (int a = 0; a < 3; ++a)
            d.yh[(size_t)((ord - 1) * 3 + a) * d.N + i] = y[ord * n3 + 3 * (size_t)i + a];
    // the skin test sees the new positions like any other displacement
    int r = d.rep_of[i];
    if (r < 0) return;
    double disp = dist2_exact(d.rep[r].box, p, d.orig[i]);   // squared, as k_force records it
    atomicMax(&d.rep[r].maxdisp, (unsigned long long)__double_as_longlong(disp));
}
__global__ void k_pack_positions(Dev d, double *__restrict__ r, int cur) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.N) return;
    double4_32a p = d.pos[cur][i];
    r[3 * (size_t)i] = p.x;
    r[3 * (size_t)i + 1] = p.y;
    r[3 * (size_t)i + 2] = p.z;
}

__global__ void k_pack_history(Dev d, double *__restrict__ y, int cur) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d.N) return;
    const size_t n3 = 3 * (size_t)d.N;
    double4_32a p = d.pos[cur][i];
    y[3 * (size_t)i] = p.x;
    y[3 * (size_t)i + 1] = p.y;
    y[3 * (size_t)i + 2] = p.z;
    for (int ord = 1; ord < 6; ++ord)
        for (int a = 0; a < 3; ++a)
            y[ord * n3 + 3 * (size_t)i + a] = d.yh[(size_t)((ord - 1) * 3 + a) * d.N + i];
}

void Engine::upload_history_all(const double *y) {
    use_device();
    ready();
    if (!staging) staging = (double *)dalloc(sizeof(double) * 18 * (size_t)d.N);
    CK(cudaMemcpyAsync(staging, y, sizeof(double) * 18 * (size_t)d.N, cudaMemcpyHostToDevice, stream));
    k_unpack_history<<<(d.N + 255) / 256, 256, 0, stream>>>(d, staging, cur);
    ++launches;
}

void Engine::download_history_all(double *y) {
    use_device();
    ready();
    if (!staging) staging = (double *)dalloc(sizeof(double) * 18 * (size_t)d.N);
    k_pack_history<<<(d.N + 255) / 256, 256, 0, stream>>>(d, staging, cur);
    ++launches;
    CK(cudaMemcpyAsync(y, staging, sizeof(double) * 18 * (size_t)d.N, cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
}

void Engine::download_positions_all(double *r) {
    use_device();
    ready();
    if (!staging) staging = (double *)dalloc(sizeof(double) * 18 * (size_t)d.N);
    k_pack_positions<<<(d.N + 255) / 256, 256, 0, stream>>>(d, staging, cur);
    ++launches;
    CK(cudaMemcpyAsync(r, staging, sizeof(double) * 3 * (size_t)d.N, cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
}

void Engine::stats(int64_t *out) {
    use_device();
    for (int k = 0; k < XMD_NUM_STATS; ++k) out[k] = 0;
    int64_t nb = 0;
    int64_t nr = 0;
    for (auto &r : reps)
        if (r.in_use) { nb += r.n; ++nr; }
    out[XMD_STAT_BEADS] = nb;
    out[XMD_STAT_REPLICAS] = nr;
    out[XMD_STAT_LAUNCHES] = launches;
    out[XMD_STAT_MD_STEPS] = md_steps;
    if (!finalized) return;
    std::vector<int32_t> cnt(d.N);
    CK(cudaMemcpyAsync(cnt.data(), d.nl_cnt, sizeof(int32_t) * d.N, cudaMemcpyDeviceToHost, stream));
    const int32_t nn = cap.nat;   // entries of free native ranges are kept at 0
    std::vector<uint8_t> on(nn > 0 ? nn : 1);
    if (nn) CK(cudaMemcpyAsync(on.data(), d.nat_on, nn, cudaMemcpyDeviceToHost, stream));
    std::vector<RepDev> rd(d.R);
    CK(cudaMemcpyAsync(rd.data(), d.rep, sizeof(RepDev) * d.R, cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    unsigned long long in_passes = 0;   // launches of the rebuild passes so far
    CK(cudaMemcpyAsync(&in_passes, d.ctr, sizeof(in_passes), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    out[XMD_STAT_LAUNCHES] = launches + (int64_t)in_passes;
    for (int i = 0; i < d.N; ++i)
        if (owner_h[i] >= 0) out[XMD_STAT_NL_ENTRIES] += cnt[i];
    for (int k = 0; k < nn; ++k) out[XMD_STAT_GO_ACTIVE] += on[k];
    for (auto &r : rd)
        if (r.active) out[XMD_STAT_REBUILDS] += (int64_t)r.rebuilds;
}

int Engine::qa_contacts(int rep, int cap, int32_t *out4, double *ref_time) {
    check_rep(reps, rep);
    ready();
    if (!d.qa_on) return 0;
    RepDev rd;
    CK(cudaMemcpyAsync(&rd, d.rep + rep, sizeof(RepDev), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    int n = rd.ct_n, o = rd.ct_off;
    std::vector<int32_t> i1(n), i2(n), ty(n);
    std::vector<uint8_t> st(n), vac(n);
    std::vector<double> rf(n);
    if (n) {
        CK(cudaMemcpyAsync(i1.data(), d.qa.ct_i1 + o, 4 * n, cudaMemcpyDeviceToHost, stream));
        CK(cudaMemcpyAsync(i2.data(), d.qa.ct_i2 + o, 4 * n, cudaMemcpyDeviceToHost, stream));
        CK(cudaMemcpyAsync(ty.data(), d.qa.ct_type + o, 4 * n, cudaMemcpyDeviceToHost, stream));
        CK(cudaMemcpyAsync(st.data(), d.qa.ct_status + o, n, cudaMemcpyDeviceToHost, stream));
        CK(cudaMemcpyAsync(vac.data(), d.qa.ct_vac + o, n, cudaMemcpyDeviceToHost, stream));
        CK(cudaMemcpyAsync(rf.data(), d.qa.ct_ref + o, 8 * n, cudaMemcpyDeviceToHost, stream));
        CK(cudaStreamSynchronize(stream));
    }
    int m = 0;
    const int b = reps[rep].begin;
    for (int k = 0; k < n; ++k) {
        if (vac[k]) continue;
        if (m < cap) {
            if (out4) {
                out4[4 * m] = i1[k] - b; out4[4 * m + 1] = i2[k] - b;
                out4[4 * m + 2] = ty[k]; out4[4 * m + 3] = st[k];
            }
            if (ref_time) ref_time[m] = rf[k];
        }
        ++m;
    }
    return m;
}

int Engine::verlet_pairs(int rep, int cap, int32_t *out2, uint8_t *flags) {
    check_rep(reps, rep);
    ready();
    ensure_nl();
    const RepHost &h = reps[rep];
    std::vector<int32_t> cnt(h.n), rows((size_t)nl_cap * h.n);
    CK(cudaMemcpyAsync(cnt.data(), d.nl_cnt + h.begin, sizeof(int32_t) * h.n, cudaMemcpyDeviceToHost, stream));
    for (int k = 0; k < nl_cap; ++k)
        CK(cudaMemcpyAsync(rows.data() + (size_t)k * h.n, d.nl_row + (size_t)k * d.N + h.begin,
                           sizeof(int32_t) * h.n, cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    std::vector<std::tuple<int, int, int>> v;
    for (int i = 0; i < h.n; ++i)
        for (int k = 0; k < cnt[i]; ++k) {
            int e = rows[(size_t)k * h.n + i];
            int j = (e & NL_MASK) - h.begin;
            if (j > i) v.emplace_back(i, j, ((e & NL_PAULI) ? 1 : 0) | ((e & NL_ES) ? 2 : 0) | ((e & NL_PID) ? 4 : 0));
        }
    std::sort(v.begin(), v.end());
    for (size_t k = 0; k < v.size() && (int)k < cap; ++k) {
        out2[2 * k] = std::get<0>(v[k]);
        out2[2 * k + 1] = std::get<1>(v[k]);
        if (flags) flags[k] = (uint8_t)std::get<2>(v[k]);
    }
    return (int)v.size();
}

void Engine::qa_sync(int rep, int8_t *out) {
    check_rep(reps, rep);
    ready();
    const RepHost &h = reps[rep];
    if (!d.qa_on) {
        for (int i = 0; i < h.n; ++i)
            for (int k = 0; k < 4; ++k) out[4 * i + k] = (int8_t)params.limits[h.atype[i]][k];
        return;
    }
    std::vector<int32_t> s(h.n);
    CK(cudaMemcpyAsync(s.data(), d.qa.sync + h.begin, 4 * (size_t)h.n, cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    for (int i = 0; i < h.n; ++i)
        for (int k = 0; k < 4; ++k) out[4 * i + k] = (int8_t)((s[i] >> (8 * k)) & 0xff);
}

void Engine::set_kernel_timing(bool on) {
    timing = on;
    n_ev_force = n_ev_rebuild = 0;
}

void Engine::kernel_times(double *force_ms, int64_t *nf, double *rebuild_ms, int64_t *nr) {
    use_device();
    CK(cudaStreamSynchronize(stream));
    double f = 0, r = 0;
    for (size_t k = 0; k + 1 < n_ev_force; k += 2) {
        float ms = 0;
        CK(cudaEventElapsedTime(&ms, ev_force[k], ev_force[k + 1]));
        f += ms;
    }
    for (size_t k = 0; k + 1 < n_ev_rebuild; k += 2) {
        float ms = 0;
        CK(cudaEventElapsedTime(&ms, ev_rebuild[k], ev_rebuild[k + 1]));
        r += ms;
    }
    if (force_ms) *force_ms = f;
    if (nf) *nf = (int64_t)(n_ev_force / 2);
    if (rebuild_ms) *rebuild_ms = r;
    if (nr) *nr = (int64_t)(n_ev_rebuild / 2);
}

void Engine::observables(int rep, double *E, double *K, double *Rg, double *Q) {
    check_rep(reps, rep);
    double V[XMD_NUM_TERMS];
    eval_forces(rep, nullptr, V);
    const RepHost &h = reps[rep];
    std::vector<double> r(3 * (size_t)h.n), v(3 * (size_t)h.n);
    get_state(rep, r.data(), v.data(), nullptr);
    double Vt = 0;
    for (double x : V) Vt += x;
    double K_ = 0;   // total_energy.cpp:4-11
    for (int i = 0; i < h.n; ++i)
        K_ += 0.5 * 1.0 * (v[3 * i] * v[3 * i] + v[3 * i + 1] * v[3 * i + 1] + v[3 * i + 2] * v[3 * i + 2]);
    double cm[3] = {0, 0, 0};   // gyration.cpp:4-19
    for (int i = 0; i < h.n; ++i) for (int a = 0; a < 3; ++a) cm[a] += r[3 * i + a];
    for (int a = 0; a < 3; ++a) cm[a] /= h.n;
    double g = 0;
    for (int i = 0; i < h.n; ++i)
        for (int a = 0; a < 3; ++a) g += (r[3 * i + a] - cm[a]) * (r[3 * i + a] - cm[a]);
    double act = 0;   // report_structure.cpp:85
    double thr = params.go_active_threshold * std::pow(2.0, -1.0 / 6.0);
    for (size_t k = 0; k < h.nat_i1.size(); ++k) {
        int a = h.nat_i1[k], b = h.nat_i2[k];
        double dx = r[3 * a] - r[3 * b], dy = r[3 * a + 1] - r[3 * b + 1], dz = r[3 * a + 2] - r[3 * b + 2];
        if (std::sqrt(dx * dx + dy * dy + dz * dz) < thr * h.nat_d[k]) act += 1;
    }
    if (E) *E = Vt + K_;
    if (K) *K = K_;
    if (Rg) *Rg = std::sqrt(g / h.n);
    if (Q) *Q = h.nat_i1.empty() ? 0.0 : act / h.nat_i1.size();
}

int Engine::device_status() {
    if (!finalized) return 0;
    int st = 0;
    CK(cudaMemcpyAsync(&st, d.status, sizeof(int), cudaMemcpyDeviceToHost, stream));
    CK(cudaStreamSynchronize(stream));
    return st;
}

void Engine::sync() { CK(cudaStreamSynchronize(stream)); }

}  // namespace xmdg
