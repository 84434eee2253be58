// step.cuh - the block of the step kernel (included by engine.cu).
//
// A block of FB bead slots takes FBT = FB - 5 beads, so that everything it
// derives from the chain geometry is one full round of FB lanes: FB bonds and
// cross products, FB - 2 bonded centres (the beads' own and three of the
// neighbours').  The work passes through shared memory in phases, each dealt
// so that whole warps do one thing with every lane busy (GB300 issues an FP64
// warp instruction over 16 cycles of the SM's FP64 pipe however few lanes
// are active, and the mixed path is bound by latency and issue):
//   A  the tile's positions; per bead its list lengths (prefix sum)
//   B  per slot: bond vector, cross product, their inverse lengths, once for
//      every term that uses them; beside it the beads' noise
//   D  per centre: tether + angle, and dihedral + chirality, on separate warps
//   E  pair entries: the lists of all beads of the block as one sequence,
//      one thread per entry whatever bead it belongs to, forces to shared
//      memory.  Warps without a part in B and D start here at once; every
//      warp takes the next 32 entries until none is left
//   F  one thread per (axis, bead): the bead's force summed in a fixed order,
//      then the integrator; G  new positions, skin test
// A bead's entries are its active native contacts, its Verlet row and its
// quasi-adiabatic contacts, summed in that order after the bonded forces: the
// trajectory is the same bits for every launch shape.
//
// What it measured, us per MD step, against a block whose threads kept to one
// bead each from list loops to integrator (bonded geometry formed per term, a
// third of the bonded warps with 3 live lanes, noise and skin test on a quarter
// of the lanes): 256 chains of 50-800 beads (66,007) FP64 458 -> 141, mixed
// 66 -> 44; 61 native chains mixed 38 -> 24; 16 x 500 periodic FP64 111 -> 40,
// mixed 32 -> 20; one chain of 100 beads FP64 54 -> 17.  FP64 is bound by its
// pipe (81 % active while blocks run) and the tail of the last wave, mixed by
// latency: index load, position load and arithmetic of a round of entries,
// the barriers between the phases, 32 warps per SM to hide them.
#pragma once

namespace xmdg {

template <int FB> constexpr int step_beads() { return FB - 5; }

// one term into the running force: FP64 rounded on its own; FP32 terms into a
// float-float sum whose low part collects the exact errors of the high part
__device__ __forceinline__ void sum_acc(double &a, double v) { a = __dadd_rn(a, v); }
__device__ __forceinline__ void sum_acc(FF &a, float v) {
    const FF s = two_sum(a.h, v);
    a.h = s.h;
    a.l = __fadd_rn(a.l, s.l);
}
__device__ __forceinline__ double sum_total(double a) { return a; }
__device__ __forceinline__ double sum_total(FF a) { return ff_to_d(a); }
template <class FT> struct StepSum { using T = double; };
template <> struct StepSum<float> { using T = FF; };

// dot and cross products with the contractions written out, so that every
// instantiation of the block rounds alike
template <class T> __device__ __forceinline__ T fma_(T a, T b, T c);
template <> __device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
template <> __device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_(float a, float b) { return __fadd_rn(a, b); }
template <class T> __device__ __forceinline__ T fdot(V3<T> a, V3<T> b) {
    return fma_<T>(a.x, b.x, fma_<T>(a.y, b.y, mul_(a.z, b.z)));
}
template <class T> __device__ __forceinline__ V3<T> fcross(V3<T> a, V3<T> b) {
    return V3<T>{fma_<T>(a.y, b.z, -mul_(a.z, b.y)), fma_<T>(a.z, b.x, -mul_(a.x, b.z)),
                 fma_<T>(a.x, b.y, -mul_(a.y, b.x))};
}
template <class T> __device__ __forceinline__ V3<T> fscl(T s, V3<T> a) {
    return V3<T>{mul_(s, a.x), mul_(s, a.y), mul_(s, a.z)};
}

// ---- noise of the FP64 path -------------------------------------------------------
// Box-Muller on the bead's next four 32-bit draws k / 2^32, in the order radius
// and angle of x and y, radius and angle of z (normal_x2 then normal,
// rand_gen.h:22-58, lang_pc.cpp:15-16), with the reductions done on the
// integer draws: no FP64 conversion, argument reduction or special-case path
// (84 FP64 instructions a bead; 150 with the library's log, sincos and cos).
// Results are within a few 2^-53 of the library's.
__device__ __forceinline__ double int_to_d(int k) {   // exact, one addition
    return __dsub_rn(__hiloint2double(0x43300000, (int)((unsigned)k ^ 0x80000000u)), 4503601774854144.0);
}
// sqrt(-2 log(k / 2^32)); k = 0 gives infinity, as log(0) does.  k / 2^32 =
// z 2^e with z in [0.75, 1.5); log z = log c + log1p(z / c - 1) with c from a
// table of 128 (c = 1 on both sides of 1, so that results near 0 keep their
// relative accuracy), log1p by its series to the 8th power (|r| <= 2^-7).
__device__ __forceinline__ double radius_of(unsigned k, const double2 *__restrict__ logt) {
    const int n = __clz((int)(k | 1u));
    const unsigned m = k << n;                    // leading one at bit 31
    const int j = (m >> 24) & 127;
    const bool up = j >= 64;
    const double z = __hiloint2double((up ? 0x3fe00000 : 0x3ff00000) | (int)((m & 0x7fffffffu) >> 11), (int)(m << 21));
    const double2 c = __ldg(logt + j);            // 1 / c, log c
    const double r = __fma_rn(z, c.x, -1.0);
    double q = __fma_rn(r, -0.125, 1.0 / 7.0);
    q = __fma_rn(r, q, -1.0 / 6.0);
    q = __fma_rn(r, q, 0.2);
    q = __fma_rn(r, q, -0.25);
    q = __fma_rn(r, q, 1.0 / 3.0);
    q = __fma_rn(r, q, -0.5);
    const double l1 = __fma_rn(__dmul_rn(r, r), q, r);
    const double e = int_to_d((up ? 0 : -1) - n);
    const double x = __dmul_rn(-2.0, __dadd_rn(__fma_rn(e, 0.6931471805599453, c.y), l1));
    const double y = rsqrt(x), w = __dmul_rn(x, y);   // the square root, with one Newton correction
    return k ? __fma_rn(__fma_rn(-w, w, x), __dmul_rn(0.5, y), w) : __longlong_as_double(0x7ff0000000000000ll);
}
// sine and cosine of 2 pi k / 2^32: the quadrant from the top bits, the rest in
// [-pi/4, pi/4] by Taylor series (remainders below 1e-19)
__device__ __forceinline__ double sin_series(double x, double x2) {
    double p = __fma_rn(x2, 2.8114572543455206e-15, -7.647163731819816e-13);
    p = __fma_rn(x2, p, 1.6059043836821613e-10);
    p = __fma_rn(x2, p, -2.505210838544172e-08);
    p = __fma_rn(x2, p, 2.7557319223985893e-06);
    p = __fma_rn(x2, p, -0.0001984126984126984);
    p = __fma_rn(x2, p, 0.008333333333333333);
    p = __fma_rn(x2, p, -0.16666666666666666);
    return __fma_rn(__dmul_rn(x, x2), p, x);
}
__device__ __forceinline__ double cos_series(double x2) {
    double p = __fma_rn(x2, 4.779477332387385e-14, -1.1470745597729725e-11);
    p = __fma_rn(x2, p, 2.08767569878681e-09);
    p = __fma_rn(x2, p, -2.755731922398589e-07);
    p = __fma_rn(x2, p, 2.48015873015873e-05);
    p = __fma_rn(x2, p, -0.001388888888888889);
    p = __fma_rn(x2, p, 0.041666666666666664);
    p = __fma_rn(x2, p, -0.5);
    return __fma_rn(x2, p, 1.0);
}
__device__ __forceinline__ double turn_rest(unsigned k, unsigned *quad) {
    *quad = (k + 0x20000000u) >> 30;
    return __dmul_rn(int_to_d((int)(k - (*quad << 30))), 1.4629180792671596e-09);   // 2 pi / 2^32
}
__device__ __forceinline__ double flip(double x, unsigned neg) {
    return __hiloint2double(__double2hiint(x) ^ (int)(neg << 31), __double2loint(x));
}
__device__ __forceinline__ void noise3_turns(uint64_t st, const double2 *logt, double *nx, double *ny, double *nz) {
    const unsigned k1 = (unsigned)(rng_next(st) >> 32), k2 = (unsigned)(rng_next(st) >> 32);
    const unsigned k3 = (unsigned)(rng_next(st) >> 32), k4 = (unsigned)(rng_next(st) >> 32);
    unsigned q;
    double x = turn_rest(k2, &q), x2 = __dmul_rn(x, x);
    const double s = sin_series(x, x2), c = cos_series(x2), r = radius_of(k1, logt);
    // quadrants 0..3: cos = c, -s, -c, s; sin = s, c, -s, -c
    *nx = __dmul_rn(r, flip(q & 1 ? s : c, (q ^ (q >> 1)) & 1));
    *ny = __dmul_rn(r, flip(q & 1 ? c : s, q >> 1));
    x = turn_rest(k4, &q);
    x2 = __dmul_rn(x, x);
    *nz = __dmul_rn(radius_of(k3, logt), flip(q & 1 ? sin_series(x, x2) : cos_series(x2), (q ^ (q >> 1)) & 1));
}

// ---- geometry slots -------------------------------------------------------------
// FP64: bond e (3), unit cross product u (3), |e|, 1/|e|, 1/|x|.  Bonds, cross
// products, lengths and units are formed with every operation rounded on its
// own, as the reference's uncontracted build forms them: on extended starts
// triples are straight to ~1e-6 rad, where a contracted cross product moves
// a dihedral force by 1e-10 of itself.
// Mixed: bond and cross product in float-float (6 + 6), 1/|e|, 1/|x|, |e|, |x|.
enum : int { GE = 0, GU = 3, GLEN = 6, GRN = 7, GRX = 8, GN64 = 9 };
enum : int { MEH = 0, MEL = 3, MXH = 6, MXL = 9, MRN = 12, MRX = 13, MLEN = 14, MLX = 15, GN32 = 16 };

// energies of the evaluation pass: per thread for the block's first replica,
// reduced over the warp at the end; other replicas at once
enum : int { EV_N = XMD_NUM_TERMS };
template <int MODE> struct Ener {
    __device__ __forceinline__ void add(const Dev &, int, int, double) {}
    __device__ __forceinline__ void flush(const Dev &) {}
    __device__ __forceinline__ void start(int) {}
};
template <> struct Ener<0> {
    double v[EV_N];
    int r0;
    __device__ __forceinline__ void start(int r) {
        r0 = r;
#pragma unroll
        for (int k = 0; k < EV_N; ++k) v[k] = 0.0;
    }
    __device__ __forceinline__ void add(const Dev &d, int r, int term, double e) {
        if (r == r0) {
#pragma unroll
            for (int k = 0; k < EV_N; ++k)
                if (k == term) v[k] += e;
        } else {
            atomicAdd(&d.Vrep[r * XMD_NUM_TERMS + term], e);
        }
    }
    __device__ __forceinline__ void flush(const Dev &d) {
        if (r0 < 0) return;
#pragma unroll
        for (int k = 0; k < EV_N; ++k) {
            double e = v[k];
            if (!__any_sync(0xffffffffu, e != 0.0)) continue;
            for (int o = 16; o; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
            if ((threadIdx.x & 31) == 0) atomicAdd(&d.Vrep[r0 * XMD_NUM_TERMS + k], e);
        }
    }
};

// ---- bonded centres ----------------------------------------------------------------
// a centre's parameters: bond length, angle, cosine and sine of the dihedral
// (mixed: the dihedral itself)
template <class FT> struct CentreP { FT r0, t0, c0, s0; };
template <> struct CentreP<float> { float r0, t0, p0; };

// sp: the centre's position slot.  g: geometry slots [.][FB].

// tether (c, c+1), angle (c-1, c, c+1): the force on c from its bond, the
// angle's forces on c-1 and c+1 (on c: minus their sum)
template <class FT, int MODE, int FB>
__device__ __forceinline__ void bond_angle(const Dev &d, const TermP &p, const FT (*g)[FB], int sp, uint32_t fl,
                                           const CentreP<FT> &cp, bool own, int rc, Ener<MODE> &en, V3<FT> *ft,
                                           V3<FT> *a1, V3<FT> *a2, V3<FT> *a3) {
    constexpr bool MIX = sizeof(FT) == 4;
    const bool h_ang = (fl & BF_HANG) && p.on[XMD_TERM_HEUR_ANG];
    const bool do_ang = ((fl & BF_ANG) && p.on[XMD_TERM_NAT_ANG]) || h_ang;
    const double *hac = h_ang ? d.heur_ang + 7 * ((fl >> BF_HANG_SHIFT) & 15u) : nullptr;
    const V3<FT> e1{g[0][sp - 1], g[1][sp - 1], g[2][sp - 1]}, e2{g[0][sp], g[1][sp], g[2][sp]};
    const FT rn1 = g[MIX ? MRN : GRN][sp - 1], rn2 = g[MIX ? MRN : GRN][sp];
    if ((fl & BF_TETH) && p.on[XMD_TERM_TETHER]) {
        // eval_tether_forces::iter tether.cpp:21-36, harmonic.h:18-25
        FT V_;
        if constexpr (MIX) {
            *ft = tether_mixed(p, e2, g[MLEN][sp], rn2, cp.r0, &V_);
        } else {
            const double dr = g[GLEN][sp] - cp.r0, dr2 = mul_(dr, dr);
            double dV = mul_(dr, fma_<double>(mul_(2.0, p.tether_H2), dr2, p.tether_H1));
            dV = clampv<double>(dV, -1.0e3, 1.0e3);
            *ft = fscl<double>(mul_(dV, rn2), e2);
            V_ = clampv<double>(mul_(mul_(0.5, dr2), fma_<double>(p.tether_H2, dr2, p.tether_H1)), -1.0e3, 1.0e3);
        }
        if (MODE == 0 && own) en.add(d, rc, XMD_TERM_TETHER, (double)V_);
    }
    if (do_ang) {
        // eval_native_angle_forces::iter angle/native.cpp:13-39
        double V_ = 0.0;
        if constexpr (MIX) {
            const V3<float> x{g[MXH][sp], g[MXH + 1][sp], g[MXH + 2][sp]};
            float Vf;
            angle_mixed(p, e1, e2, x, rn1, rn2, g[MLX][sp], cp.t0, hac, a1, a2, a3, &Vf);
            V_ = (double)Vf;
        } else {
            // the cross products of the bonds with the plane's unit normal have
            // lengths |r12| and |r23| (the bonds lie in the plane), so the
            // reference's unit vectors along them need no further square root
            const V3<double> u{g[GU][sp], g[GU + 1][sp], g[GU + 2][sp]};
            const V3<DN> b1{e1.x, e1.y, e1.z}, b2{e2.x, e2.y, e2.z};
            const double theta = acos_c<DN>(-dot(b1, b2) * DN(rn1) * DN(rn2)).v;
            double dV;
            if (hac) {
                const double2 vd = heur_poly_nl(hac, theta);
                V_ = vd.x;
                dV = vd.y;
            } else {
                const double dt = theta - cp.t0;
                dV = mul_(p.nat_ang_k, dt);
                if (MODE == 0) V_ = mul_(0.5, mul_(dV, dt));
            }
            *a1 = fscl<double>(-mul_(dV, mul_(rn1, rn1)), fcross(e1, u));
            *a3 = fscl<double>(-mul_(dV, mul_(rn2, rn2)), fcross(e2, u));
            *a2 = V3<double>{-add_(a1->x, a3->x), -add_(a1->y, a3->y), -add_(a1->z, a3->z)};
        }
        if (MODE == 0 && own) en.add(d, rc, h_ang ? XMD_TERM_HEUR_ANG : XMD_TERM_NAT_ANG, V_);
    }
}

// dihedral and chirality of (c-1, c, c+1, c+2): forces on the four beads
template <class FT, int MODE, int FB>
__device__ __forceinline__ void dihedral_chiral(const Dev &d, const TermP &p, const FT (*g)[FB], int c, int sp,
                                                uint32_t fl, const CentreP<FT> &cp, bool own, int rc, Ener<MODE> &en,
                                                V3<FT> *q) {
    constexpr bool MIX = sizeof(FT) == 4;
    const bool h_dih = (fl & BF_HDIH) && p.on[XMD_TERM_HEUR_DIH];
    const bool do_dih = ((fl & BF_DIH) && (p.on[XMD_TERM_CND] || p.on[XMD_TERM_SND])) || h_dih;
    const int hdt = (int)((fl >> BF_HDIH_SHIFT) & 15u);
    const V3<FT> e1{g[0][sp - 1], g[1][sp - 1], g[2][sp - 1]}, e2{g[0][sp], g[1][sp], g[2][sp]},
        e3{g[0][sp + 1], g[1][sp + 1], g[2][sp + 1]};
    if (do_dih) {
        // eval_cnd_forces::iter dihedral/complex_native.cpp:13-49,
        // eval_snd_forces::iter dihedral/simple_native.cpp:13-45
        double Vc = 0.0, Vs = 0.0;
        if constexpr (MIX) {
            const V3<float> x1{g[MXH][sp], g[MXH + 1][sp], g[MXH + 2][sp]},
                x2{g[MXH][sp + 1], g[MXH + 1][sp + 1], g[MXH + 2][sp + 1]};
            // the triple product in float-float: small against its factors for
            // flat quads
            const V3<FF> xf{FF{x1.x, g[MXL][sp]}, FF{x1.y, g[MXL + 1][sp]}, FF{x1.z, g[MXL + 2][sp]}};
            const V3<FF> ef{FF{e3.x, g[MEL][sp + 1]}, FF{e3.y, g[MEL + 1][sp + 1]}, FF{e3.z, g[MEL + 2][sp + 1]}};
            float Vcf, Vsf;
            dihedral_mixed(p, e1, e2, e3, x1, x2, g[MLEN][sp], g[MRX][sp], g[MRX][sp + 1], dot(x1, x2),
                           ff_dot(xf, ef).h, cp.p0, p.on[XMD_TERM_CND] != 0, p.on[XMD_TERM_SND] != 0,
                           h_dih ? d.heur_dih_f + 6 * hdt : nullptr, q, &Vcf, &Vsf);
            Vc = (double)Vcf;
            Vs = (double)Vsf;
        } else {
            // sine and cosine of phi come from the geometry, those of
            // phi - phi0 and 3 (phi - phi0) by the addition theorems: no arc
            // cosine and no sine of an angle, except for the terms that need
            // phi itself
            const double rx1 = g[GRX][sp], rx2 = g[GRX][sp + 1], rn2 = g[GRN][sp], len2 = g[GLEN][sp];
            const V3<double> u1{g[GU][sp], g[GU + 1][sp], g[GU + 2][sp]},
                u2{g[GU][sp + 1], g[GU + 1][sp + 1], g[GU + 2][sp + 1]};
            // the cosine as the reference rounds it, clamped; the sine of its
            // arc cosine is sqrt((1 - c)(1 + c))
            const V3<DN> a{u1.x, u1.y, u1.z}, b{u2.x, u2.y, u2.z};
            const double cphi = clampv<double>(dot(a, b).v, -1.0, 1.0);
            const double s2 = __dmul_rn(__dsub_rn(1.0, cphi), __dadd_rn(1.0, cphi));
            double sphi = s2 > 0.0 ? __dmul_rn(s2, rsqrt(s2)) : s2;
            const double tsign = fdot(u1, e3);
            if (tsign < 0.0) sphi = -sphi;
            double dV = 0.0;
            if (h_dih) {
                heur_dih_nl<double>(d.heur_dih + 6 * hdt, sphi, cphi, &Vc, &dV);
            } else if (p.on[XMD_TERM_CND]) {
                const double c0 = cp.c0, s0 = cp.s0, CDA = p.cnd_CDA, CDB = p.cnd_CDB;
                const double sd = fma_<double>(sphi, c0, -mul_(cphi, s0));
                // sin 3x = sin x (3 - 4 sin^2 x), cos 3x = cos x (1 - 4 sin^2 x)
                const double sd2 = mul_(sd, sd), s3 = mul_(sd, fma_<double>(-4.0, sd2, 3.0));
                dV = fma_<double>(mul_(3.0, CDB), s3, mul_(CDA, sd));
                if (MODE == 0) {
                    const double cd = fma_<double>(cphi, c0, mul_(sphi, s0));
                    const double c3 = mul_(cd, fma_<double>(-4.0, sd2, 1.0));
                    // 1 - cos x = sin^2 x / (1 + cos x), without cancellation at the minimum
                    const double v1 = cd > 0.0 ? sd2 / (1.0 + cd) : 1.0 - cd;
                    const double v3 = c3 > 0.0 ? s3 * s3 / (1.0 + c3) : 1.0 - c3;
                    Vc = CDA * v1 + CDB * v3;
                }
            }
            if (p.on[XMD_TERM_SND] && !h_dih) {
                double phi = acos(cphi);
                if (tsign < 0.0) phi = -phi;
                const double df = phi - d.dih_p0[c];
                dV = fma_<double>(p.snd_CDH, df, dV);
                Vs = 0.5 * p.snd_CDH * df * df;
            }
            const double k = mul_(dV, len2), iden = mul_(rn2, rn2);
            q[0] = fscl<double>(mul_(k, rx1), u1);
            q[3] = fscl<double>(-mul_(k, rx2), u2);
            const double k1 = mul_(fdot(e1, e2), iden), k4 = mul_(fdot(e2, e3), iden);
            const V3<double> w{fma_<double>(q[0].x, k1, -mul_(q[3].x, k4)), fma_<double>(q[0].y, k1, -mul_(q[3].y, k4)),
                               fma_<double>(q[0].z, k1, -mul_(q[3].z, k4))};
            q[1] = V3<double>{-add_(q[0].x, w.x), -add_(q[0].y, w.y), -add_(q[0].z, w.z)};
            q[2] = V3<double>{add_(w.x, -q[3].x), add_(w.y, -q[3].y), add_(w.z, -q[3].z)};
        }
        if (MODE == 0 && own) {
            if (h_dih) en.add(d, rc, XMD_TERM_HEUR_DIH, Vc);
            else {
                if (p.on[XMD_TERM_CND]) en.add(d, rc, XMD_TERM_CND, Vc);
                if (p.on[XMD_TERM_SND]) en.add(d, rc, XMD_TERM_SND, Vs);
            }
        }
    }
    if ((fl & BF_CHIR) && p.on[XMD_TERM_CHIR]) {
        // eval_chiral_forces::iter chiral.cpp:15-37
        V3<FT> h[4];
        double Vch;
        if constexpr (MIX) {
            const float2 ch = d.chir_f32[c];
            const V3<float> x1{g[MXH][sp], g[MXH + 1][sp], g[MXH + 2][sp]},
                x2{g[MXH][sp + 1], g[MXH + 1][sp + 1], g[MXH + 2][sp + 1]};
            const V3<FF> ef{FF{e1.x, g[MEL][sp - 1]}, FF{e1.y, g[MEL + 1][sp - 1]}, FF{e1.z, g[MEL + 2][sp - 1]}};
            const V3<FF> xf{FF{x2.x, g[MXL][sp + 1]}, FF{x2.y, g[MXL + 1][sp + 1]}, FF{x2.z, g[MXL + 2][sp + 1]}};
            float Vf;
            chiral_mixed(p, e1, e2, e3, x1, x2, ff_dot(ef, xf).h, ch.x, ch.y, h, &Vf);
            Vch = (double)Vf;
        } else {
            const double2 ch = d.chir[c];
            V3<DN> gn[4];
            DN Vn;
            const V3<DN> b1{e1.x, e1.y, e1.z}, b2{e2.x, e2.y, e2.z}, b3{e3.x, e3.y, e3.z};
            chiral_bonds<DN>(p, b1, b2, b3, DN(ch.x), DN(ch.y), gn, &Vn);
#pragma unroll
            for (int k = 0; k < 4; ++k) h[k] = v3d(gn[k]);
            Vch = (double)Vn;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = q[k] + h[k];
        if (MODE == 0 && own) en.add(d, rc, XMD_TERM_CHIR, Vch);
    }
}

// ---- the block ----------------------------------------------------------------------
template <class FT, int FB> struct StepSh {
    static constexpr bool MIX = sizeof(FT) == 4;
    // pair forces held at once; a block with more entries takes several passes
    static constexpr int FCAP = FB <= 32 ? 512 : 8 * FB;
    double F[3][FB];                  // new positions
    uint64_t rng[FB];                 // generator states after the step
    FT p[MIX ? 7 : 4][FB + 4];        // positions; mixed: h, l per axis, charge; FP64: x, y, z, charge
    FT g[MIX ? (int)GN32 : (int)GN64][FB];   // geometry
    FT c[24][FB];                     // centre forces: tether, angle on c-1, c, c+1, dihedral on c-1 .. c+2
    FT f[3][FCAP];                    // pair forces
    // mixed: the second force of entries with two, and which those are
    FT f2[3][MIX ? FCAP : 1];
    unsigned two[MIX ? FCAP / 32 : 1];
    FT n[3][FB];                      // noise
    FT e[3][FB];                      // skin-test displacement per axis (FP64: squared)
    // FP64: electrostatic entries set aside (their charge product, and which)
    FT ew[MIX ? 1 : FCAP];
    int eq[MIX ? 1 : FCAP], neq, next_es;
    int off[FB + 4], ng[FB], nl[FB], nat0[FB], rep[FB], state[FB], per[FB], ss0[FB], ss1[FB], ws[4], next;
    // followed, in contexts with the quasi-adiabatic term, by the beads'
    // contact slots in ascending order, int [FB][QA_REF_CAP]
};
template <class FT, int FB> constexpr size_t step_smem(bool qa) {
    return (sizeof(StepSh<FT, FB>) + 15) / 16 * 16 + (qa ? sizeof(int) * QA_REF_CAP * FB : 0);
}

// Debye-Hueckel force factor of the FP64 path: eval_const_es_forces::iter
// es/const.cpp:13-32, eval_relative_es_forces::iter es/relative.cpp:13-32
__device__ __forceinline__ double es_factor(const TermP &p, double vq, double len, double rn, double *V) {
    *V = mul_(mul_(vq, exp_(-mul_(len, p.es_sdi))), mul_(rn, rn));
    return -mul_(*V, fma_<double>(p.es_rel ? 2.0 : 1.0, rn, p.es_sdi));
}

// a pair entry of the block: its bead's slot, the partner, the row's flags (0:
// a native contact of length rm), the contact slot (-1: none)
template <class FT> struct PairRef { int lo, j, ent, slot; FT rm; };
template <class FT, int FB>
__device__ __forceinline__ PairRef<FT> pair_fetch(const Dev &d, const TermP &p, const StepSh<FT, FB> &s,
                                                  const int (*s_q)[QA_REF_CAP], int i0, int e, bool on) {
    PairRef<FT> q{0, -1, 0, -1, FT(0)};
    if (!on) return q;
    // the entry's bead: the last one that starts at or before it
    int lo = 0;
#pragma unroll
    for (int h = FB / 2; h; h >>= 1)
        if (s.off[lo + h] <= e) lo += h;
    const int i = i0 + lo, m = e - s.off[lo], k = m - s.ng[lo];
    q.lo = lo;
    if (k < s.nl[lo]) {
        // one load for both lists, so that it diverges nowhere
        const int at = s.nat0[lo] + m;
        const int32_t *src = k < 0 ? d.act_j + at : d.nl_row + (size_t)k * d.N + i;
        const int v = *src;
        if (k < 0) {
            const double nd = d.act_d[at];
            if constexpr (sizeof(FT) == 4) q.rm = narrow_f(nd);
            else q.rm = nd;
            q.j = v;
        } else {
            q.ent = v;
            q.j = v & (NL_PAULI | NL_ES) ? v & NL_MASK : -1;   // or a PID bundle only
            q.rm = tpar<FT>(p.pauli_r_excl, p.f.pauli_r_excl);
        }
    } else {
        q.slot = s_q[lo][k - s.nl[lo]];
        const int x = d.qa.ct_i1[q.slot];
        q.j = x == i ? d.qa.ct_i2[q.slot] : x;
    }
    return q;
}
// the partner's position, and the pair vector from it
template <class FT> struct PairPos { double4_32a p; };
template <> struct PairPos<float> { float4 h, l; };
template <class FT> __device__ __forceinline__ PairPos<FT> pair_pos(const Dev &d, int cur, int j) {
    PairPos<FT> x{};
    if constexpr (sizeof(FT) == 4) {
        if (j >= 0) {
            x.h = d.spl[cur][2 * (size_t)j];
            x.l = d.spl[cur][2 * (size_t)j + 1];
        }
    } else {
        if (j >= 0) x.p = d.pos[cur][j];
    }
    return x;
}

// force of a pair entry on its bead.
// Mixed: a pair on both the Pauli and the electrostatic list has two forces,
// which enter the bead's sum one after the other: the second one goes to *two
// and the entry says so.
// FP64: the electrostatic part (an exponential, half the pair's FP64 work) is
// set aside when it is all there is to the pair: *es gets its charge factor
// and the pair vector is returned, so that whole warps of such pairs do it
// later instead of every warp that holds one.
// Returns what became of it.
enum : int { PE_DONE = 0, PE_TWO = 1, PE_ES = 2 };
template <class FT, int MODE, int FB>
__device__ __forceinline__ int pair_entry(const Dev &d, const TermP &p, const StepSh<FT, FB> &s, int i0,
                                          const PairRef<FT> &e, const PairPos<FT> &x, Ener<MODE> &en, V3<FT> *f,
                                          V3<FT> *two, FT *es) {
    constexpr bool MIX = sizeof(FT) == 4;
    const int lo = e.lo, i = i0 + lo, j = e.j, ent = e.ent, slot = e.slot;
    const FT rm = e.rm;
    *f = V3<FT>{FT(0), FT(0), FT(0)};
    if (j < 0) return PE_DONE;
    const int r = s.rep[lo];
    const RepDev &rp = d.rep[r];
    V3<FT> r12;
    FT qj, rn, len;
    if constexpr (MIX) {
        const F2 pa[3] = {{s.p[0][lo + 3], s.p[3][lo + 3]}, {s.p[1][lo + 3], s.p[4][lo + 3]},
                          {s.p[2][lo + 3], s.p[5][lo + 3]}};
        const F2 pb[3] = {{x.h.x, x.l.x}, {x.h.y, x.l.y}, {x.h.z, x.l.z}};
        r12 = pair_vec(rp, s.per[lo] != 0, pa, pb);
        qj = x.h.w;
        len = norm(r12);
        rn = 1.0f / len;
    } else {
        const double4_32a pi = make_double4_32a(s.p[0][lo + 3], s.p[1][lo + 3], s.p[2][lo + 3], 0.0);
        r12 = r_uv_p<double>(rp.box, s.per[lo] != 0, pi, x.p);
        qj = x.p.w;
        const double s2 = fdot(r12, r12);
        rn = rsqrt(s2);
        len = mul_(rn, s2);
    }
    FT dV = FT(0);
    if (slot >= 0) {
        // quasi-adiabatic contact: the force part of process_contacts::iter
        // (process_contacts.cpp:25-40)
        double sat = fmin(rp.t - d.qa.ct_ref[slot], p.qa_cycle) * p.qa_cycle_inv;
        if (d.qa.ct_status[slot] == QA_BREAKING) sat = 1.0 - sat;
        double depth, rmin, rmax;
        qa_lj(p, d.qa, d.qa.ct_type[slot], &depth, &rmin, &rmax);
        FT V_, dq;
        if constexpr (MIX) len = rn * nsq(r12);
        sink_lj_eval<FT>((FT)depth, (FT)rmin, (FT)rmax, len, rn, &V_, &dq);
        dV = mul_((FT)sat, dq);
        if (MODE == 0 && i < j) en.add(d, r, XMD_TERM_QA, sat * (double)V_);
    } else {
        // Go (go.cpp:31-46, lj.h:22-30) and Pauli (pauli.cpp:32-48,
        // shifted_lj.h:14-21) have one force law, Pauli inside r_excl only
        const bool go = ent == 0;
        const FT w = mul_(rn, rm);
        const bool lj = go || ((ent & NL_PAULI) && FT(1) < w);
        if (lj) {
            const FT depth = go ? tpar<FT>(p.go_depth, p.f.go_depth) : tpar<FT>(p.pauli_depth, p.f.pauli_depth);
            FT V_;
            if constexpr (MIX) {
                lj_mixed(depth, rm, rn, go ? 0.0f : 1.0f, &V_, &dV);
            } else {
                const double w2 = mul_(w, w), w3 = mul_(w2, w), s6 = mul_(w3, w3);
                // s6 - s12 = s6 (1 - s6)
                dV = mul_(mul_(mul_(12.0, depth), rn), mul_(s6, add_(1.0, -s6)));
                dV = clampv<double>(dV, -1.0e3, 1.0e3);
                V_ = mul_(depth, add_(mul_(s6, add_(s6, -2.0)), go ? 0.0 : 1.0));
                V_ = clampv<double>(V_, -1.0e3, 1.0e3);
            }
            if (MODE == 0 && i < j) en.add(d, r, go ? XMD_TERM_GO : XMD_TERM_PAULI, (double)V_);
        }
        if (ent & NL_ES) {
            FT V_;
            if constexpr (MIX) {
                const float dE = es_mixed(p, len, rn, __fmul_rn(s.p[6][lo + 3], qj), &V_);
                if (MODE == 0 && i < j) en.add(d, r, p.es_rel ? XMD_TERM_REL_ES : XMD_TERM_CONST_ES, (double)V_);
                if (lj) {
                    const V3<float> u = rn * r12;
                    *f = dV * u;
                    *two = dE * u;
                    return PE_TWO;
                }
                dV = dE;
            } else {
                const double vq = mul_(p.es_Vf, mul_(s.p[3][lo + 3], qj));
                if (MODE == 1 && dV == 0.0) {
                    *es = vq;
                    *f = r12;
                    return PE_ES;
                }
                dV = add_(dV, es_factor(p, vq, len, rn, &V_));
                if (MODE == 0 && i < j) en.add(d, r, p.es_rel ? XMD_TERM_REL_ES : XMD_TERM_CONST_ES, V_);
            }
        }
    }
    if constexpr (MIX) *f = dV * (rn * r12);
    else *f = fscl<double>(mul_(dV, rn), r12);
    return PE_DONE;
}

// MODE 0: forces and per-term energies at pos[cur] (eval).
// MODE 1: forces, then one Langevin predictor-corrector step (lang_pc.cpp:5-41)
//         writing pos[cur^1], y1..y5, the generator state and the skin-test
//         displacement (verify.cpp:10-15).
// gated: the kernel does nothing while the gate is closed; returns whether it
// was open.
template <class FT, int MODE, int FB, int LPB>
__device__ __forceinline__ bool force_block(const Dev &d, const TermP &p, int cur, bool gated) {
    constexpr bool MIX = sizeof(FT) == 4;
    constexpr int NT = FB * LPB;
    constexpr int FBT = step_beads<FB>(), NP = FB + 1, NC = FBT + 3;
    constexpr int FCAP = StepSh<FT, FB>::FCAP;
    // first thread of the (axis, bead) tasks: with four threads per slot or
    // more, past the warps of the geometry and the angles
    constexpr int W0 = LPB >= 4 ? FB : 0;
    constexpr int TT = (3 * FBT + NT - W0 - 1) / (NT - W0);   // tasks per thread
    static_assert(LPB < 4 || TT == 1, "one task per thread");
    using ST = typename StepSum<FT>::T;
    extern __shared__ __align__(16) unsigned char step_mem[];
    StepSh<FT, FB> &s = *reinterpret_cast<StepSh<FT, FB> *>(step_mem);
    int(*const s_q)[QA_REF_CAP] = reinterpret_cast<int(*)[QA_REF_CAP]>(step_mem + step_smem<FT, FB>(false));
    const int N = d.N, t = threadIdx.x, i0 = blockIdx.x * FBT, lane = t & 31;
    const size_t Ns = (size_t)N;
    const bool qa = d.qa_on && p.on[XMD_TERM_QA];
    const unsigned FULL = 0xffffffffu;

    // ---- A: what no kernel writes is loaded before the kernels before this
    // one have finished: owners, flags and parameters of the thread's centre,
    // the native ranges
    const int r = t < FBT && i0 + t < N ? d.rep_of[i0 + t] : -1;   // replica of bead t
    const int sc = t & (FB - 1), c = i0 - 2 + sc;                  // the thread's centre (t < 2 FB)
    uint32_t fl = 0;
    CentreP<FT> cp{};
    if (t < 2 * FB && sc < NC && c >= 0 && c < N) {
        fl = d.bflags[c];
        if constexpr (MIX) {
            const float4 q = d.bond_f[c];
            cp = CentreP<float>{q.x, q.y, q.z};
        } else {
            if (LPB == 1 || t < FB) { cp.r0 = d.teth_r0[c]; cp.t0 = d.ang_t0[c]; }
            if (LPB == 1 || t >= FB) { const double2 q = d.dih_cs[c]; cp.c0 = q.x; cp.s0 = q.y; }
        }
    }
    int nat0 = 0, ss0 = 0, ss1 = 0;
    if (t < FBT && i0 + t < N) {
        nat0 = d.nat_start[i0 + t];
        if (p.on[XMD_TERM_NAT_SS]) {
            ss0 = d.ss_start[i0 + t];
            ss1 = d.ss_end[i0 + t];
        }
    }
    step_order();
    if (gated && d.gate[0]) return false;   // uniform: the gate changes between launches

    // the tile, the list lengths, and what later phases load without needing
    // a result, so that its latency passes once
    const int bn = LPB == 1 ? t : t - FB;                          // the bead whose noise this thread draws
    const bool draws = MODE == 1 && bn >= 0 && bn < FBT && i0 + bn < N;
    uint64_t st0 = 0;
    if (draws) st0 = d.rng[i0 + bn];
    int ng = 0, nl = 0, nq = 0;
    long long left = -1;
    if (t < FBT && i0 + t < N) {
        if (MODE == 1) left = d.rep[max(r, 0)].steps_left;
        nl = d.nl_cnt[i0 + t];
        if (p.on[XMD_TERM_GO]) ng = d.go_cnt[i0 + t];
        if (qa) nq = min(d.qa.ref_cnt[i0 + t], QA_REF_CAP);
    }
    double y[TT][6], o[TT];
#pragma unroll
    for (int u = 0; u < TT; ++u) {
        const int w = t - W0 + u * NT, a = w / FBT, i = i0 + w - a * FBT;
        o[u] = 0.0;
#pragma unroll
        for (int q = 0; q < 6; ++q) y[u][q] = 0.0;
        if (MODE == 1 && w >= 0 && w < 3 * FBT && i < N) {
            y[u][0] = reinterpret_cast<const double *>(d.pos[cur] + i)[a];
#pragma unroll
            for (int q = 0; q < 5; ++q) y[u][q + 1] = d.yh[(size_t)(q * 3 + a) * Ns + i];
            o[u] = reinterpret_cast<const double *>(d.orig + i)[a];
        }
    }
    for (int k = t; k < NP; k += NT) {
        const int idx = i0 - 3 + k;
        const bool ok = idx >= 0 && idx < N;
        if constexpr (MIX) {
            const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float4 h = ok ? d.spl[cur][2 * (size_t)idx] : z, l = ok ? d.spl[cur][2 * (size_t)idx + 1] : z;
            s.p[0][k] = h.x; s.p[1][k] = h.y; s.p[2][k] = h.z;
            s.p[3][k] = l.x; s.p[4][k] = l.y; s.p[5][k] = l.z;
            s.p[6][k] = h.w;
        } else {
            const double4_32a q = ok ? d.pos[cur][idx] : make_double4_32a(0, 0, 0, 0);
            s.p[0][k] = q.x; s.p[1][k] = q.y; s.p[2][k] = q.z; s.p[3][k] = q.w;
        }
    }
    // 1: the bead steps, 0: its replica has taken its steps (or is frozen) and
    // keeps its state, -1: free slot
    const int state = r < 0 ? -1 : left != 0;
    int scan = 0, cnt = 0;
    if (t < FB) {
        if (state != 1) ng = nl = nq = 0;
        scan = cnt = ng + nl + nq;
#pragma unroll
        for (int o_ = 1; o_ < 32; o_ <<= 1) {
            const int x = __shfl_up_sync(FULL, scan, o_);
            if (lane >= o_) scan += x;
        }
        if (lane == 31) s.ws[t >> 5] = scan;
        s.ng[t] = ng; s.nl[t] = nl; s.nat0[t] = nat0; s.rep[t] = r;
        s.ss0[t] = ss0; s.ss1[t] = r >= 0 ? ss1 : ss0;
        s.state[t] = state;
    }
    if (t == 0) s.next = s.neq = s.next_es = 0;
    if (!__syncthreads_or(state == 1)) {   // no bead of the block steps
        if (MODE == 1 && state == 0) {
            d.pos[cur ^ 1][i0 + t] = d.pos[cur][i0 + t];
            if (MIX || qa) {
                d.spl[cur ^ 1][2 * (size_t)(i0 + t)] = d.spl[cur][2 * (size_t)(i0 + t)];
                d.spl[cur ^ 1][2 * (size_t)(i0 + t) + 1] = d.spl[cur][2 * (size_t)(i0 + t) + 1];
            }
        }
        return true;
    }
    int T = 0;
#pragma unroll
    for (int k = 0; k < FB / 32; ++k) T += s.ws[k];
    if (t < FB) {
        int base = 0;
        for (int k = 0; k < (t >> 5); ++k) base += s.ws[k];
        s.off[t] = base + scan - cnt;
        if (t == FB - 1) s.off[FB] = T;
        s.per[t] = r >= 0 ? d.rep[r].per_any : 0;
    }
    __syncthreads();
    if (qa) {
        // the beads' contact slots (at most QA_REF_CAP, held QA_REF_CAP / LPB
        // per thread of the bead) in ascending order, by rank
        const int b = t / LPB, ln = t % LPB;
        const unsigned qm = ((1u << LPB) - 1u) << (lane & ~(LPB - 1));
        const int nref = s.off[b + 1] - s.off[b] - s.ng[b] - s.nl[b];
        constexpr int HOLD = QA_REF_CAP / LPB;
        int v[HOLD], rk[HOLD];
#pragma unroll
        for (int u = 0; u < HOLD; ++u) {
            const int k = u * LPB + ln;
            v[u] = k < nref ? d.qa.ref[(size_t)k * N + i0 + b] : INT_MAX;
            rk[u] = 0;
        }
        for (int m = 0; m < nref; ++m) {
            int x = 0;
#pragma unroll
            for (int u = 0; u < HOLD; ++u) {
                const int w = __shfl_sync(qm, v[u], m % LPB, LPB);
                if (m / LPB == u) x = w;
            }
#pragma unroll
            for (int u = 0; u < HOLD; ++u) rk[u] += x < v[u];
        }
#pragma unroll
        for (int u = 0; u < HOLD; ++u)
            if (u * LPB + ln < nref) s_q[b][rk[u]] = v[u];
        __syncthreads();
    }

    Ener<MODE> en;
    en.start(s.rep[0]);
    const V3<FT> z{FT(0), FT(0), FT(0)};
    if (t < 2 * FB) {
        // ---- B: bonds, cross products; noise
        if (t < FB) {
            const int k = t;
            if constexpr (MIX) {
                auto bond = [&](int a) {
                    return V3<FF>{ff_diff(F2{s.p[0][a], s.p[3][a]}, F2{s.p[0][a + 1], s.p[3][a + 1]}),
                                  ff_diff(F2{s.p[1][a], s.p[4][a]}, F2{s.p[1][a + 1], s.p[4][a + 1]}),
                                  ff_diff(F2{s.p[2][a], s.p[5][a]}, F2{s.p[2][a + 1], s.p[5][a + 1]})};
                };
                const V3<FF> e = bond(k);
                s.g[MEH][k] = e.x.h; s.g[MEH + 1][k] = e.y.h; s.g[MEH + 2][k] = e.z.h;
                s.g[MEL][k] = e.x.l; s.g[MEL + 1][k] = e.y.l; s.g[MEL + 2][k] = e.z.l;
                const V3<float> ef{e.x.h, e.y.h, e.z.h};
                const float len = norm(ef);
                s.g[MLEN][k] = len;
                s.g[MRN][k] = 1.0f / len;
                if (k > 0) {
                    const V3<FF> x = ff_cross(bond(k - 1), e);
                    s.g[MXH][k] = x.x.h; s.g[MXH + 1][k] = x.y.h; s.g[MXH + 2][k] = x.z.h;
                    s.g[MXL][k] = x.x.l; s.g[MXL + 1][k] = x.y.l; s.g[MXL + 2][k] = x.z.l;
                    const V3<float> xf{x.x.h, x.y.h, x.z.h};
                    const float lx = norm(xf);
                    s.g[MLX][k] = lx;
                    s.g[MRX][k] = 1.0f / lx;
                }
            } else {
                auto bond = [&](int a) {
                    return V3<DN>{DN(s.p[0][a + 1]) - DN(s.p[0][a]), DN(s.p[1][a + 1]) - DN(s.p[1][a]),
                                  DN(s.p[2][a + 1]) - DN(s.p[2][a])};
                };
                const V3<DN> e = bond(k);
                const DN len = norm(e);
                s.g[GE][k] = e.x.v; s.g[GE + 1][k] = e.y.v; s.g[GE + 2][k] = e.z.v;
                s.g[GLEN][k] = len.v;
                s.g[GRN][k] = (DN(1.0) / len).v;
                if (k > 0) {
                    const V3<DN> x = cross(bond(k - 1), e);
                    const DN rx = ninv(x);
                    s.g[GRX][k] = rx.v;
                    s.g[GU][k] = (rx * x.x).v; s.g[GU + 1][k] = (rx * x.y).v; s.g[GU + 2][k] = (rx * x.z).v;
                }
            }
        }
        if (draws) {
            // four draws per bead (normal_x2 then normal, lang_pc.cpp:15-16)
            FT a, b, g;
            if constexpr (MIX) noise3m(st0, &a, &b, &g);
            else noise3_turns(st0, d.logt, &a, &b, &g);
            s.n[0][bn] = a; s.n[1][bn] = b; s.n[2][bn] = g;
            const int rb = s.rep[bn];
            s.rng[bn] = rb >= 0 ? gf2_apply_nib(d.jump + JUMP_WORDS * rb, st0) : 0;
        }
        // the geometry is read by the warps of this part only
        if constexpr (LPB >= 4) asm volatile("bar.sync 1, %0;" ::"n"(2 * FB) : "memory");
        else __syncthreads();

        // ---- D: bonded centres
        const int sp = sc + 1;
        const bool own = MODE == 0 && c >= i0 && c < i0 + FBT && c < N;
        const int rc = own ? s.rep[c - i0] : 0;
        if (sc < NC && (LPB == 1 || t < FB)) {
            V3<FT> ft = z, a1 = z, a2 = z, a3 = z;
            bond_angle<FT, MODE, FB>(d, p, s.g, sp, fl, cp, own, rc, en, &ft, &a1, &a2, &a3);
            s.c[0][sc] = ft.x; s.c[1][sc] = ft.y; s.c[2][sc] = ft.z;
            s.c[3][sc] = a1.x; s.c[4][sc] = a1.y; s.c[5][sc] = a1.z;
            s.c[6][sc] = a2.x; s.c[7][sc] = a2.y; s.c[8][sc] = a2.z;
            s.c[9][sc] = a3.x; s.c[10][sc] = a3.y; s.c[11][sc] = a3.z;
        }
        if (sc < NC && (LPB == 1 || t >= FB)) {
            V3<FT> q[4] = {z, z, z, z};
            dihedral_chiral<FT, MODE, FB>(d, p, s.g, c, sp, fl, cp, own, rc, en, q);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                s.c[12 + 3 * k][sc] = q[k].x; s.c[13 + 3 * k][sc] = q[k].y; s.c[14 + 3 * k][sc] = q[k].z;
            }
        }
        if (MODE == 1 && qa && t < FBT && state == 1) {
            // n and h at this step's positions (precompute_nh.cpp:12-20) to
            // FP32 accuracy, for the sift's FP32 decisions (which recompute
            // them in FP64 near a threshold)
            const int i = i0 + t;
            const uint32_t fb = d.bflags[i];
            V3<float> n{0.0f, 0.0f, 0.0f}, h{0.0f, 0.0f, 0.0f};
            if ((fb & BF_PREV) && (fb & BF_NEXT)) {
                const int s1 = t + 2, s2 = t + 3;    // bonds to the bead and from it
                float dv[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    if constexpr (MIX) {
                        const FF x1{s.g[MEH + a][s1], s.g[MEL + a][s1]}, x2{s.g[MEH + a][s2], s.g[MEL + a][s2]};
                        dv[a] = ff_sub(x2, x1).h;
                    } else {
                        dv[a] = narrow_f(__dsub_rn(s.g[GE + a][s2], s.g[GE + a][s1]));
                    }
                }
                n = unit_f(V3<float>{dv[0], dv[1], dv[2]});
                if constexpr (MIX) {
                    h = -unit_f(V3<float>{s.g[MXH][s2], s.g[MXH + 1][s2], s.g[MXH + 2][s2]});
                } else {
                    h = V3<float>{-narrow_f(s.g[GU][s2]), -narrow_f(s.g[GU + 1][s2]), -narrow_f(s.g[GU + 2][s2])};
                }
            }
            d.qa.nh[2 * (size_t)i] = make_float4(n.x, n.y, n.z, 0.0f);
            d.qa.nh[2 * (size_t)i + 1] = make_float4(h.x, h.y, h.z, 0.0f);
        }
    }

    // ---- E: pair entries, FCAP at a time; between the passes every (axis,
    // bead) thread adds its bead's forces.  A warp fetches the index data of
    // its next 32 entries before it computes the last ones.
    double err0[TT], sum0[TT], sd[TT];
    ST acc[TT];
    for (int p0 = 0;; p0 += FCAP) {
        const int pe = min(T - p0, FCAP);
        auto grab = [&]() {
            int at = 0;
            if (lane == 0) at = atomicAdd(&s.next, 32);
            return __shfl_sync(FULL, at, 0) + lane;
        };
        int at = grab();
        PairRef<FT> ref = pair_fetch<FT, FB>(d, p, s, s_q, i0, p0 + at, at < pe);
        if (MODE == 1 && p0 == 0) {
            // what the integrator does before the force is known:
            // lang_pc_step::operator(), lang_pc.cpp:11-37, mass = 1
            // (main.cpp:156), is linear in the force, so corrector and
            // predictor (the Taylor shift by repeated addition) are applied to
            // y1..y5 alone here, beside the other warps' work, and the force
            // and noise enter with one multiply-add per order at the end.  The
            // position is rounded where the reference rounds it, once by the
            // corrector and once by the predictor: a rounding more at its
            // scale grows to 5e-8 A in 50 steps from a stiff extended start.
#pragma unroll
            for (int u = 0; u < TT; ++u) {
                err0[u] = sum0[u] = sd[u] = 0.0;
                const int w = t - W0 + u * NT, b = w % FBT;
                if (w < 0 || w >= 3 * FBT) continue;
                if (s.rep[b] >= 0) sd[u] = d.rep[s.rep[b]].noise_sd;
                double(&q)[6] = y[u];
                const double err = __fma_rn(__dmul_rn(p.gamma_factor, __dmul_rn(q[1], p.dt_inv)), p.dt2_half, q[2]);
                err0[u] = err;
                q[1] = __fma_rn(-(251.0 / 360.0), err, q[1]);
                q[2] = __dsub_rn(q[2], err);
                q[3] = __fma_rn(-(11.0 / 18.0), err, q[3]);
                q[4] = __fma_rn(-(1.0 / 6.0), err, q[4]);
                q[5] = __fma_rn(-(1.0 / 60.0), err, q[5]);
#pragma unroll
                for (int m = 0; m < 5; ++m) {
#pragma unroll
                    for (int k = 4; k >= (m ? m : 1); --k) q[k] = __dadd_rn(q[k], q[k + 1]);
                    if (m == 0) sum0[u] = q[1];
                }
            }
        }
        while (at - lane < pe) {
            const PairPos<FT> x = pair_pos<FT>(d, cur, ref.j);
            const int nx = grab();
            const PairRef<FT> nref = pair_fetch<FT, FB>(d, p, s, s_q, i0, p0 + nx, nx < pe);
            FT es = FT(0);
            int kind = PE_DONE;
            if (at < pe) {
                V3<FT> f, two;
                kind = pair_entry<FT, MODE, FB>(d, p, s, i0, ref, x, en, &f, &two, &es);
                s.f[0][at] = f.x; s.f[1][at] = f.y; s.f[2][at] = f.z;
                if (MIX && kind == PE_TWO) { s.f2[0][at] = two.x; s.f2[1][at] = two.y; s.f2[2][at] = two.z; }
            }
            if constexpr (MIX) {
                const unsigned m = __ballot_sync(FULL, kind == PE_TWO);
                if (lane == 0) s.two[at >> 5] = m;
            } else if constexpr (MODE == 1) {
                const unsigned m = __ballot_sync(FULL, kind == PE_ES);
                int to = 0;
                if (lane == 0 && m) to = atomicAdd(&s.neq, __popc(m));
                to = __shfl_sync(FULL, to, 0) + __popc(m & ((1u << lane) - 1u));
                if (kind == PE_ES) {
                    s.eq[to] = at;
                    s.ew[to] = es;
                }
            }
            at = nx;
            ref = nref;
        }
        if constexpr (!MIX && MODE == 1) {
            // the electrostatic entries set aside
            __syncthreads();
            const int ne = s.neq;
            for (;;) {
                int k0 = 0;
                if (lane == 0) k0 = atomicAdd(&s.next_es, 32);
                k0 = __shfl_sync(FULL, k0, 0);
                if (k0 >= ne) break;
                if (k0 + lane < ne) {
                    const int k = s.eq[k0 + lane];
                    const V3<FT> r12{s.f[0][k], s.f[1][k], s.f[2][k]};
                    const double s2 = fdot(r12, r12), rn = rsqrt(s2);
                    double V_;
                    const V3<double> f = fscl<double>(mul_(es_factor(p, s.ew[k0 + lane], mul_(s2, rn), rn, &V_), rn), r12);
                    s.f[0][k] = f.x; s.f[1][k] = f.y; s.f[2][k] = f.z;
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < TT; ++u) {
            const int w = t - W0 + u * NT, a = w / FBT, b = w - a * FBT;
            if (w < 0 || w >= 3 * FBT) continue;
            if (p0 == 0) {
                const int k = b + 2;   // centre slot of the bead
                const FT v[9] = {s.c[a][k], -s.c[a][k - 1], s.c[9 + a][k - 1], s.c[6 + a][k], s.c[3 + a][k + 1],
                                 s.c[12 + a][k + 1], s.c[15 + a][k], s.c[18 + a][k - 1], s.c[21 + a][k - 2]};
                acc[u] = ST{};
                if constexpr (MIX) {
                    // FP32 contributions are summed in FP32 and enter once
                    float x = v[0];
#pragma unroll
                    for (int q = 1; q < 9; ++q) x = __fadd_rn(x, v[q]);
                    sum_acc(acc[u], x);
                } else {
#pragma unroll
                    for (int q = 0; q < 9; ++q) sum_acc(acc[u], v[q]);
                }
            }
            const int e0 = max(s.off[b] - p0, 0), e1 = min(s.off[b + 1] - p0, FCAP);
            bool two = false;
            if constexpr (MIX) {
                for (int q = e0 & ~31; q < e1; q += 32) {
                    unsigned m = s.two[q >> 5];
                    if (q < e0) m &= ~0u << (e0 - q);
                    if (q + 32 > e1) m &= ~0u >> (q + 32 - e1);
                    two |= m != 0u;
                }
            }
            if (!two) {
                for (int q = e0; q < e1; ++q) sum_acc(acc[u], s.f[a][q]);
            } else if constexpr (MIX) {
                for (int q = e0; q < e1; ++q) {
                    sum_acc(acc[u], s.f[a][q]);
                    if ((s.two[q >> 5] >> (q & 31)) & 1u) sum_acc(acc[u], s.f2[a][q]);
                }
            }
        }
        if (p0 + FCAP >= T) break;
        __syncthreads();
        if (t == 0) s.next = s.neq = s.next_es = 0;
        __syncthreads();
    }

    // the rest of the bead's force: native disulfides, AFM pulls and walls
    // (k_ext), pseudo-improper dihedral bundles (k_pid: the bead's own side
    // and its chain neighbours' parts for it)
    double F[TT];
#pragma unroll
    for (int u = 0; u < TT; ++u) {
        const int w = t - W0 + u * NT, a = w / FBT, b = w - a * FBT, i = i0 + b;
        F[u] = 0.0;
        if (w < 0 || w >= 3 * FBT || s.state[b] != 1) continue;
        for (int k = s.ss0[b]; k < s.ss1[b]; ++k) {
            if (!d.ss_on[k]) continue;
            const int j = d.ss_j[k], rb = s.rep[b];
            V3<FT> r12;
            if constexpr (MIX) {
                F2 pa[3], pb[3];
                spl_load(d.spl[cur], i, pa);
                spl_load(d.spl[cur], j, pb);
                r12 = pair_vec(d.rep[rb], s.per[b] != 0, pa, pb);
            } else {
                r12 = r_uv_p<double>(d.rep[rb].box, s.per[b] != 0, d.pos[cur][i], d.pos[cur][j]);
            }
            FT V_;
            const V3<FT> f = ss_pair<FT>(p, r12, &V_);
            sum_acc(acc[u], a == 0 ? f.x : (a == 1 ? f.y : f.z));
            if (MODE == 0 && i < j && a == 0) en.add(d, rb, XMD_TERM_NAT_SS, (double)V_);
        }
        F[u] = sum_total(acc[u]);
        if (p.ext_on) F[u] += d.fext[3 * (size_t)i + a];
        if (p.on[XMD_TERM_PID]) {
            const double *pf = d.pid_f;
            const uint32_t fb = d.bflags[i];
            double g = pf[3 * (size_t)i + a];
            if (fb & BF_PREV) g += pf[6 * Ns + 3 * (size_t)(i - 1) + a];   // next-bead part of i - 1
            if (fb & BF_NEXT) g += pf[3 * Ns + 3 * (size_t)(i + 1) + a];   // previous-bead part of i + 1
            F[u] += g;
        }
        if constexpr (MODE == 0) d.F[3 * (size_t)i + a] = F[u];
        // a non-finite force: the replica is frozen from the next step on (its
        // skin check sets steps_left = 0); this bead keeps its state, so no
        // non-finite position ever reaches a list build
        if (!finite_bits(F[u])) {
            atomicOr(d.status, ST_NONFINITE);
            if (MODE == 1) s.state[b] = 2;
        }
    }
    if constexpr (MODE == 0) {
        en.flush(d);
    } else {
        // ---- F: force and noise into the history.  K[k], k > 0: the
        // corrector's factors c_m (lang_pc.cpp:24-29) after the predictor's
        // shift, sum of binomial(m, k) c_m over m >= k; K[0]: their sum over
        // m >= 1, for the predictor's change of the position
        constexpr double c0 = 3.0 / 16.0, c1 = 251.0 / 360.0, c2 = 1.0;
        constexpr double c3 = 11.0 / 18.0, c4 = 1.0 / 6.0, c5 = 1.0 / 60.0;
        constexpr double K[6] = {c1 + c2 + c3 + c4 + c5, c1 + 2.0 * c2 + 3.0 * c3 + 4.0 * c4 + 5.0 * c5,
                                 c2 + 3.0 * c3 + 6.0 * c4 + 10.0 * c5, c3 + 4.0 * c4 + 10.0 * c5, c4 + 5.0 * c5, c5};
        __syncthreads();
#pragma unroll
        for (int u = 0; u < TT; ++u) {
            const int w = t - W0 + u * NT, a = w / FBT, b = w - a * FBT, i = i0 + b;
            if (w < 0 || w >= 3 * FBT || s.state[b] != 1) continue;
            double nz;
            if constexpr (MIX) nz = widen_f(s.n[a][b]);
            else nz = s.n[a][b];
            double(&q)[6] = y[u];
            const double fh = __dmul_rn(__fma_rn(sd[u], nz, F[u]), p.dt2_half);
            q[0] = __dadd_rn(__fma_rn(-c0, __dsub_rn(err0[u], fh), q[0]), __fma_rn(K[0], fh, sum0[u]));
#pragma unroll
            for (int k = 1; k < 6; ++k) q[k] = __fma_rn(K[k], fh, q[k]);
#pragma unroll
            for (int k = 0; k < 5; ++k) d.yh[(size_t)(k * 3 + a) * Ns + i] = q[k + 1];
            s.F[a][b] = q[0];
            // skin test: norm(box->r_uv(r_, orig_r_)), verify.cpp:12-14, squared;
            // the check takes one square root of the maximum (sqrt is monotone
            // and correctly rounded, so that equals the max of the norms).
            // Open axes wrap by exactly zero.  The mixed path takes the
            // displacement from split positions and squares it in FP32.
            if constexpr (MIX) {
                const RepDev &rp = d.rep[s.rep[b]];
                s.e[a][b] = mi_axis(split_d(o[u]), split_d(q[0]), rp.Lh[a], rp.Ll[a], rp.Li[a], s.per[b] != 0);
            } else {
                double e = __dsub_rn(o[u], q[0]);
                if (s.per[b]) {
                    const BoxD &bx = d.rep[s.rep[b]].box;
                    e = __dsub_rn(e, __dmul_rn(bx.cell[a], rint(__dmul_rn(e, bx.cell_inv[a]))));
                }
                s.e[a][b] = __dmul_rn(e, e);
            }
        }
        __syncthreads();

        // ---- G: new positions, generator, skin-test displacement
        if (t < FB) {
            const int i = i0 + t, st = s.state[t];
            double disp = 0.0;
            if (st == 0 || st == 2) {
                // the replica has taken its steps, or the bead keeps its state
                if (st == 2) d.rep[r].fault = 1;
                d.pos[cur ^ 1][i] = d.pos[cur][i];
                if (MIX || qa) {
                    d.spl[cur ^ 1][2 * (size_t)i] = d.spl[cur][2 * (size_t)i];
                    d.spl[cur ^ 1][2 * (size_t)i + 1] = d.spl[cur][2 * (size_t)i + 1];
                }
            } else if (st == 1) {
                const FT q = s.p[MIX ? 6 : 3][t + 3];
                double4_32a pn = make_double4_32a(s.F[0][t], s.F[1][t], s.F[2][t], 0.0);
                if (MIX || qa) {   // (the sift reads them too)
                    const P2 x = split_p(pn);
                    d.spl[cur ^ 1][2 * (size_t)i] = make_float4(x.x.h, x.y.h, x.z.h, MIX ? (float)q : narrow_f((double)q));
                    d.spl[cur ^ 1][2 * (size_t)i + 1] = make_float4(x.x.l, x.y.l, x.z.l, 0.0f);
                }
                if constexpr (MIX) {
                    pn.w = widen_f(q);
                    disp = widen_f(nsq(V3<float>{s.e[0][t], s.e[1][t], s.e[2][t]}));
                } else {
                    pn.w = q;
                    disp = __dadd_rn(__dadd_rn(s.e[0][t], s.e[1][t]), s.e[2][t]);
                }
                d.pos[cur ^ 1][i] = pn;
                d.rng[i] = s.rng[t];
            }
            // one atomic per warp where its beads are of one replica
            const unsigned act = __ballot_sync(FULL, st == 1);
            if (act) {
                const int r0 = __shfl_sync(FULL, r, __ffs(act) - 1);
                const unsigned long long db = (unsigned long long)__double_as_longlong(disp);
                if (__all_sync(FULL, st != 1 || r == r0)) {
                    const unsigned long long m = warp_max_bits(db);
                    if (lane == 0) atomicMax(&d.rep[r0].maxdisp, m);
                } else if (st == 1) {
                    atomicMax(&d.rep[r].maxdisp, db);
                }
            }
        }
    }
    return true;
}

}  // namespace xmdg
