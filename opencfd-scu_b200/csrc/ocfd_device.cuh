// ocfd_device.cuh -- device-side arithmetic of the RHS path (sm_100a, FP64).
//
// Point formulas restate the reference scheme kernels: the split, the sensor
// and the eigen-rows in the reference's expression order, the reconstructions
// and the viscous differences in differences of their points with the
// multiply-adds spelled out (fewer operations, less cancellation; they agree
// with the reference's sums to rounding).  References are to the OpenCFD-SCU
// tree.
#pragma once
#include <cstdint>

#define OCFD_LAP 4

namespace ocfd {

// per-direction constants of a uniform grid (see k_dirconst)
struct DirConst {
    double A[3];       // metric row of the direction (Akx Aky Akz for x, ...)
    double ss;         // |A|
    double An[3];      // A / |A|
    double n[3], l[3], m[3];   // characteristic basis of a face
};

// ---------------------------------------------------------------------------
// kernel parameter block (passed by value to every kernel)
// ---------------------------------------------------------------------------
struct Params {
    int nx, ny, nz;
    int pitch;              // x stride of LAP-box fields, elements
    long long ys, zs;       // y / z strides of LAP-box fields
    long long lapN;         // elements per LAP-box field
    long long N;            // interior cells
    double hx, hy, hz;
    double Ama, Gamma, epsl_sw, Cv, Tsb, amu_C0, tmp0, split_C1, split_C3, vis_c, dt, p00;
    double tv_lim, tv_max;
    double dp1, dp2;
    int scheme_invis, scheme_vis, charteric;
    int nochar_comp_flag;   // flag of components 1-4, non-characteristic hybrid (0 = face flag)
    int periodic[3];
    // whether the local z faces k = 0 / k = nz-1 are faces of the whole grid
    // (1 on one GPU; with the grid split in z, only on the first / last slab)
    int zface_lo, zface_hi;
    // faces of each direction: boundary closures where DIF_BOUND is 1
    // (OCFD_bound, src/OCFD_bound_Scheme.cu:436-469) and the NON_REFLETION
    // value (OCFD_bound_non_ref, :352-433); has_bnd: any of them is set
    int bnd_lo[3], bnd_hi[3];
    int nonref_lo[3], nonref_hi[3];
    int has_bnd;
    // state
    double *prim[5];        // d u v w T on the LAP box
    // precision form (mixed = 1): the primitives the stencils read, the stage
    // RHS and the viscous fluxes in FP32; the conserved state, the RK
    // update and cons->prim stay FP64 (null when the form is off)
    int mixed;
    float *prim32[5];
    float *du32;
    float *ev32;
    const double *met[13];  // Axx Ayy Azz Akx Aky Akz Aix Aiy Aiz Asx Asy Asz Ajac (LAP box)
    double *f, *fn, *du;    // [5][nz][ny][nx]
    double *ev;             // [12] LAP-box fields: Ev1..4 of x, then y, then z
    int8_t *flag[3];        // hybrid scheme flags (nx+1)ny nz, nx(ny+1)nz, nx ny(nz+1)
    // uniform grids: every metric field is one value; kernels read mc[] instead
    int uniform_metrics;
    double mc[13];
    DirConst dc[3];
    double inv_h[3], inv_Ama;   // reciprocals for div_const
    double d0_h[3], d0_ih[3];   // divisor of the viscous scheme's difference (60 h or 840 h) and its reciprocal
    int sweep_impl;         // 4: the walks chosen per direction (default); 5: every face through the in-loop dispatch; 6: the in-line walk
    // viscous kernels of whole steps: 0 inputs staged in shared memory in the
    // precision form on a million cells or more without closed faces, read
    // through L1/L2 elsewhere (vis_staged); 1 read through L1/L2; 2 staged
    int vis_impl;
    // cells whose du the call-free sweep leaves to the fix-up kernel, per
    // direction (interior cell indices; capacity N each), and their counts
    unsigned *defer[3];
    unsigned *defer_count;
    unsigned *flag_count;          // faces per direction whose hybrid flag is not 1 (sensor), or null
    // set to 1 by a kernel whose wait on a staged copy ran out (the host
    // reports it as an error at the next synchronisation)
    int *kerr;
    // shock filter (null when no filter is set): U after the stage-3 update
    // before the face re-projection (5 LAP-box fields) and the pressure
    // cons_to_pri leaves after the last stage (1 LAP-box field)
    double *flap;
    double *pfil;
    // precision form: the filter's pressure in FP32 (1 LAP-box field; the
    // filter's weights are formed from it, its U update stays FP64)
    float *pfil32;
    // boundary-condition family (IBC; 0 none, 108 compression corner): the
    // inflow profile [4][ny] (d,u,v,T), wall blowing shapes fx [nx], gz [nz],
    // first x of the upper inflow row, wall treatment (0 none, 1 TW > 0,
    // 2 TW <= 0), wall temperature and blowing amplitude
    int ibc;
    const double *bc_ub1, *bc_fx, *bc_gz;
    int bc_xbegin, bc_wall_mode;
    double bc_tw, bc_epsl;
};

// host transport of the z split (ocfd_b200_slab_transport in the C ABI):
// op 0 swaps the packed ghost planes with the neighbour ranks, op 1 sums a
// buffer over the ranks in place; type 0 FP64, 1 uint64, 2 uint32, 3 FP32
typedef int (*SlabTransport)(void *user, int op, void *send, void *recv, size_t count, int type);

enum { M_AXX = 0, M_AYY, M_AZZ, M_AKX, M_AKY, M_AKZ, M_AIX, M_AIY, M_AIZ,
       M_ASX, M_ASY, M_ASZ, M_AJAC };

// Bounds-checked build (make bounds: -DOCFD_BOUNDS, libocfd_b200_bounds.so).
// The index helpers and the walks' global accesses check their indexes; one
// outside its array sets error word 3 and is replaced by 0, so that the
// access stays inside the allocation and the call that ran the kernel
// reports the error.  The default build compiles the checks away.
#ifdef OCFD_BOUNDS
// the first failed check also leaves, after the error word, the source line
// of the check and the offending value (an index, or packed coordinates)
__device__ __forceinline__ bool bounds_ok(const Params &p, bool ok, int line, long long value) {
    if (!ok && p.kerr && atomicCAS(p.kerr, 0, 3) == 0) {
        p.kerr[1] = line;
        p.kerr[2] = (int)(value & 0xffffffffLL);
        p.kerr[3] = (int)(value >> 32);
    }
    return ok;
}
__device__ __forceinline__ long long bounds_idx(const Params &p, long long q, long long n, int line) {
    return bounds_ok(p, q >= 0 && q < n, line, q) ? q : 0;
}
#define OCFD_IDX(p, q, n) ::ocfd::bounds_idx((p), (q), (n), __LINE__)
#else
#define OCFD_IDX(p, q, n) (q)
#endif

__device__ __forceinline__ long long lap_index(const Params &p, int i, int j, int k) {
    // i,j,k are LAP-box coordinates (0 .. n+2*LAP-1)
#ifdef OCFD_BOUNDS
    if (!bounds_ok(p, i >= 0 && j >= 0 && k >= 0 && i < p.nx + 2 * OCFD_LAP && j < p.ny + 2 * OCFD_LAP &&
                          k < p.nz + 2 * OCFD_LAP, __LINE__,
                   (long long)(i & 0xfffff) | (long long)(j & 0xfffff) << 20 | (long long)(k & 0xfffff) << 40))
        return 0;
#endif
    return (long long)i + p.ys * j + p.zs * k;
}
// metric m at LAP offset o; UNI selects the constant of a uniform grid (the
// same value every cell would hold, so the arithmetic is unchanged)
template <bool UNI>
__device__ __forceinline__ double metric(const Params &p, int m, long long o) {
    if (UNI) return p.mc[m];
    return p.met[m][OCFD_IDX(p, o, p.lapN)];
}

__device__ __forceinline__ long long in_index(const Params &p, int i, int j, int k) {
#ifdef OCFD_BOUNDS
    if (!bounds_ok(p, i >= 0 && j >= 0 && k >= 0 && i < p.nx && j < p.ny && k < p.nz, __LINE__,
                   (long long)(i & 0xfffff) | (long long)(j & 0xfffff) << 20 | (long long)(k & 0xfffff) << 40))
        return 0;
#endif
    return (long long)i + (long long)p.nx * ((long long)j + (long long)p.ny * k);
}
// entries of direction d's hybrid flag array ((n_d + 1) along d)
__device__ __forceinline__ long long flag_entries(const Params &p, int d) {
    return (long long)(p.nx + (d == 0)) * (p.ny + (d == 1)) * (p.nz + (d == 2));
}
// entry q of direction d's flag array from a pointer fl into it (checked in
// the bounds build, where an entry outside the array reads as flag 2)
__device__ __forceinline__ int flag_at(const Params &p, int d, const int8_t *fl, long long q) {
#ifdef OCFD_BOUNDS
    const long long a = (long long)(fl - p.flag[d]) + q;
    if (!bounds_ok(p, a >= 0 && a < flag_entries(p, d), __LINE__, a)) return 2;
#endif
    return (int)fl[q];
}

// x / c for a run-time constant c with inv = RN(1/c): the product plus one
// FMA residual correction (Markstein) returns the correctly rounded quotient
// except in rare last-ulp cases, at 3 FP64 operations instead of a full
// IEEE division sequence.
__device__ __forceinline__ double div_const(double x, double c, double inv) {
    double q = x * inv;
    double r = fma(-q, c, x);
    return fma(r, inv, q);
}

// ---------------------------------------------------------------------------
// Steger-Warming splitting of one point, src/OCFD_split.cu:92-142
// ---------------------------------------------------------------------------
__device__ __forceinline__ void sw_split(double tmp0, double u, double v, double w, double cc,
                                         double A1, double A2, double A3, double G, double eps,
                                         double split_C1, double split_C3,
                                         double *fp, double *fm) {
    double ss = sqrt(A1 * A1 + A2 * A2 + A3 * A3);
    double E1 = A1 * u + A2 * v + A3 * w;
    double E2 = E1 - cc * ss;
    double E3 = E1 + cc * ss;
    ss = 1.0 / ss;
    A1 *= ss; A2 *= ss; A3 *= ss;
    double E1P = (E1 + sqrt(E1 * E1 + eps * eps)) * 0.50;
    double E2P = (E2 + sqrt(E2 * E2 + eps * eps)) * 0.50;
    double E3P = (E3 + sqrt(E3 * E3 + eps * eps)) * 0.50;
    double E1M = E1 - E1P, E2M = E2 - E2P, E3M = E3 - E3P;
    double uc1 = u - cc * A1, uc2 = u + cc * A1;
    double vc1 = v - cc * A2, vc2 = v + cc * A2;
    double wc1 = w - cc * A3, wc2 = w + cc * A3;
    double vvc1 = (uc1 * uc1 + vc1 * vc1 + wc1 * wc1) * 0.50;
    double vvc2 = (uc2 * uc2 + vc2 * vc2 + wc2 * wc2) * 0.50;
    double vv = (G - 1.0) * (u * u + v * v + w * w);
    double W2 = split_C3 * cc * cc;
    fp[0] = tmp0 * (split_C1 * E1P + E2P + E3P);
    fp[1] = tmp0 * (split_C1 * E1P * u + E2P * uc1 + E3P * uc2);
    fp[2] = tmp0 * (split_C1 * E1P * v + E2P * vc1 + E3P * vc2);
    fp[3] = tmp0 * (split_C1 * E1P * w + E2P * wc1 + E3P * wc2);
    fp[4] = tmp0 * (E1P * vv + E2P * vvc1 + E3P * vvc2 + W2 * (E2P + E3P));
    fm[0] = tmp0 * (split_C1 * E1M + E2M + E3M);
    fm[1] = tmp0 * (split_C1 * E1M * u + E2M * uc1 + E3M * uc2);
    fm[2] = tmp0 * (split_C1 * E1M * v + E2M * vc1 + E3M * vc2);
    fm[3] = tmp0 * (split_C1 * E1M * w + E2M * wc1 + E3M * wc2);
    fm[4] = tmp0 * (E1M * vv + E2M * vvc1 + E3M * vvc2 + W2 * (E2M + E3M));
}

// ---------------------------------------------------------------------------
// reconstruction point formulas.  Stencil convention for a face F+1/2:
// s[t] = f(F-3+t), t = 0..7, for both signs.
// ---------------------------------------------------------------------------

// Differences of a stencil in upwind order (P: v[t] = f(F-3+t); M:
// f(F+4-t)): 6 first differences d[2], d[3] beside the face's cell, second
// differences e[i] = v[i+2] - 2 v[i+1] + v[i] (i = 1 .. 3) and third ones
// f[i] = e[i+1] - e[i].  The derivatives and candidates of the four-point
// stencils are two or three multiply-adds of these, where each takes four of
// the points, and cancel less.
template <typename R> struct Diff7 {
    R d2, d3, e1, e2, e3, f0, f1, f2, f3;
    __device__ __forceinline__ explicit Diff7(const R *v) {
        const R d0 = v[1] - v[0], d1 = v[2] - v[1], d4 = v[5] - v[4], d5 = v[6] - v[5];
        d2 = v[3] - v[2]; d3 = v[4] - v[3];
        const R e0 = d1 - d0, e4 = d5 - d4;
        e1 = d2 - d1; e2 = d3 - d2; e3 = d4 - d3;
        f0 = e1 - e0; f1 = e2 - e1; f2 = e3 - e2; f3 = e4 - e3;
        d2 = (R)6.0 * d2; d3 = (R)6.0 * d3;
    }
    // six times the stencils' first derivatives at the face's cell, a sixth
    // of their second ones as the smoothness indicators take them, and
    // candidate - 12 v[3]
    __device__ __forceinline__ R t0() const { return fma((R)2.0, f0, fma((R)3.0, e1, d2)); }
    __device__ __forceinline__ R t1() const { return fma((R)3.0, e2, d2) - f1; }
    __device__ __forceinline__ R t2() const { return fma((R)-3.0, e2, d3) - f2; }
    __device__ __forceinline__ R t3() const { return fma((R)2.0, f3, fma((R)-3.0, e3, d3)); }
    __device__ __forceinline__ R g0() const { return e1 + f0; }
    __device__ __forceinline__ R g3() const { return e3 - f3; }
    __device__ __forceinline__ R c0() const { return fma((R)3.0, f0, fma((R)4.0, e1, d2)); }
    __device__ __forceinline__ R c1() const { return fma((R)4.0, e2, d2) - f1; }
    __device__ __forceinline__ R c2() const { return fma((R)-2.0, e2, d3) - f2; }
    __device__ __forceinline__ R c3() const { return fma((R)-2.0, e3, d3) + f3; }
};

// WENO7 of a stencil in upwind order (uses v[0..6]), src/OCFD_Schemes.cu:616-741:
// smoothness 960 t^2 + 1040 (6 g)^2 + 1043 (6 f)^2 + 80 t (6 f) plus its
// epsilon.  Bound by FP64 issue; in differences about 100 FP64 operations a
// value where the reference's point sums take 150 (64^3 Taylor-Green, five
// steps: 2.59 -> 2.32 ms; ramp 512x128x64, two steps: 30.2 -> 28.3 ms).
__device__ __forceinline__ double weno7_core(const double *v) {
    const Diff7<double> q(v);
    auto beta = [](double t, double g, double f) {
        return fma(t, fma(960.0, t, 480.0 * f), fma(37440.0 * g, g, fma(37548.0 * f, f, 3.456e-4)));
    };
    double b0 = beta(q.t0(), q.g0(), q.f0), b1 = beta(q.t1(), q.e2, q.f1);
    double b2 = beta(q.t2(), q.e3, q.f2), b3 = beta(q.t3(), q.g3(), q.f3);
    b0 *= b0; b1 *= b1; b2 *= b2; b3 *= b3;
    const double b01 = b0 * b1, b23 = b2 * b3;
    const double a0 = b1 * b23, a1 = 12.0 * b0 * b23, a2 = 18.0 * b3 * b01, a3 = 4.0 * b2 * b01;
    const double r = fma(a0, q.c0(), fma(a1, q.c1(), fma(a2, q.c2(), a3 * q.c3())));
    return v[3] + r / (12.0 * ((a0 + a1) + (a2 + a3)));
}
__device__ __forceinline__ double weno7_p(const double *s) { return weno7_core(s); }
__device__ __forceinline__ double weno7_m(const double *s8) {
    const double v[7] = { s8[7], s8[6], s8[5], s8[4], s8[3], s8[2], s8[1] };
    return weno7_core(v);
}

// WENO5 of a stencil in upwind order (v[1..5]; P: src/OCFD_Schemes.cu:1118-1151,
// M: :1176-1208) over the candidates of mask (bit 0: v[3..5], 1: v[2..4], 2:
// v[1..3]); the boundary closures take fewer than all (src/OCFD_bound_Scheme.cu:554-745).
// Differences as in Diff7, candidates as their distance from v[3].  FP32
// forms the weights as one quotient each, where the common denominator could overflow.
template <typename R>
__device__ __forceinline__ R weno5_core(const R *v, int mask = 7) {
    const R d1 = v[2] - v[1], d2 = v[3] - v[2], d3 = v[4] - v[3], d4 = v[5] - v[4];
    const R e1 = d2 - d1, e2 = d3 - d2, e3 = d4 - d3;
    auto beta = [](R g, R t) { return fma((R)13.0 * g, g, fma((R)3.0 * t, t, (R)(12.0 * 1e-6))); };
    R b0 = beta(e3, fma((R)-2.0, d3, e3)), b1 = beta(e2, d2 + d3), b2 = beta(e1, fma((R)2.0, d2, e1));
    // (a candidate left out takes no part in the common denominator)
    b0 = mask & 1 ? b0 * b0 : (R)1.0; b1 = mask & 2 ? b1 * b1 : (R)1.0; b2 = mask & 4 ? b2 * b2 : (R)1.0;
    const R k0 = mask & 1 ? (R)3.0 : (R)0.0, k1 = mask & 2 ? (R)6.0 : (R)0.0, k2 = mask & 4 ? (R)1.0 : (R)0.0;
    R a0, a1, a2;
    if constexpr (sizeof(R) == 8) {
        a0 = k0 * b1 * b2; a1 = k1 * b0 * b2; a2 = k2 * b0 * b1;
    } else {
        a0 = k0 / b0; a1 = k1 / b1; a2 = k2 / b2;
    }
    // (nor in the sum: beside a closed face its points are ghosts, whose values must not reach the face)
    const R q0 = mask & 1 ? fma((R)3.0, d3, -e3) : (R)0.0, q1 = mask & 2 ? fma((R)2.0, d3, d2) : (R)0.0;
    const R q2 = mask & 4 ? fma((R)2.0, e1, (R)3.0 * d2) : (R)0.0;
    return v[3] + fma(a0, q0, fma(a1, q1, a2 * q2)) / ((R)6.0 * (a0 + a1 + a2));
}
__device__ __forceinline__ double weno5_p(const double *s) { return weno5_core(s); }
__device__ __forceinline__ double weno5_m(const double *s8) {
    const double v[6] = { s8[7], s8[6], s8[5], s8[4], s8[3], s8[2] };
    return weno5_core(v);
}

// sign / minmod, src/OCFD_Schemes.cu:766-797 (minmod4 keeps the fmin of the
// signed arguments as the reference writes it)
__device__ __forceinline__ double sgn1(double x2) { return x2 >= 0 ? 1.0 : -1.0; }
__device__ __forceinline__ double minmod2(double x1, double x2) {
    return 0.5*(sgn1(x1) + sgn1(x2))*fmin(fabs(x1), fabs(x2));
}
__device__ __forceinline__ double minmod4(double x1, double x2, double x3, double x4) {
    double m = 0.5*(sgn1(x1) + sgn1(x2));
    m = m*fabs(0.5*(sgn1(x1) + sgn1(x3)));
    m = m*fabs(0.5*(sgn1(x1) + sgn1(x4)));
    double t = fmin(fmin(x1, x2), fmin(x3, x4));
    return m*t;
}

// NND2 of a stencil in upwind order, src/OCFD_Schemes.cu:800-837
__device__ __forceinline__ double nnd2_up(const double *v) {
    return v[3] + 0.5*minmod2(v[4] - v[3], v[3] - v[2]);
}
__device__ __forceinline__ double nnd2_p(const double *s8) { return nnd2_up(s8); }
__device__ __forceinline__ double nnd2_m(const double *s8) {
    const double v[5] = { 0.0, 0.0, s8[5], s8[4], s8[3] };
    return nnd2_up(v);
}

__device__ __forceinline__ void omp6_mn(int flag, double &m, double &n) {
    if (flag == 1) { m = 0.001; n = 0.0; }
    else if (flag == 2) { m = 0.0; n = -1.0/140.0; }
    else { m = 0.015; n = 0.0; }
}

// OMP6, src/OCFD_Schemes.cu:972-1095: coefficients of the linear flux (times 60) ...
struct Omp6 {
    double c[8];
    __device__ __forceinline__ explicit Omp6(int flag) {
        double m, n;
        omp6_mn(flag, m, n);
        const double mid = 0.5*(m + n);
        m = 0.5*(m - n);
        c[0] = -60.0*m;
        c[1] = 1.0 + 360.0*m + 60.0*mid;
        c[2] = -8.0 - 900.0*m - 360.0*mid;
        c[3] = 37.0 + 1200.0*m + 900.0*mid;
        c[4] = 37.0 - 900.0*m - 1200.0*mid;
        c[5] = -8.0 + 360.0*m + 900.0*mid;
        c[6] = 1.0 - 60.0*m - 360.0*mid;
        c[7] = 60.0*mid;
    }
};
// ... and the limited value of a stencil in upwind order.  The negative side
// (S = 1) takes its large-curvature bound from the downwind difference and
// the point behind the cell in its lower bound.
template <int S>
__device__ __forceinline__ double omp6_up(const Omp6 &k, const double *v) {
    double f = k.c[7]*v[7] + k.c[6]*v[6] + k.c[5]*v[5] + k.c[4]*v[4] + k.c[3]*v[3] + k.c[2]*v[2] + k.c[1]*v[1] + k.c[0]*v[0];
    f = div_const(f, 60.0, 1.0 / 60.0);
    const double mp = v[3] + minmod2(v[4] - v[3], v[3] - v[2]);
    if ((f - v[3])*(f - mp) >= 1.e-10) {
        const double c0 = v[2] + v[4] - 2.0*v[3], c1 = v[3] + v[5] - 2.0*v[4], cm = v[1] + v[3] - 2.0*v[2];
        const double md = 0.5*(v[3] + v[4]) - 0.5*minmod4(4.0*c0 - c1, 4.0*c1 - c0, c1, c0);
        const double lc = v[3] + 0.5*(S ? v[3] - v[4] : v[3] - v[2])
                        + div_const(4.0*minmod4(4.0*cm - c0, 4.0*c0 - cm, c0, cm), 3.0, 1.0 / 3.0);
        const double ul = v[3] + 4.0*(v[3] - v[2]);
        const double lo = fmax(fmin(fmin(S ? v[2] : v[3], v[4]), md), fmin(fmin(v[3], ul), lc));
        const double hi = fmin(fmax(v[4], fmax(v[3], md)), fmax(fmax(v[3], ul), lc));
        f = f + minmod2(hi - f, lo - f);
    }
    return f;
}
__device__ __forceinline__ double omp6_p(int flag, const double *s) { return omp6_up<0>(Omp6(flag), s); }
__device__ __forceinline__ double omp6_m(int flag, const double *s8) {
    const double v[8] = { s8[7], s8[6], s8[5], s8[4], s8[3], s8[2], s8[1], s8[0] };
    return omp6_up<1>(Omp6(flag), v);
}

// WENO7-SYMBO weights and reconstruction, shared by both signs once the
// stencil is mirrored; src/OCFD_Schemes.cu:391-478 (P) and :506-590 (M).
// v[t] is the stencil in upwind order (P: f(F-3+t); M: f(F+4-t)).
__device__ __forceinline__ double symbo_core(bool linear, const double *v) {
    // (stencils 0 .. 3 are WENO7's; the fifth, v[4..7], in the same differences)
    const Diff7<double> q(v);
    const double d4 = v[5] - v[4], d5 = v[6] - v[5], e4 = d5 - d4, f4 = (v[7] - v[6]) - d5 - e4;
    double a0, a1, a2, a3, a4;
    if (linear) {
        a0 = 0.0401954833730; a1 = 0.2493800006710; a2 = 0.4802686256260;
        a3 = 0.2009775476730; a4 = 0.0291783426580;
    } else {
        auto beta = [](double t, double g, double f) {
            return fma(720.0 * t, t, fma(28080.0 * g, g, 28116.0 * f * f));
        };
        const double S0 = beta(q.t0(), q.g0(), q.f0), S1 = beta(q.t1(), q.e2, q.f1);
        const double S2 = beta(q.t2(), q.e3, q.f2), S3 = beta(q.t3(), q.g3(), q.f3);
        double S4 = beta(fma(11.0, f4, fma(-9.0, e4, 6.0 * d4)), fma(-2.0, f4, e4), f4);
        S4 = fmax(fmax(fmax(S0, S1), fmax(S2, S3)), S4);
        const double e = 2.592e-6;
        const double b0 = e + S0, b1 = e + S1, b2 = e + S2, b3 = e + S3, b4 = e + S4;
        const double b01 = b0 * b1, b23 = b2 * b3, b014 = b01 * b4, b234 = b23 * b4;
        a0 = 0.0401954833730 * b1 * b234;
        a1 = 0.2493800006710 * b0 * b234;
        a2 = 0.4802686256260 * b3 * b014;
        a3 = 0.2009775476730 * b2 * b014;
        a4 = 0.0291783426580 * b01 * b23;
    }
    const double am = ((a0 + a1) + (a2 + a3)) + a4;
    // candidate 4: 12 v[4] - 6 d4 + 4 e4 - 3 f4 = 12 v[3] + 6 d3 - 6 e3 + 4 e4 - 3 f4
    const double c4 = fma(-3.0, f4, fma(4.0, e4, fma(-6.0, q.e3, q.d3)));
    const double r = fma(a0, q.c0(), fma(a1, q.c1(), fma(a2, q.c2(), fma(a3, q.c3(), a4 * c4))));
    return v[3] + r / (12.0 * am);
}

__device__ __forceinline__ double symbo_p(int lmt, double tv_lim, double tv_max, const double *s) {
    double TVmin = 0, TVmax = 1;
    if (lmt == 1) {
        double S0 = fabs(s[1] - s[0]) + fabs(s[2] - s[1]) + fabs(s[3] - s[2]);
        double S1 = fabs(s[2] - s[1]) + fabs(s[3] - s[2]) + fabs(s[4] - s[3]);
        double S2 = fabs(s[3] - s[2]) + fabs(s[4] - s[3]) + fabs(s[5] - s[4]);
        double S3 = fabs(s[4] - s[3]) + fabs(s[5] - s[4]) + fabs(s[6] - s[5]);
        double S4 = fabs(s[5] - s[4]) + fabs(s[6] - s[5]) + fabs(s[7] - s[6]);
        TVmin = fmin(fmin(fmin(S0, S1), fmin(S2, S3)), S4);
        TVmax = fmax(fmax(fmax(S0, S1), fmax(S2, S3)), S4);
    }
    return symbo_core(TVmax < tv_lim*TVmin && TVmax < tv_max, s);
}

__device__ __forceinline__ double symbo_m(int lmt, double tv_lim, double tv_max, const double *s) {
    // mirrored stencil; the reference never sets TVmin on this side, so the
    // linear branch cannot be taken (it only evaluates TVmax)
    double v[8];
#pragma unroll
    for (int t = 0; t < 8; t++) v[t] = s[7 - t];
    double TVmin = 0, TVmax = 1;
    if (lmt == 1) {
        double S0 = fabs(v[0] - v[1]) + fabs(v[1] - v[2]) + fabs(v[2] - v[3]);
        double S1 = fabs(v[1] - v[2]) + fabs(v[2] - v[3]) + fabs(v[3] - v[4]);
        double S2 = fabs(v[2] - v[3]) + fabs(v[3] - v[4]) + fabs(v[4] - v[5]);
        double S3 = fabs(v[3] - v[4]) + fabs(v[4] - v[5]) + fabs(v[5] - v[6]);
        double S4 = fabs(v[4] - v[5]) + fabs(v[5] - v[6]) + fabs(v[6] - v[7]);
        TVmax = fmax(fmax(fmin(S0, S1), fmin(S2, S3)), S4);
    }
    return symbo_core(TVmax < tv_lim*TVmin && TVmax < tv_max, v);
}

// CD6 / CD8 first difference, 60 h or 840 h times the derivative, src/OCFD_Schemes.cu:96-126
// (multiply-adds spelled out, so that every kernel forms the same bits)
__device__ __forceinline__ double cd6(double sm3, double sm2, double sm1, double sp1, double sp2, double sp3) {
    return fma(45.0, sp1 - sm1, fma(-9.0, sp2 - sm2, sp3 - sm3));
}
__device__ __forceinline__ double cd8(double sm4, double sm3, double sm2, double sm1,
                                      double sp1, double sp2, double sp3, double sp4) {
    return fma(672.0, sp1 - sm1, fma(-168.0, sp2 - sm2, fma(32.0, sp3 - sm3, -3.0*(sp4 - sm4))));
}

// ---------------------------------------------------------------------------
// characteristic system at a face, src/OCFD_flux_charteric.cu:321-752
// ---------------------------------------------------------------------------
struct CharPara { double u1, v1, w1, c1, n1, n2, n3, l1, l2, l3, m1, m2, m3, KK; };

__device__ __forceinline__ void char_para(double u1, double v1, double w1, double c1,
                                          double a1, double a2, double a3, double G, CharPara &p) {
    double ss = sqrt(a1*a1 + a2*a2 + a3*a3);
    double n1 = a1/ss, n2 = a2/ss, n3 = a3/ss, l1, l2, l3;
    if (fabs(n3) <= fabs(n2)) {
        ss = sqrt(n1*n1 + n2*n2);
        l1 = -n2/ss; l2 = n1/ss; l3 = 0.0;
    } else {
        ss = sqrt(n1*n1 + n3*n3);
        l1 = -n3/ss; l2 = 0.0; l3 = n1/ss;
    }
    p.u1 = u1; p.v1 = v1; p.w1 = w1; p.c1 = c1;
    p.n1 = n1; p.n2 = n2; p.n3 = n3; p.l1 = l1; p.l2 = l2; p.l3 = l3;
    p.m1 = n2*l3 - n3*l2; p.m2 = n3*l1 - n1*l3; p.m3 = n1*l2 - n2*l1;
    p.KK = (G - 1.0)/(c1*c1);
}

// face eigen-system kept in shared memory as NCP planes of nf faces
constexpr int NCP = 14;
__device__ __forceinline__ void store_para(const CharPara &p, double *b, int i, int nf) {
    b[0 * nf + i] = p.u1; b[1 * nf + i] = p.v1; b[2 * nf + i] = p.w1; b[3 * nf + i] = p.c1;
    b[4 * nf + i] = p.n1; b[5 * nf + i] = p.n2; b[6 * nf + i] = p.n3;
    b[7 * nf + i] = p.l1; b[8 * nf + i] = p.l2; b[9 * nf + i] = p.l3;
    b[10 * nf + i] = p.m1; b[11 * nf + i] = p.m2; b[12 * nf + i] = p.m3; b[13 * nf + i] = p.KK;
}
__device__ __forceinline__ void load_para(CharPara &p, const double *b, int i, int nf) {
    p.u1 = b[0 * nf + i]; p.v1 = b[1 * nf + i]; p.w1 = b[2 * nf + i]; p.c1 = b[3 * nf + i];
    p.n1 = b[4 * nf + i]; p.n2 = b[5 * nf + i]; p.n3 = b[6 * nf + i];
    p.l1 = b[7 * nf + i]; p.l2 = b[8 * nf + i]; p.l3 = b[9 * nf + i];
    p.m1 = b[10 * nf + i]; p.m2 = b[11 * nf + i]; p.m3 = b[12 * nf + i]; p.KK = b[13 * nf + i];
}

// row r of the left eigenvector matrix (flux_charteric_ptoc_kernel :617-676)
__device__ __forceinline__ void char_L_row(const CharPara &p, int r, double S[5]) {
    double X1 = 1.0/(2.0*p.c1);
    double un = p.u1*p.n1 + p.v1*p.n2 + p.w1*p.n3;
    double v2 = (p.u1*p.u1 + p.v1*p.v1 + p.w1*p.w1)*0.5;
    double KK = p.KK;
    switch (r) {
    case 0: S[0] = 1.0 - KK*v2; S[1] = KK*p.u1; S[2] = KK*p.v1; S[3] = KK*p.w1; S[4] = -KK; break;
    case 1: S[0] = -(p.u1*p.l1 + p.v1*p.l2 + p.w1*p.l3); S[1] = p.l1; S[2] = p.l2; S[3] = p.l3; S[4] = 0.0; break;
    case 2: S[0] = -(p.u1*p.m1 + p.v1*p.m2 + p.w1*p.m3);
            S[1] = p.n2*p.l3 - p.n3*p.l2; S[2] = p.n3*p.l1 - p.n1*p.l3; S[3] = p.n1*p.l2 - p.n2*p.l1; S[4] = 0.0; break;
    case 3: S[0] = KK*v2*0.5 + X1*un; S[1] = -X1*p.n1 - KK*p.u1*0.5; S[2] = -X1*p.n2 - KK*p.v1*0.5;
            S[3] = -X1*p.n3 - KK*p.w1*0.5; S[4] = KK*0.5; break;
    default: {
            double s41 = KK*v2*0.5 + X1*un, s42 = -X1*p.n1 - KK*p.u1*0.5;
            double s43 = -X1*p.n2 - KK*p.v1*0.5, s44 = -X1*p.n3 - KK*p.w1*0.5;
            S[0] = s41 - 2*X1*un; S[1] = 2*X1*p.n1 + s42; S[2] = 2*X1*p.n2 + s43;
            S[3] = 2*X1*p.n3 + s44; S[4] = KK*0.5; break; }
    }
}

// row r of the right eigenvector matrix (flux_charteric_ctop_kernel :678-752)
__device__ __forceinline__ void char_R_row(const CharPara &p, int r, double S[5]) {
    switch (r) {
    case 0: S[0] = 1.0; S[1] = 0.0; S[2] = 0.0; S[3] = 1.0; S[4] = 1.0; break;
    case 1: S[0] = p.u1; S[1] = p.l1; S[2] = p.n2*p.l3 - p.n3*p.l2; S[3] = p.u1 - p.c1*p.n1; S[4] = 2*p.u1 - S[3]; break;
    case 2: S[0] = p.v1; S[1] = p.l2; S[2] = p.n3*p.l1 - p.n1*p.l3; S[3] = p.v1 - p.c1*p.n2; S[4] = 2*p.v1 - S[3]; break;
    case 3: S[0] = p.w1; S[1] = p.l3; S[2] = p.n1*p.l2 - p.n2*p.l1; S[3] = p.w1 - p.c1*p.n3; S[4] = 2*p.w1 - S[3]; break;
    default: {
            S[0] = (p.u1*p.u1 + p.v1*p.v1 + p.w1*p.w1)*0.5;
            double H = S[0] + 1.0/p.KK;
            S[1] = p.u1*p.l1 + p.v1*p.l2 + p.w1*p.l3;
            S[2] = p.u1*p.m1 + p.v1*p.m2 + p.w1*p.m3;
            S[3] = H - p.c1*(p.u1*p.n1 + p.v1*p.n2 + p.w1*p.n3);
            S[4] = 2*H - S[3]; break; }
    }
}

__device__ __forceinline__ double dot5(const double S[5], double x0, double x1, double x2, double x3, double x4) {
    return S[0]*x0 + S[1]*x1 + S[2]*x2 + S[3]*x3 + S[4]*x4;
}

}  // namespace ocfd
