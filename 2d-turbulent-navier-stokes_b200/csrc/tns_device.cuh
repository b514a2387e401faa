// tns_device.cuh -- device-side constants, parameter block, mesh view and the per-cell
// physics of the RK4 / JST / viscous / source / boundary hot path.
//
// The arithmetic restates the reference solver's Fortran (paths relative to the
// reference project) in its operation order, except where one reciprocal replaces a
// run of divisions by the same value, T**0.6 is computed by a division-free Newton
// refinement, and stored gradient coefficients fold a division by a static determinant
// (each a few ulp).  The memory layout is new: cells live in a structured (i, j) block
// (j fastest), ghosts in four side arrays; face vectors come from the node coordinates
// in each tile, the static gradient coefficients and volumes from per-mesh arrays.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

// Host-and-device helpers: the discrete adjoint calls the same arithmetic from its
// point functions, which also compile for the host.
#define TNS_HD __host__ __device__ __forceinline__

namespace tns {

// constants.f90:15-60
constexpr double CMU = 0.09;
constexpr double ALPHA_T = 0.00052;
constexpr double BETA_T = 0.2;
constexpr double CONST1 = 21.479;
constexpr double CONST2 = 21.394;
constexpr double CONST3 = 1.5;
constexpr double C02 = 0.25;
constexpr double C04 = 0.00390625;
constexpr double CFLTURB = 0.5;
constexpr double HALF = 0.5;
constexpr double QUARTER = 0.25;
constexpr double YAXIS_THRESH = 0.001;
constexpr double AMU_THRESH = 0.001;
constexpr double GTH = 35.0;
constexpr double CONVKSC = 1.0 / 98066.5;
constexpr double RK_ALPHA[4] = {0.25, 1.0 / 3.0, 0.5, 1.0};  // constants.f90:30-33

// Scalar inputs plus every constant the Fortran folds left to right (computed once on
// the host with the same operation order, so device values equal the reference's).
struct Params {
    double gama, amol, cfl, prandtl, prandtlt, p0, t0, pamb, rtred, rinit;
    double tflame, ancomb, acomb, rhoprop, pinf, aminf, deltabl;
    int local, npseudo, iaxis, pad_;
    double rr, cv, cp, s0, tinf, rtol;  // turbnstwod.f90:37-42, RTOLERANCE
    double gamrr;                        // GAMA*RR
    double suth_amol;                    // SUTH_COEF*DSQRT(AMOL)
    double div23;                        // 2/3
    double fr2k;                         // DSQRT(2*DSQRT(CMU))
    double inv1mg;                       // 1/(1-GAMA)
    double gth08;                        // GTH**0.8
    double rtol_rtred;                   // RTOLERANCE*RTRED
    double bl_u;                         // 2*AMINF*DSQRT(GAMA*RR*TINF)
    double bl_exp;                       // 1/7
    double inv_cv;                       // 1/CV
    double cp_pr, cp_prt;                // CP/PRANDTL, CP/PRANDTLT
    double inv_cmu_suth;                 // 1/(CMU*SUTH_COEF*DSQRT(AMOL))
    double inv_cp, inv_t0;               // 1/CP, 1/T0
    double rho0, inv_gm1;                // P0/(RR*T0), 1/(GAMA-1)
};

// Static per-face geometry of the viscous flux (viscous.f90:130-217), stored per tile
// (tns_tile.cuh), each face in the orientation of the cell that evaluates it (an i-face
// between cells (i-1, j) and (i, j) in that of (i-1, j) as its face 2, or of (0, j) as its
// face 4; a j-face between (i, j-1) and (i, j) in that of (i, j-1) as its face 3, or of
// (i, 0) as its face 1):
//   FG_SX, FG_SY  face vector; FG_GA..FG_GD diamond-gradient coefficients (A = the cell,
//   C = the neighbour, B, D = the face's nodes: dF/dx = (F_A - F_C) GA + (F_B - F_D) GB,
//   dF/dy = (F_A - F_C) GC + (F_B - F_D) GD); FG_RYAVG 1/YAVG of the axisymmetric v/y
//   term, or 0 where YAVG is below the axis threshold (then dv/dy).
enum FaceGeo { FG_SX, FG_SY, FG_GA, FG_GB, FG_GC, FG_GD, FG_RYAVG, FG_N };

// Ghost-side numbering: side 1 (j=-1) and 3 (j=NJ) are indexed by i, sides 2 (i=NI)
// and 4 (i=-1) by j; the four runs are stored back to back.
struct TileRefMx;

// Static geometry of one ghost: its parent's face vector on the ghost's side, the mirrored
// centroid's y and the parent's.
struct alignas(16) GhostRec {
    double psx, psy, ycg, ycp;
};

struct Mesh {
    int ni, nj;             // cells in i and j
    const double* x;        // node x [(ni+1)*(nj+1)], node (i,j) at i*(nj+1)+j
    const double* y;
    const double* cfldl;    // CFL*DL per cell
    const int* gtype;       // BC type per ghost
    const int* grank;       // bc.in line of each ghost (node-average order)
    const double* gxc;      // mirrored ghost centroids (geometry.f90:114-142)
    const double* gyc;
    const GhostRec* grec;   // static geometry per ghost
    const double* ginj;     // type-6 burn-rate multiplier
    const double* gport;    // type-6 port mass flux of the current stage
    // weights DELY(*YCC) of the port sums per cell (null without such ports): of side 3, along
    // j, and of side 2, along i
    const double *wport, *wport_i;
    const double* cvol;     // VOL per cell (geometry.f90:87,98,101)
    const double* vcfl;     // VOL / (CFL*DL) per cell
    const double* stile;    // static data of the stage tiles, one block per tile (tns_tile.cuh)
    const double* vtile;    // static face geometry of the viscous tiles (tns_tile.cuh)
    // per boundary node (rows b = 0 and b = nj along a, then a = 0 and a = ni along b): the
    // BC types of its two ghosts in bc.in order (bits 0-2, 3-5) and whether that order is the
    // reverse of their ascending position order (bit 6)
    const int* bnode;
    // (mixed precision) each stage tile's reference state for the current iteration,
    // written by the dissipation kernel from Q_old, read by the four stages
    TileRefMx* tref = nullptr;
    __host__ __device__ int ghost_index(int side, int along) const {
        return side == 1 ? along : side == 2 ? ni + along : side == 3 ? ni + nj + along
                                                                      : 2 * ni + nj + along;
    }
    __host__ __device__ int nghosts() const { return 2 * (ni + nj); }
};

TNS_HD double dmax1(double a, double b) { return a >= b ? a : b; }
TNS_HD double dmin1(double a, double b) { return a <= b ? a : b; }

// Fortran REAL**INTEGER by square-and-multiply.
TNS_HD double powi(double x, int n) {
    double r = 1.0, b = x;
    int m = n < 0 ? -n : n;
    while (m) {
        if (m & 1) r *= b;
        m >>= 1;
        if (m) b *= b;
    }
    return n < 0 ? 1.0 / r : r;
}

// 1/x and sqrt(x) by Newton's method on the hardware's reciprocal and reciprocal-square-root
// estimates (rcp.approx.ftz.f64, rsqrt.approx.ftz.f64: 20 bits or more), two quadratic steps
// each, the last one rounding the final sum: within one ulp for normal arguments.  They have no
// slow path (a call with its register and branch cost), which the arguments here -- densities,
// temperatures, squared speeds -- never need.  The kernels are bound by instruction issue and
// dependent FP64 latency: with these, the cubic T**-1/5 step, the shorter expm1 and the skipped
// denominators below, a FP64 iteration of the 1024 x 384 nozzle-plume went 0.180 -> 0.160 ms
// (0.041 -> 0.0375 ms on the 115 x 50 nozzle).  A product with recip() is rounded twice: where it
// becomes part of the state, use quot().  recip(0), recip(inf) and root(inf) are NaN: a state that
// holds them is non-finite either way.  root() takes a subnormal for zero.
TNS_HD double recip(double x) {
#ifdef __CUDA_ARCH__
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    r = fma(r, fma(-x, r, 1.0), r);
    return fma(r, fma(-x, r, 1.0), r);
#else
    return 1.0 / x;
#endif
}
TNS_HD double root(double x) {
#ifdef __CUDA_ARCH__
    double r;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    double g = x * r, h = 0.5 * r;
    const double e = fma(-g, h, 0.5);
    g = fma(g, e, g);
    h = fma(h, e, h);
    g = fma(h, fma(-g, g, x), g);
    return fabs(x) < 2.2250738585072014e-308 ? 0.0 : g;
#else
    return sqrt(x);
#endif
}

// a/b as recip's estimate after its first step (2^-40), the product with it and one correction of
// the quotient (Markstein, IBM J. Res. Dev. 34(1), 1990), which leaves 2^-80 before the last
// rounding: the correctly rounded quotient but for rare cases, in as many operations as a product
// with recip(), which is rounded twice.  For quotients that become part of the state.
TNS_HD double quot(double a, double b) {
#ifdef __CUDA_ARCH__
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    r = fma(r, fma(-b, r, 1.0), r);
    const double q = a * r;
    return fma(fma(-q, b, a), r, q);
#else
    return a / b;
#endif
}

// T**-0.4 and T**-0.6 for T > 0: a single-precision estimate y = exp2(-0.2 log2 T) of
// T**(-1/5) (about 1e-7 relative) and one cubically convergent step for the inverse fifth
// root,
//   t = 1 - T y^5,  y (1 + c),  c = t/5 + 3 t^2/25,
// whose truncation error is below 1e-19; (1 + c)^2 and (1 + c)^3 then correct y^2 (exact: y
// has 24 bits) and y^3 in one rounding each.  The viscosity, T**0.6 = T T**-0.4, and its
// reciprocal thus come from one evaluation without a division (T**0.6 within 1.5 ulp).
struct FifthRoots {
    double m04, m06;
};
TNS_HD FifthRoots fifth_roots(double T) {
#ifdef __CUDA_ARCH__
    const double y = (double)exp2f(-0.2f * __log2f((float)T));
#else
    const double y = (double)exp2f(-0.2f * log2f((float)T));
#endif
    const double y2 = y * y, y3 = y2 * y;
    const double t = fma(-T, y2 * y3, 1.0);
    const double c = t * fma(0.12, t, 0.2);
    return FifthRoots{fma(y2, fma(c, c, 2.0 * c), y2), fma(y3, c * fma(3.0, c, 3.0), y3)};
}

// T**0.6, within a few ulp of pow.
TNS_HD double pow06(double T) { return T * fifth_roots(T).m04; }

// expm1(x) for 0 <= x <= 40 (device; libm on the host), by the classical additive
// argument reduction (Cody & Waite; the structure of Tang's expm1, ACM TOMS 18(2), 1992,
// without its table):
//   x = k ln2 + r, k = rint(x / ln2), |r| <= ln2 / 2, with ln2 = LN2_HI + LN2_LO and
//   LN2_HI carrying 32 significant bits, so k LN2_HI is exact and r has no cancellation
//   error;
//   expm1(r) = r + r^2 q(r), q the degree-9 interpolant of (e^r - 1 - r)/r^2 at the
//   Chebyshev points of [-ln2/2, ln2/2] (error of the whole below 4.1e-17 relative),
//   its even and odd powers summed apart so that the dependent chain is half as long;
//   expm1(x) = 2^k expm1(r) + (2^k - 1) in one fused multiply-add (2^k - 1 is exact
//   for k <= 53, and k <= 58 here).
TNS_HD double expm1_nonneg(double x) {
#ifdef __CUDA_ARCH__
    constexpr double INV_LN2 = 1.4426950408889634;
    constexpr double LN2_HI = 0.6931471804855391;    // ln 2 to 32 significant bits
    constexpr double LN2_LO = 7.440617110012397e-11;  // ln 2 - LN2_HI
    const double k = rint(x * INV_LN2);
    const double r = fma(-k, LN2_LO, fma(-k, LN2_HI, x));
    const double s = r * r;
    double a = 2.7620138719733994e-07, b = 2.5100424157005067e-08;
    a = fma(a, s, 2.480152119021773e-05);
    b = fma(b, s, 2.7557268378684192e-06);
    a = fma(a, s, 0.0013888888917281794);
    b = fma(b, s, 0.00019841269863105968);
    a = fma(a, s, 0.04166666666662399);
    b = fma(b, s, 0.008333333333330051);
    a = fma(a, s, 0.5000000000000001);
    b = fma(b, s, 0.16666666666666669);
    const double p = fma(s, fma(b, r, a), r);
    const double w = __longlong_as_double((long long)((int)k + 1023) << 52);  // 2^k
    return fma(w, p, w - 1.0);
#else
    return expm1(x);
#endif
}

// tanh(a) / tanh(b) for a, b >= 0, from tanh(x) = E / (E + 2) with E = expm1(2x), as
// num / den = Ea (Eb + 2) / (Eb (Ea + 2)).  Arguments are capped at 20, where tanh is 1 to
// double precision, so E stays finite; a denominator's tanh(b) that is 1 (b >= 20: the
// damping of a cell whose eddy viscosity is ten times the molecular one or more) is left
// out, expm1 and all.
struct Ratio {
    double num, den;
};
TNS_HD Ratio tanh_ratio_parts(double a, double b) {
    const double ea = expm1_nonneg(2.0 * fmin(a, 20.0));
    Ratio r{ea, ea + 2.0};
    if (!(b >= 20.0)) {
        const double eb = expm1_nonneg(2.0 * b);
        r.num = ea * (eb + 2.0);
        r.den = eb * (ea + 2.0);
    }
    return r;
}
TNS_HD double tanh_ratio(double a, double b) {
    const Ratio r = tanh_ratio_parts(a, b);
    return r.num * recip(r.den);
}

// The damping ratios of the turbulence model at CHI = RHO nu~ / (CMU AMU):
// FMU = tanh(ALPHA_T CHI^2) / tanh(BETA_T CHI^2) and FR2 = tanh(sqrt CHI) / tanh(FR2K CHI), the
// sources' two by one reciprocal.  The scale, an exact factor of both parts of FR2, keeps the
// product of the denominators, some CHI^3 for small CHI, from underflowing before CHI^2 does.
TNS_HD double damping_fmu(double chi) {
    const double chi2 = chi * chi;
    return tanh_ratio(ALPHA_T * chi2, BETA_T * chi2);
}
struct Damping {
    double fmu, fr2;
};
TNS_HD Damping damping(const Params& P, double chi) {  // (P by reference: FR2K is loaded at its use)
    const double chi2 = chi * chi;
    const Ratio m = tanh_ratio_parts(ALPHA_T * chi2, BETA_T * chi2);
    const Ratio r = tanh_ratio_parts(root(chi), chi * P.fr2k);
    const double num = r.num * 0x1p700, den = r.den * 0x1p700;
    const double inv = recip(m.den * den);
    return Damping{m.num * den * inv, num * m.den * inv};
}

// Sutherland-type molecular viscosity SUTH_COEF*DSQRT(AMOL)*T**0.6 (viscous.f90:188).
TNS_HD double amu_of(const Params& P, double T) {
    return P.suth_amol * pow06(T);
}

// A value made opaque to the optimizer (device code; the identity on the host).  The
// compiler fuses a multiply into a later add (FMA contraction) or not depending on how
// many uses the product has, so a value whose uses differ between kernels (a slot kept in
// a register for the thread's own cell in one, only stored in another) could round
// differently in each.  Passing it through kept() rounds it once, the same way in every
// kernel and build, which keeps the tile-height builds and the batched kernels
// bit-identical to one another.
TNS_HD double kept(double x) {
#ifdef __CUDA_ARCH__
    double r;
    asm("mov.b64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
#else
    return x;
#endif
}
TNS_HD float kept(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("mov.b32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return x;
#endif
}

// Primitive variables and fluxes of one interior cell (turbnstwod.f90:204-227).
struct Prim {
    double u, v, t, p, rho, ri, c5, qm;
    double f[5], g[5];
};

TNS_HD void primitive(const Params& P, double c1, double c2, double c3,
                                          double c4, double c5, Prim& s) {
    const double RHO = c1;
    const double rr = recip(RHO);  // one reciprocal instead of four divisions
    s.rho = RHO;
    s.u = c2 * rr;
    s.v = c3 * rr;
    const double E = c4 * rr;
    s.t = (E - 0.5 * (s.u * s.u + s.v * s.v)) * P.inv_cv;
    s.p = kept(RHO * P.rr * s.t);
    s.f[0] = c2;
    s.f[1] = RHO * s.u * s.u + s.p;
    s.f[2] = RHO * s.u * s.v;
    s.f[3] = (c4 + s.p) * s.u;
    s.g[0] = c3;
    s.g[1] = s.f[2];
    s.g[2] = RHO * s.v * s.v + s.p;
    s.g[3] = (c4 + s.p) * s.v;
    const double RT = c5 * rr;
    s.f[4] = RHO * RT * s.u;
    s.g[4] = RHO * RT * s.v;
    s.ri = RT;
    s.c5 = c5;
    s.qm = root(s.u * s.u + s.v * s.v);
}

// The mixed path's reference state of a stage tile: a FP64 state of the tile (its first
// cell's Q_old), its primitives and fluxes, and the primitives in FP32 that the
// deviation formulas multiply by.  Any state of the tile serves: the kernels only form
// differences from it.
struct TileRefMx {
    double c[5];  // conservative state
    Prim q;       // its primitives and fluxes
    float rho, u, v, e, t, ri, qm, c2, c3, c4p, c5;  // (e = C4/C1, c4p = C4 + P)
    float pad;
};
static_assert(sizeof(TileRefMx) % 8 == 0, "a tile reference is copied as 8-byte words");
constexpr int TREF_WORDS = (int)(sizeof(TileRefMx) / 8);

TNS_HD void make_tile_ref(const Params& P, const double c[5], TileRefMx& R) {
    for (int m = 0; m < 5; m++) R.c[m] = c[m];
    primitive(P, c[0], c[1], c[2], c[3], c[4], R.q);
    R.rho = (float)c[0];
    R.u = (float)R.q.u;
    R.v = (float)R.q.v;
    R.e = (float)(c[3] / c[0]);
    R.t = (float)R.q.t;
    R.ri = (float)R.q.ri;
    R.qm = (float)R.q.qm;
    R.c2 = (float)c[1];
    R.c3 = (float)c[2];
    R.c4p = (float)(c[3] + R.q.p);
    R.c5 = (float)c[4];
    R.pad = 0.0f;
}

// Conservative + flux tail shared by BC types 2,3,4,6,7 (e.g. boundary.f90:62-70).
TNS_HD void ghost_tail(const Params& P, double RHO, Prim& g) {
    g.rho = RHO;
    const double C2 = RHO * g.u;
    const double C3 = RHO * g.v;
    const double E = P.cv * g.t + 0.5 * (g.u * g.u + g.v * g.v);
    const double C4 = RHO * E;
    g.f[0] = C2;
    g.f[1] = RHO * g.u * g.u + g.p;
    g.f[2] = RHO * g.u * g.v;
    g.f[3] = (C4 + g.p) * g.u;
    g.g[0] = C3;
    g.g[1] = g.f[2];
    g.g[2] = RHO * g.v * g.v + g.p;
    g.g[3] = (C4 + g.p) * g.v;
}

// Face surface vector (geometry.f90:77-99) for face k (1..4) of a cell with nodes 1..4.
TNS_HD void face_vector(int iaxis, int k, const double X[4],
                                            const double Y[4], double& sx, double& sy) {
    const int a = k - 1, b = k & 3;  // nodes (k, k+1)
    if (iaxis == 1) {
        sx = (Y[b] - Y[a]) * (Y[a] + Y[b]) * HALF;
        sy = -(X[b] - X[a]) * (Y[a] + Y[b]) * HALF;
    } else {
        sx = (Y[b] - Y[a]);
        sy = -(X[b] - X[a]);
    }
}

// Cell volume (geometry.f90:87,98,101).
TNS_HD double cell_volume(int iaxis, const double X[4], const double Y[4],
                                              double ycc) {
    double v = HALF * ((X[2] - X[0]) * (Y[3] - Y[1]) - (X[3] - X[1]) * (Y[2] - Y[0]));
    if (iaxis == 1) v = v * ycc;
    if (v <= 0.0) v = -v;
    return v;
}

// Density of the type-2 inlet at temperature T, (S0/(RR T))**(1/(1-GAMA)): the isentrope
// through (P0, T0), RHO0 (T/T0)**(1/(GAMA-1)).  With z = 1 - T/T0 = (GAMA-1)/2 M^2 T/T0 small
// (M < 1.29 at GAMA = 1.4), log(1 - z) = -2 atanh(z/(2-z)) by its series to the 19th power
// (the next term is below 4e-18), so the exponent carries no rounding of a large logarithm;
// pow elsewhere.  A third of pow's instructions on the path a boundary tile waits for.
TNS_HD double inlet_density(const Params& P, double T) {
#ifdef __CUDA_ARCH__
    const double z = (P.t0 - T) * P.inv_t0;
    if (z >= 0.0 && z < 0.25) {
        const double w = z * recip(2.0 - z), w2 = w * w;
        double a = 1.0 / 19.0;
        a = fma(a, w2, 1.0 / 17.0);
        a = fma(a, w2, 1.0 / 15.0);
        a = fma(a, w2, 1.0 / 13.0);
        a = fma(a, w2, 1.0 / 11.0);
        a = fma(a, w2, 1.0 / 9.0);
        a = fma(a, w2, 1.0 / 7.0);
        a = fma(a, w2, 0.2);
        a = fma(a, w2, 1.0 / 3.0);
        a = fma(a, w2, 1.0);
        return P.rho0 * exp(-2.0 * P.inv_gm1 * (w * a));
    }
#endif
    return pow(P.s0 / (P.rr * T), P.inv1mg);
}

// DT of one cell (turbnstwod.f90:97-108).  The reverse of a global time step finds the cell
// that DTMIN came from by comparing this value, so no two kernels may round it differently:
// each product that meets a sum does so in a named fused multiply-add, and the compiler has no
// choice left.  (On the host, as a program that divides computes it.)
TNS_HD double local_dt(const Params& P, double c1, double c2, double c3, double c4, double cfldl) {
#ifdef __CUDA_ARCH__
    const double rr = 1.0 / c1;
    const double U = c2 * rr, V = c3 * rr;
    const double q2 = fma(U, U, V * V);
    const double T = fma(c4, rr, -0.5 * q2) * P.inv_cv;
    return cfldl / (sqrt(q2) + sqrt(P.gamrr * T));
#else
    const double U = c2 / c1, V = c3 / c1;
    const double T = (c4 / c1 - 0.5 * (U * U + V * V)) / P.cv;
    return cfldl / (sqrt(U * U + V * V) + sqrt(P.gamrr * T));
#endif
}

// Ghost state from its parent (and the parent's opposite neighbour) for BC types 2..7
// (boundary.f90:53-327; type 6 with the port flux supplied by the caller).
// par: parent cell, opp: parent's neighbour across the face opposite the ghost.
// psx, psy: parent's surface vector on the ghost side; ycc_g, ycc_p: ghost / parent
// centroid y; gport: summed port flux (type 6 only); inj: burn-rate multiplier.
TNS_HD void boundary_ghost(const Params& P, int type, const Prim& par,
                                               const Prim& opp, double psx, double psy,
                                               double ycc_g, double ycc_p, double gport,
                                               double inj, Prim& g) {
    double RHO, AMU, C5;
    switch (type) {
        case 2: {  // subsonic inlet :53-71
            g.u = fabs(par.u);
            g.v = -par.v;
            g.t = P.t0 - 0.5 * (g.u * g.u + g.v * g.v) * P.inv_cp;
            RHO = inlet_density(P, g.t);
            g.p = RHO * P.rr * g.t;
            ghost_tail(P, RHO, g);
            C5 = amu_of(P, g.t);  // RHO * (AMU / RHO)
            g.f[4] = C5 * g.u;
            g.g[4] = C5 * g.v;
            break;
        }
        case 3: {  // farfield / extrapolation :76-95
            g.u = fabs(2.0 * par.u - opp.u);
            g.v = 2.0 * par.v - opp.v;
            g.t = 2.0 * par.t - opp.t;
            g.p = 2.0 * par.p - opp.p;
            if (P.pamb >= 0.0) g.p = P.pamb;
            RHO = g.p * recip(P.rr * g.t);
            ghost_tail(P, RHO, g);
            C5 = par.c5;
            g.f[4] = par.f[4];
            g.g[4] = par.g[4];
            break;
        }
        case 4: {  // symmetry :100-109
            g.u = par.u;
            g.v = -par.v;
            g.t = par.t;
            RHO = par.rho;
            g.p = par.p;
            ghost_tail(P, RHO, g);
            C5 = par.c5;
            g.f[4] = par.f[4];
            g.g[4] = -par.g[4];
            break;
        }
        case 5: {  // no-slip wall / axis :114-122
            g.u = -par.u;
            g.v = -par.v;
            g.t = par.t;
            RHO = par.rho;
            g.p = par.p;
            g.rho = RHO;
            g.f[0] = -par.f[0];
            g.f[1] = 2.0 * par.p - par.f[1];
            g.f[2] = -par.f[2];
            g.f[3] = -par.f[3];
            g.g[0] = -par.g[0];
            g.g[1] = -par.g[1];
            g.g[2] = 2.0 * par.p - par.g[2];
            g.g[3] = -par.g[3];
            C5 = -par.c5;
            g.f[4] = -par.f[4];
            g.g[4] = -par.g[4];
            break;
        }
        case 6: {  // mass injection :128-163
            const double DNR = sqrt(psx * psx + psy * psy);
            const double ENX = -psx / DNR, ENY = -psy / DNR;
            const double DHYD = fabs(ycc_g + ycc_p);
            double GP = (P.iaxis == 1) ? 2.0 * gport / (DHYD * DHYD) : gport / DHYD;
            RHO = par.rho;
            const double RDOT = P.acomb * pow(par.p * CONVKSC, P.ancomb) * inj;
            double RDOTEB = RDOT;
            double VEL = P.rhoprop / RHO * RDOTEB;
            g.p = par.p;
            g.u = VEL * ENX + VEL * ENX - par.u;
            g.v = VEL * ENY + VEL * ENY - par.v;
            g.t = P.tflame - 0.5 * (g.u * g.u + g.v * g.v) * P.inv_cp;
            AMU = amu_of(P, g.t);
            const double GVAL =
                (GP / (P.rhoprop * RDOT)) * pow(P.rhoprop * RDOT * DHYD / AMU, -0.125);
            if (GVAL > GTH) RDOTEB = RDOTEB * (1.0 + 0.023 * (pow(GVAL, 0.8) - P.gth08));
            VEL = P.rhoprop / RHO * RDOTEB;
            g.u = VEL * ENX + VEL * ENX - par.u;
            g.v = VEL * ENY + VEL * ENY - par.v;
            g.t = P.tflame - 0.5 * (g.u * g.u + g.v * g.v) * P.inv_cp;
            RHO = g.p * recip(P.rr * g.t);
            C5 = amu_of(P, g.t);
            ghost_tail(P, RHO, g);
            g.f[4] = C5 * g.u;
            g.g[4] = C5 * g.v;
            break;
        }
        default: {  // 7: boundary-layer inlet :310-327
            g.p = P.pinf;
            g.t = P.tinf;
            g.v = -par.v;
            RHO = g.p * recip(P.rr * g.t);
            if (ycc_g <= P.deltabl)
                g.u = P.bl_u * pow(ycc_g / P.deltabl, P.bl_exp) - par.u;
            else
                g.u = P.bl_u - par.u;
            ghost_tail(P, RHO, g);
            C5 = amu_of(P, g.t);
            g.f[4] = C5 * g.u;
            g.g[4] = C5 * g.v;
            break;
        }
    }
    g.c5 = C5;
    g.ri = C5 * recip(g.rho);
    g.qm = root(g.u * g.u + g.v * g.v);
}

// Turbulence / radial sources of one cell (source_terms.f90:24-104).  Neighbours
// a,b,c,d are NC1..NC4; ga..gd are the cell's stored coefficients of the centroid-
// difference gradient (source_terms.f90:24-60): dF/dx = (F_a - F_c) ga + (F_b - F_d) gb,
// dF/dy = (F_a - F_c) gc + (F_b - F_d) gd, i.e. ga = (y_b - y_d)/DNR, gb = -(y_a - y_c)/DNR,
// gc = -(x_b - x_d)/DNR, gd = (x_a - x_c)/DNR with DNR = (x_a - x_c)(y_b - y_d) -
// (x_b - x_d)(y_a - y_c) over the four neighbour centroids; RYCC is 1/YCC.
struct SrcIn {
    double ga, gb, gc, gd;
    double ua, ub, uc, ud, va, vb, vc, vd, ra, rb, rc, rd, qa, qb, qc, qd;
};

__device__ __forceinline__ void source_terms(const Params& P, const SrcIn& s, double RHO,
                                             double RI, double TI, double PI, double VI,
                                             double YCCI, double RYCC, double& src3,
                                             double& src5) {
    const double dqac = s.qa - s.qc, dqbd = s.qb - s.qd, drac = s.ra - s.rc, drbd = s.rb - s.rd;
    const double duac = s.ua - s.uc, dubd = s.ub - s.ud, dvac = s.va - s.vc, dvbd = s.vb - s.vd;
    const double DQX = dqac * s.ga + dqbd * s.gb, DQY = dqac * s.gc + dqbd * s.gd;
    const double DRX = drac * s.ga + drbd * s.gb, DRY = drac * s.gc + drbd * s.gd;
    const double DUX = duac * s.ga + dubd * s.gb, DUY = duac * s.gc + dubd * s.gd;
    const double DVX = dvac * s.ga + dvbd * s.gb, DVY = dvac * s.gc + dvbd * s.gd;
    // AMU = SUTH T^0.6, CHI = RHO RI / (CMU AMU) with T^-0.6, and both damping ratios by one
    // reciprocal
    const FifthRoots tr = fifth_roots(TI);
    const double AMU = P.suth_amol * (TI * tr.m04);
    const double CHI = RHO * RI * (P.inv_cmu_suth * tr.m06);
    const Damping damp = damping(P, CHI);
    const double FMU = damp.fmu, FR2 = damp.fr2;
    const double AMUT = FMU * RHO * RI;
    const double PHI = DQX * DRX + DQY * DRY;
    double DEE = 0.0;
    if (PHI > 0.0) DEE = DRX * DRX + DRY * DRY;
    double PK;
    const double DIV23 = P.div23;
    // (AMUT / DMAX1(AMUT, AMU_THRESH*AMU))**NPSEUDO: exactly 1 when AMUT is the larger
    const double thr = AMU_THRESH * AMU;
    const double pw = AMUT >= thr ? 1.0 : powi(AMUT / thr, P.npseudo);
    if (P.iaxis == 1) {
        const double VBYY = (YCCI < YAXIS_THRESH) ? DVY : VI * RYCC;
        const double DIVVEL = DUX + DVY + VBYY;
        PK = FMU * RI *  // AMUT / RHO
             (DUX * DUX + DVY * DVY + VBYY * VBYY + DUX * DUX + DVY * DVY + VBYY * VBYY +
              (DUY + DVX) * (DUY + DVX) - DIV23 * DIVVEL * DIVVEL);
        PK = dmax1(PK, 0.0);
        src5 = (RHO * (CONST1 - CONST2 * FR2) * root(RI * PK) - RHO * CONST3 * DEE) * pw;
        const double TTT = (AMU + AMUT) * (VBYY + VBYY - DIV23 * DIVVEL);
        src3 = (PI - TTT) * RYCC;
    } else {
        const double DIVVEL = DUX + DVY;
        PK = FMU * RI *
             (DUX * DUX + DVY * DVY + DUX * DUX + DVY * DVY + (DUY + DVX) * (DUY + DVX) -
              DIV23 * DIVVEL * DIVVEL);
        PK = dmax1(PK, 0.0);
        src5 = (RHO * (CONST1 - CONST2 * FR2) * root(RI * PK) - RHO * CONST3 * DEE) * pw;
        src3 = 0.0;
    }
}

// One face of the thin-layer viscous flux (viscous.f90:130-217): A = the cell, C = the
// face neighbour, B, D = the face's nodes (node averages).  FaceIn holds the coordinates
// (the discrete adjoint's face reverse reads them).
struct FaceIn {
    double sx, sy, xa, ya, xb, yb, xc, yc, xd, yd;
    double ua, va, ta, ub, vb, tb, uc, vc, tc, ud, vd, td;
    double rhoa, rhob, rhoc, rhod, ra, rb, rc, rd;
};

// Sums of one boundary face with the face state (parent + ghost)/2 (U, V averaged; T, P
// of both sides).  mode 0: v = P*SX, P*SY, RHO*(U*SX+V*SY), |S|; mode 1: v[0] = P0*|MDOT|,
// v[1] = |MDOT| with the face's total pressure P0 = P (1 + (GAMA-1)/2 M^2)^(GAMA/(GAMA-1)),
// M^2 = (U^2+V^2)/(GAMA RR T) and mass flux MDOT = RHO (U SX + V SY); RHO is the average of
// P/(RR*T) on both sides.
__device__ __forceinline__ void face_sums(const Params& P, int mode, double u, double vv, double tp, double tg,
                                          double pp, double pg, double sx, double sy, double v[4]) {
    const double pf = 0.5 * (pp + pg);
    const double rho = 0.5 * (pp / (P.rr * tp) + pg / (P.rr * tg));
    if (mode == 1) {
        const double tf = 0.5 * (tp + tg);
        const double m2 = (u * u + vv * vv) / (P.gama * P.rr * tf);
        const double p0 = pf * pow(1.0 + 0.5 * (P.gama - 1.0) * m2, P.gama / (P.gama - 1.0));
        const double md = fabs(rho * (u * sx + vv * sy));
        v[0] = p0 * md;
        v[1] = md;
        return;
    }
    v[0] = pf * sx;
    v[1] = pf * sy;
    v[2] = rho * (u * sx + vv * sy);
    v[3] = sqrt(sx * sx + sy * sy);
}

// One face from its stored geometry (FG_*): the flux of viscous.f90:130-217 with the
// diamond gradient from the coefficients.  Assigns vis[0..3].
struct FaceVals {
    double ua, va, ta, ub, vb, tb, uc, vc, tc, ud, vd, td;
    double rhoa, rhob, rhoc, rhod, ra, rb, rc, rd;
};

__device__ __forceinline__ void viscous_face(const Params& P, const FaceVals& f, double sx,
                                             double sy, double ga, double gb, double gc,
                                             double gd, double ryavg, double vis[4]) {
    const double duac = f.ua - f.uc, dubd = f.ub - f.ud, dvac = f.va - f.vc, dvbd = f.vb - f.vd;
    const double dtac = f.ta - f.tc, dtbd = f.tb - f.td, drac = f.ra - f.rc, drbd = f.rb - f.rd;
    const double DUX = duac * ga + dubd * gb, DUY = duac * gc + dubd * gd;
    const double DVX = dvac * ga + dvbd * gb, DVY = dvac * gc + dvbd * gd;
    const double DTX = dtac * ga + dtbd * gb, DTY = dtac * gc + dtbd * gd;
    const double DRX = drac * ga + drbd * gb, DRY = drac * gc + drbd * gd;
    const double UAVG = QUARTER * (f.ua + f.ub + f.uc + f.ud);
    const double VAVG = QUARTER * (f.va + f.vb + f.vc + f.vd);
    const double TAVG = QUARTER * (f.ta + f.tb + f.tc + f.td);
    const double RHOAVG = QUARTER * (f.rhoa + f.rhob + f.rhoc + f.rhod);
    const double RAVG = QUARTER * (f.ra + f.rb + f.rc + f.rd);
    double DIVVEL;
    if (P.iaxis == 1) {
        const double VBYY = (ryavg == 0.0) ? DVY : VAVG * ryavg;
        DIVVEL = DUX + DVY + VBYY;
    } else {
        DIVVEL = DUX + DVY;
    }
    const FifthRoots tr = fifth_roots(TAVG);
    const double AMU = P.suth_amol * (TAVG * tr.m04);
    const double AK = AMU * P.cp_pr;
    const double CHI = RHOAVG * RAVG * (P.inv_cmu_suth * tr.m06);
    const double FMU = damping_fmu(CHI);
    const double AMUT = RHOAVG * RAVG * FMU;
    const double AKT = AMUT * P.cp_prt;
    const double AMUEFF = AMU + AMUT;
    const double AKEFF = AK + AKT;
    const double TXX = AMUEFF * (DUX + DUX - P.div23 * DIVVEL);
    const double TYY = AMUEFF * (DVY + DVY - P.div23 * DIVVEL);
    const double TXY = AMUEFF * (DUY + DVX);
    const double QXX = UAVG * TXX + VAVG * TXY + AKEFF * DTX;
    const double QYY = UAVG * TXY + VAVG * TYY + AKEFF * DTY;
    vis[0] = TXX * sx + TXY * sy;
    vis[1] = TXY * sx + TYY * sy;
    vis[2] = QXX * sx + QYY * sy;
    vis[3] = AMUEFF * DRX * sx + AMUEFF * DRY * sy;
}

}  // namespace tns
