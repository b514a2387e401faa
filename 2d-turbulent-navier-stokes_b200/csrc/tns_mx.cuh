// tns_mx.cuh -- FP32 helpers of the mixed-precision kernels (structured and general
// meshes): the FP32 transcendentals and the deviation form of a stage slot.
//
// A stage slot is formed as deviations from a reference state of its tile or chunk
// (TileRefMx, tns_device.cuh): dC = C - Cref, and every quantity the residual and the
// sources difference follows by exact algebra (dU = (dC2 - Uref dC1) / C1,
// d(C2 U) = dC2 U + C2ref dU, P - Pref = R (dC1 T + C1ref dT), |V| - |V|ref =
// (|V|^2 - |V|ref^2) / (|V| + |V|ref), ...), so each FP32 rounding is a fraction of a
// deviation, as when a FP64 value is rounded after the subtraction.
#pragma once

#include "tns_batch.cuh"
#include "tns_device.cuh"

namespace tns {

__device__ __forceinline__ float pow06f(float T) { return __expf(0.6f * __logf(T)); }

// tanh for the FP32 path: the Maclaurin series x - x^3/3 + 2x^5/15 - 17x^7/315 +
// 62x^9/2835 - 1382x^11/155925 + 21844x^13/6081075 for |x| < 1/4 (the first omitted
// term is below 2e-12 relative there), and the identity tanh|x| = 1 - 2/(exp(2|x|)+1)
// above, where its cancellation costs at most ~5e-7 relative.
__device__ __forceinline__ float tanh_f32(float x) {
    const float ax = fabsf(x);
    if (ax < 0.25f) {
        const float x2 = x * x;
        return x * (1.0f + x2 * (-1.0f / 3.0f + x2 * (2.0f / 15.0f + x2 * (-17.0f / 315.0f +
                    x2 * (62.0f / 2835.0f + x2 * (-1382.0f / 155925.0f + x2 * (21844.0f / 6081075.0f)))))));
    }
    const float r = 1.0f - __fdividef(2.0f, __expf(2.0f * ax) + 1.0f);
    return copysignf(r, x);
}

// The FP32 values of one stage slot: flux deviations (F_m - Fref_m, G_m - Gref_m; F_2 = G_1),
// (U - Uref, V - Vref), C5/C1 - ref, |V| - ref, and for the cell itself its T, RHO and
// P - Pref (each rounded once, kept()).
struct SlotMx {
    float f0, g0, f1, f2, g2, f3, g3, f4, g4, du, dv, dri, dqm;
    float3 own;
};

// Slots in shared memory, packed for 16-byte loads.
struct SlotsMx {
    float4* a;  // f0 g0 f1 f2
    float4* b;  // g2 f3 g3 f4
    float4* c;  // g4 du dv dri
    float* q;   // dqm
    __device__ __forceinline__ void put(int s, const SlotMx& o) const {
        a[s] = make_float4(o.f0, o.g0, o.f1, o.f2);
        b[s] = make_float4(o.g2, o.f3, o.g3, o.f4);
        c[s] = make_float4(o.g4, o.du, o.dv, o.dri);
        q[s] = o.dqm;
    }
};

// A cell's slot from its state's deviation dC = C - Cref (d1..d5).
__device__ __forceinline__ void slot_dev_mx(const Params& P, const TileRefMx& R, float d1, float d2, float d3,
                                            float d4, float d5, SlotMx& o) {
    const float rho = R.rho + d1;
    const float rr = 1.0f / rho;
    const float du = (d2 - R.u * d1) * rr;
    const float dv = (d3 - R.v * d1) * rr;
    const float de = (d4 - R.e * d1) * rr;
    const float dri = (d5 - R.ri * d1) * rr;
    const float u = R.u + du, v = R.v + dv;
    const float dq2 = du * (u + R.u) + dv * (v + R.v);  // |V|^2 - |V|ref^2
    const float dt = (de - 0.5f * dq2) * (float)P.inv_cv;
    const float t = R.t + dt;
    const float dp = kept((float)P.rr * (d1 * t + R.rho * dt));
    const float qm = sqrtf(u * u + v * v);
    const float qs = qm + R.qm;
    const float dqm = qs > 0.0f ? dq2 / qs : 0.0f;
    const float f2 = d2 * v + R.c2 * dv;  // d(C2 V) = d(C3 U)
    o.f0 = d2;
    o.g0 = d3;
    o.f1 = d2 * u + R.c2 * du + dp;
    o.f2 = f2;
    o.g2 = d3 * v + R.c3 * dv + dp;
    o.f3 = (d4 + dp) * u + R.c4p * du;
    o.g3 = (d4 + dp) * v + R.c4p * dv;
    o.f4 = d5 * u + R.c5 * du;
    o.g4 = d5 * v + R.c5 * dv;
    o.du = du;
    o.dv = dv;
    o.dri = dri;
    o.dqm = dqm;
    o.own = make_float3(kept(t), kept(rho), kept(dp));
}

// A ghost's slot: its BC state in FP64, then the deviations.
__device__ __forceinline__ void slot_ghost_mx(const TileRefMx& R, const Prim& p, SlotMx& o) {
    const Prim& r = R.q;
    o.f0 = (float)(p.f[0] - r.f[0]);
    o.g0 = (float)(p.g[0] - r.g[0]);
    o.f1 = (float)(p.f[1] - r.f[1]);
    o.f2 = (float)(p.f[2] - r.f[2]);
    o.g2 = (float)(p.g[2] - r.g[2]);
    o.f3 = (float)(p.f[3] - r.f[3]);
    o.g3 = (float)(p.g[3] - r.g[3]);
    o.f4 = (float)(p.f[4] - r.f[4]);
    o.g4 = (float)(p.g[4] - r.g[4]);
    o.du = (float)(p.u - r.u);
    o.dv = (float)(p.v - r.v);
    o.dri = (float)(p.ri - r.ri);
    o.dqm = (float)(p.qm - r.qm);
    o.own = make_float3(kept((float)p.t), kept((float)p.rho), kept((float)(p.p - r.p)));
}

// Static geometry of one cell of the mixed stage, rounded once on the host: the four face
// vectors, the source-gradient coefficients, 1/VOL, VOL, 1/YCC and 1/YCC as V/YCC takes it
// (zero near the axis, where DVY stands in), four 16-byte words; and in FP64, for the parts
// that cancel, the sums of the face vectors and VOL/YCC (axisymmetric only).
struct GeoMx {
    float4 s01, s23, g, w;  // (sx1 sy1 sx2 sy2) (sx3 sy3 sx4 sy4) (GA GB GC GD) (1/VOL VOL 1/YCC vby)
    double sumx, sumy, vr;
};

inline void geo_mx(int iaxis, const double sx[4], const double sy[4], const double grad[4], double vol, double ycc,
                   GeoMx& o) {
    auto f4 = [](double a, double b, double c, double d) {
        return float4{(float)a, (float)b, (float)c, (float)d};
    };
    o.s01 = f4(sx[0], sy[0], sx[1], sy[1]);
    o.s23 = f4(sx[2], sy[2], sx[3], sy[3]);
    o.g = f4(grad[0], grad[1], grad[2], grad[3]);
    o.w = f4(1.0 / vol, vol, 1.0 / ycc, ycc < YAXIS_THRESH ? 0.0 : 1.0 / ycc);
    o.sumx = sx[0] + sx[1] + sx[2] + sx[3];
    o.sumy = sy[0] + sy[1] + sy[2] + sy[3];
    o.vr = iaxis == 1 ? vol * (1.0 / ycc) : 0.0;
}

// Residual, source and update (source_terms.f90:24-104, residual.f90:23-83) of `cell`, whose
// slot is c and whose neighbours' are nb, as an FP32 increment on the FP64 state.  The flux
// residual: the cell's own deviation meets the sum of the face vectors and each neighbour's
// its face vector, in FP32; the reference flux (cancelling over a closed contour) meets the
// sum in FP64.  vis(float[4]) gives the cell's viscous flux (stage 1).
template <class Vis>
__device__ __forceinline__ void stage_cell_mx(const Params& P, const TileRefMx& R, const StageArgsMx& A, size_t ncell,
                                              size_t cell, const SlotsMx& S, int c, const int nb[4], const GeoMx& G,
                                              const float3& own, Vis vis, double dv[5]) {
    float r0 = 0.0f, r1 = 0.0f, r2 = 0.0f, r3 = 0.0f, r4 = 0.0f;
    float4 cn[4];
    auto add = [&](int s, const float4& k, float sx, float sy) {
        const float4 a = S.a[s], b = S.b[s];
        r0 += a.x * sx + a.y * sy;
        r1 += a.z * sx + a.w * sy;
        r2 += a.w * sx + b.x * sy;
        r3 += b.y * sx + b.z * sy;
        r4 += b.w * sx + k.x * sy;
    };
    const float4 cc = S.c[c];
    add(c, cc, (float)G.sumx, (float)G.sumy);
#pragma unroll
    for (int k = 0; k < 4; k++) cn[k] = S.c[nb[k]];
    add(nb[0], cn[0], G.s01.x, G.s01.y);
    add(nb[1], cn[1], G.s01.z, G.s01.w);
    add(nb[2], cn[2], G.s23.x, G.s23.y);
    add(nb[3], cn[3], G.s23.z, G.s23.w);
    const Prim& rq = R.q;
    double R64[5];
#pragma unroll
    for (int m = 0; m < 5; m++) R64[m] = rq.f[m] * G.sumx + rq.g[m] * G.sumy;

    float src3 = 0.0f, src5;
    {
        const float ga = G.g.x, gb = G.g.y, gc = G.g.z, gd = G.g.w;
        const float dqac = S.q[nb[0]] - S.q[nb[2]], dqbd = S.q[nb[1]] - S.q[nb[3]];
        const float drac = cn[0].w - cn[2].w, drbd = cn[1].w - cn[3].w;
        const float duac = cn[0].y - cn[2].y, dubd = cn[1].y - cn[3].y;
        const float dvac = cn[0].z - cn[2].z, dvbd = cn[1].z - cn[3].z;
        const float DQX = dqac * ga + dqbd * gb, DQY = dqac * gc + dqbd * gd;
        const float DRX = drac * ga + drbd * gb, DRY = drac * gc + drbd * gd;
        const float DUX = duac * ga + dubd * gb, DUY = duac * gc + dubd * gd;
        const float DVX = dvac * ga + dvbd * gb, DVY = dvac * gc + dvbd * gd;
        const float RHO = own.y, RI = R.ri + cc.w, T = own.x;
        const float AMU = (float)P.suth_amol * pow06f(T);
        const float CHI = RHO * RI / ((float)CMU * AMU);
        const float chi2 = CHI * CHI;
        const float FMU = tanh_f32((float)ALPHA_T * chi2) / tanh_f32((float)BETA_T * chi2);
        const float FR2 = tanh_f32(sqrtf(CHI)) / tanh_f32(CHI * (float)P.fr2k);
        const float AMUT = FMU * RHO * RI;
        const float PHI = DQX * DRX + DQY * DRY;
        const float DEE = PHI > 0.0f ? DRX * DRX + DRY * DRY : 0.0f;
        float pw = AMUT / fmaxf(AMUT, (float)AMU_THRESH * AMU);
        {
            float r = 1.0f, bb = pw;
            int mm = P.npseudo < 0 ? -P.npseudo : P.npseudo;
            while (mm) {
                if (mm & 1) r *= bb;
                mm >>= 1;
                if (mm) bb *= bb;
            }
            pw = P.npseudo < 0 ? 1.0f / r : r;
        }
        // (VBYY is 0 on a plane mesh)
        const float VBYY = P.iaxis != 1 ? 0.0f : G.w.w == 0.0f ? DVY : (R.v + cc.z) * G.w.w;
        const float DIVVEL = DUX + DVY + VBYY;
        const float trace = (float)P.div23 * DIVVEL, sxy = DUY + DVX;
        const float PK = FMU * RI * (2.0f * (DUX * DUX + DVY * DVY + VBYY * VBYY) + sxy * sxy - trace * DIVVEL);
        src5 = RHO * (((float)CONST1 - (float)CONST2 * FR2) * sqrtf(RI * fmaxf(PK, 0.0f)) - (float)CONST3 * DEE) * pw;
        if (P.iaxis == 1) {
            // SOURCE3 = (P - TTT)/YCC: the reference pressure's part cancels the reference
            // flux in FP64
            R64[2] -= rq.p * G.vr;
            src3 = (own.z - (AMU + AMUT) * (VBYY + VBYY - trace)) * G.w.z;
        }
    }

    // update (residual.f90:67-83); the frozen terms VIS + D are one array after stage 1
    float e[5];
    e[0] = A.d[cell];
    if (A.e) {
#pragma unroll
        for (int m = 1; m < 5; m++) e[m] = A.e[(m - 1) * ncell + cell];
    } else {
        float v[4];
        vis(v);
#pragma unroll
        for (int m = 1; m < 5; m++) e[m] = v[m - 1] + A.d[m * ncell + cell];
#pragma unroll
        for (int m = 1; m < 5; m++) A.eout[(m - 1) * ncell + cell] = e[m];
    }
    const float DT = P.local ? A.dt[cell] : (float)*A.dtmin;
    const float dtv = -A.alpha * (DT * G.w.x);
    float inc[5];
    inc[0] = dtv * (0.5f * r0 + (float)R64[0] - e[0]);
    inc[1] = dtv * (0.5f * r1 + (float)R64[1] - e[1]);
    inc[2] = dtv * (0.5f * r2 - G.w.y * src3 + (float)R64[2] - e[2]);
    inc[3] = dtv * (0.5f * r3 + (float)R64[3] - e[3]);
    inc[4] = dtv * (float)CFLTURB * (0.5f * r4 - G.w.y * src5 + (float)R64[4] - e[4]);
    double Co[5], Cn[5];
#pragma unroll
    for (int m = 0; m < 5; m++) {
        Co[m] = A.cold[m * ncell + cell];
        Cn[m] = Co[m] + (double)inc[m];
    }
    // nu~ floor C5 = C1*max(RTOL, C5/C1), applied only where it binds
    if (Cn[4] < P.rtol * Cn[0]) {
        Cn[4] = P.rtol * Cn[0];
        inc[4] = (float)(Cn[4] - Co[4]);
    }
    if (A.qout) {
#pragma unroll
        for (int m = 0; m < 5; m++) A.qout[m * ncell + cell] = Cn[m];
    } else {
#pragma unroll
        for (int m = 0; m < 5; m++) A.dqout[m * ncell + cell] = inc[m];
    }
    if (A.status) {
        bool bad = false;
#pragma unroll
        for (int m = 0; m < 5; m++) bad |= !isfinite(Cn[m]);
        if (bad) atomicOr(A.status, 1u);
    }
#pragma unroll
    for (int m = 0; m < 5; m++) dv[m] = fabs(Co[m] - Cn[m]);
}

// max |COLD - C| per component (the residual monitor): warp max, then one atomic per warp on
// the ordered bit pattern.
__device__ __forceinline__ void stage_cdiff_mx(const StageArgsMx& A, const double dv[5]) {
#pragma unroll
    for (int m = 0; m < 5; m++) {
        double v = dv[m];
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        if ((threadIdx.x & 31) == 0) atomicMax(&A.cdiff[m], (unsigned long long)__double_as_longlong(v));
    }
}

}  // namespace tns
