// tns_diss.cuh -- DT (turbnstwod.f90:97-108) and the frozen JST dissipation D of Q_old
// (solver_state.f90:70-225) on one tile, for the FP64 and the mixed kernels: the states and
// pressures of the tile and two rings of halo, then sensors, Laplacians and VOL/DT of the
// tile and one ring, then each cell's blend over its four faces.
//
// A ghost holds a copy of its parent, so a load clamped to the mesh is the ghost's state, and
// a ghost face's contribution is exactly zero.  What bounds it: shared memory (a cell reads 65
// words) and instruction issue; hence values in pairs for 16-byte accesses, each thread's own
// state kept in registers, one division-free VOL/DT per cell (VOL / CFL*DL is static).  The
// tile with single words, divisions and halo tests took 31 us at 1024 x 384 (FP64), this one
// 25; an iteration 0.132 -> 0.126 ms, mixed 0.135 -> 0.132 ms, 2048 x 768 port 0.534 -> 0.517.
// (A warp marching down a strip with shuffles and no shared memory issued as many
// instructions, its register rotation included, and was slower on all but the largest mesh.)
// R: precision of the sensors, Laplacians, blend and output -- FP64, or FP32 on the mixed
// path, where the state, the pressure and every difference of the state stay FP64.
#pragma once

#include "tns_batch.cuh"
#include "tns_tile.cuh"

namespace tns {

constexpr int DW = TJ + 4;  // halo-2 slot grid (TI+4) x (TJ+4)
constexpr int NDSLOT = (TI + 4) * DW;
constexpr int NDRING = NDSLOT - NTHREADS;  // its halo positions
static_assert(NRING <= NTHREADS, "one position of the inner ring per thread at most");

template <class R>
struct Pair;
template <>
struct Pair<double> { using type = double2; };
template <>
struct Pair<float> { using type = float2; };
__device__ __forceinline__ double2 pair(double a, double b) { return make_double2(a, b); }
__device__ __forceinline__ float2 pair(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double quotient(double a, double b) { return a * recip(b); }
__device__ __forceinline__ float quotient(float a, float b) { return a / b; }

template <class R>
struct DissSmem {
    using R2 = typename Pair<R>::type;
    double2 c01[NDSLOT], c23[NDSLOT], c4p[NDSLOT];  // C1..C5, P
    R2 l01[NSLOT], l23[NSLOT], l4v[NSLOT];          // Laplacians, VOL/DT
    R2 anu[NSLOT];                                  // sensors of equations 1-4 and of 5
};

// Halo position r of the halo-2 grid: its two first and last rows, then the two first and
// last columns between them.
__device__ __forceinline__ void ring2_slot(int r, int& li, int& lj) {
    if (r < 2 * DW) { li = r / DW; lj = r % DW; }
    else if (r < 4 * DW) { li = TI + r / DW; lj = r % DW; }
    else { r -= 4 * DW; li = 2 + (r >> 2); lj = (r & 3) < 2 ? r & 3 : TJ + (r & 3); }
}

// P (turbnstwod.f90:98-104), and |V| + sound speed.
__device__ __forceinline__ double diss_pressure(const Params& P, const double c[5]) {
    const double rr = recip(c[0]);
    const double U = c[1] * rr, V = c[2] * rr;
    return c[0] * P.rr * ((c[3] * rr - 0.5 * (U * U + V * V)) * P.inv_cv);
}
__device__ __forceinline__ double diss_speed(const Params& P, const double c[5], double p) {
    const double rr = recip(c[0]);
    return root(c[1] * c[1] + c[2] * c[2]) * rr + root(P.gama * p * rr);
}

template <class R, class Ref>
__device__ __forceinline__ void dissipation_tile(const Params& P, const Mesh& M, const DissArgs<R>& A, int bx, int by,
                                                 Ref ref) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    DissSmem<R>& S = *reinterpret_cast<DissSmem<R>*>(smem_raw);
    const size_t ncell = (size_t)M.ni * M.nj;
    const int j0 = bx * TJ, i0 = by * TI;
    const int tj = threadIdx.x, ti = threadIdx.y, tid = ti * TJ + tj;
    const int i = i0 + ti, j = j0 + tj;
    auto cell = [&](int ci, int cj) { return (size_t)min(max(ci, 0), M.ni - 1) * M.nj + min(max(cj, 0), M.nj - 1); };
    // VOL/DT: (VOL / CFL*DL) (|V| + c) for the local step, VOL / DTMIN for the global one
    const double* vscale = P.local ? M.vcfl : M.cvol;
    pdl_trigger();
    const size_t own = cell(i, j);
    const double vs = vscale[own];  // static
    int hi = 0, hj = 0;
    if (tid < NDRING) ring2_slot(tid, hi, hj);
    int ri = 0, rj = 0;
    double vr = 0.0;
    if (tid < NRING) {
        ring_slot(tid, ri, rj);
        vr = vscale[cell(i0 - 1 + ri, j0 - 1 + rj)];
    }
    pdl_wait();
    auto load = [&](size_t c, double q[5]) {
#pragma unroll
        for (int m = 0; m < 5; m++) q[m] = A.q[m * ncell + c];
    };
    auto put = [&](int s, const double q[5], double p) {
        S.c01[s] = make_double2(q[0], q[1]);
        S.c23[s] = make_double2(q[2], q[3]);
        S.c4p[s] = make_double2(q[4], p);
    };
    double q[5], p;
    {
        double h[5];
        load(own, q);
        if (tid < NDRING) load(cell(i0 - 2 + hi, j0 - 2 + hj), h);
        p = diss_pressure(P, q);
        put((ti + 2) * DW + tj + 2, q, p);
        if (tid < NDRING) put(hi * DW + hj, h, diss_pressure(P, h));
#pragma unroll 1
        for (int r = tid + NTHREADS; r < NDRING; r += NTHREADS) {  // (flat tiles)
            ring2_slot(r, hi, hj);
            load(cell(i0 - 2 + hi, j0 - 2 + hj), h);
            put(hi * DW + hj, h, diss_pressure(P, h));
        }
    }
    const double rdt = P.local ? 0.0 : recip(*A.dtmin);
    __syncthreads();
    // sensors, Laplacians and VOL/DT of the cell at halo-1 position (li, lj), state q
    auto sense = [&](int li, int lj, const double q[5], double p, double v) {
        const int d = (li + 1) * DW + lj + 1, s = li * SW + lj;
        const int nb[4] = {d - 1, d + DW, d + 1, d - DW};
        double l[5], an = 0.0, ad = 0.0, rn = 0.0, rd = 0.0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const double2 a = S.c01[nb[k]], b = S.c23[nb[k]], c = S.c4p[nb[k]];
            const double n[5] = {a.x, a.y, b.x, b.y, c.x};
#pragma unroll
            for (int m = 0; m < 5; m++) l[m] = k == 0 ? n[m] : l[m] + n[m];
            an += fabs(c.y - p);
            ad += fabs(c.y + p);
            rn += fabs(c.x - q[4]);
            rd += fabs(c.x + q[4]);
        }
#pragma unroll
        for (int m = 0; m < 5; m++) l[m] = l[m] - 4.0 * q[m];
        S.l01[s] = pair((R)l[0], (R)l[1]);
        S.l23[s] = pair((R)l[2], (R)l[3]);
        S.l4v[s] = pair((R)l[4], (R)v);
        S.anu[s] = pair(quotient((R)an, (R)ad), quotient((R)rn, (R)dmax1(rd, 8.0 * q[0] * P.rtol)));
    };
    {
        const double sp = P.local ? diss_speed(P, q, p) : 0.0;
        if (P.local && i < M.ni && j < M.nj) A.dt[own] = (R)(M.cfldl[own] * recip(sp));
        sense(ti + 1, tj + 1, q, p, vs * (P.local ? sp : rdt));
    }
    if (tid < NRING) {
        const int d = (ri + 1) * DW + rj + 1;
        const double2 a = S.c01[d], b = S.c23[d], c = S.c4p[d];
        const double h[5] = {a.x, a.y, b.x, b.y, c.x};
        sense(ri, rj, h, c.y, vr * (P.local ? diss_speed(P, h, c.y) : rdt));
    }
    if (tid == NTHREADS - 1) {
        const double2 a = S.c01[2 * DW + 2], b = S.c23[2 * DW + 2], c = S.c4p[2 * DW + 2];
        const double first[5] = {a.x, a.y, b.x, b.y, c.x};
        ref(first);  // the tile's first cell
    }
    __syncthreads();
    if (i >= M.ni || j >= M.nj) return;
    const int r = (ti + 1) * SW + tj + 1, d = (ti + 2) * DW + tj + 2;
    const int rn[4] = {r - 1, r + SW, r + 1, r - SW}, dn[4] = {d - 1, d + DW, d + 1, d - DW};
    const bool has[4] = {j > 0, i < M.ni - 1, j < M.nj - 1, i > 0};
    const auto l01 = S.l01[r], l23 = S.l23[r], l4v = S.l4v[r], an = S.anu[r];
    const R l[5] = {l01.x, l01.y, l23.x, l23.y, l4v.x};
    R D[5] = {(R)0, (R)0, (R)0, (R)0, (R)0};
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (!has[k]) continue;  // ghost face: exactly zero contribution
        const auto n01 = S.l01[rn[k]], n23 = S.l23[rn[k]], n4v = S.l4v[rn[k]], nan_ = S.anu[rn[k]];
        const double2 a = S.c01[dn[k]], b = S.c23[dn[k]], c = S.c4p[dn[k]];
        const R d24 = (R)HALF * (l4v.y + n4v.y);
        R e2 = (R)C02 * (an.x >= nan_.x ? an.x : nan_.x);
        R e4 = (R)C04 - e2;
        const R a2 = e2 * d24, a4 = ((R)0 >= e4 ? (R)0 : e4) * d24;
        e2 = (R)C02 * (an.y >= nan_.y ? an.y : nan_.y);
        e4 = (R)C04 - e2;
        const R t2 = e2 * d24, t4 = ((R)0 >= e4 ? (R)0 : e4) * d24;
        const double n[5] = {a.x, a.y, b.x, b.y, c.x};
        const R ln[5] = {n01.x, n01.y, n23.x, n23.y, n4v.x};
#pragma unroll
        for (int m = 0; m < 5; m++)
            D[m] += (m == 4 ? t2 : a2) * (R)(n[m] - q[m]) - (m == 4 ? t4 : a4) * (ln[m] - l[m]);
    }
#pragma unroll
    for (int m = 0; m < 5; m++) A.d[m * ncell + own] = D[m];
}

}  // namespace tns
