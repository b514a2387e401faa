// tns_kernels.cu -- FP64 kernels of one RK4 iteration on a structured i x j block.
//
// Per iteration (turbnstwod.f90:95-168):
//   [k_dtmin]      global time step (LOCAL=0 only): per-cell DT and a grid-wide min
//   k_dissipation  DT (LOCAL=1) and the frozen JST dissipation D of Q_old
//                  (solver_state.f90:70-225), radius-2 shared-memory tile
//   k_viscous      nodal averages and the frozen viscous flux VIS of Q_old, each face once
//   k_stage        primitives + ghost BCs + source + residual + update, four times (alpha 1/4,
//                  1/3, 1/2, 1); the first writes VIS + D for the others, the last one also
//                  reduces CDIFF and checks the state is finite; k_stage_pipe is its form for
//                  large meshes
//   [k_gport]      type-6 port mass flux of the stage input (only if such ghosts exist)
// Ghost cells are never stored: each tile evaluates the BC of the ghosts in its halo
// from the parent and the parent's opposite neighbour, both already in the tile.
#include <cooperative_groups.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "tns_device.cuh"
#include "tns_kernels.h"
#include "tns_tile.cuh"
#include "tns_batch.cuh"
#include "tns_diss.cuh"
#include "tns_visc.cuh"

namespace tns {

// ------------------------------------------------------------------ stage kernel

// Shared-memory fields of the stage tile: per slot the six values its neighbours' face
// fluxes are formed from and |V|, paired for 16-byte loads; the tile's static block (nodes,
// gradient coefficients, 1/VOL, 1/YCC) arrives by one bulk copy.  A cell's flux through a
// face needs its mass flux m = RHO (U SX + V SY) alone: (m, m U + P SX, m V + P SY,
// (C4 + P)(U SX + V SY), m C5/C1), ten operations a neighbour from seven stored values
// instead of ten stored flux components (a tile's slots take 19 KB, not 38).  A ghost keeps
// its own flux through its face (a wall's components are mirrored, an outflow's fifth is the
// parent's), by the tile cell it borders.
// What bounds it: instruction issue and memory latency (735 instructions a cell, a third of
// them FP64).  On a small mesh every tile borders the boundary and one tile's latency is the
// kernel's: the ghosts' static data is loaded before the previous kernel has ended and every
// state a slot needs is asked for at once, which took a boundary tile from 10,200 to 7,200
// cycles (115 x 50 nozzle, a FP64 iteration: 37.6 -> 27.4 us).
// Slot order: each thread first evaluates the slot of its own cell, then the first threads
// evaluate the ring of slots around the tile's cells (tns_tile.cuh).
static_assert(NRING <= NTHREADS, "one ring slot per thread at most");
constexpr int NGF = 2 * (TI + TJ);  // ghosts bordering a tile: sides 1, 3 by row, 4, 2 by column

// The slots of one tile.
struct StageSlots {
    double2 uv[NSLOT];     // (U, V)
    double2 rp[NSLOT];     // (RHO, P)
    double2 hr[NSLOT];     // (C4 + P, C5/C1)
    double qm[NSLOT];      // |V|
    double gf[5][NGF];     // the ghosts' fluxes through the faces they border
};

struct StageSmem {
    double st[STILE];      // static block (tns_tile.cuh)
    StageSlots w;
    unsigned long long bar;  // completion of the static block's copy
};

size_t stage_smem_bytes() { return sizeof(StageSmem); }

// With extra thread rows, the update operands of the tile's cells too: Q_old, DT and VIS + D (in
// stage 1 D and VIS), a plane of NTHREADS each, asked for with the states: their latency is then
// no longer the end of the tile's chain (115 x 50 nozzle, an iteration, 22.2 -> 20.6 us; 201 x 67
// ramp 23.1 -> 21.9; in registers instead 21.6, and 5 % slower at two blocks an SM).  With more
// tiles the other blocks hide it, and the shared memory is worth more as L1 (384 tiles: 35.7 ->
// 38.8 us, so those read the operands at the end).
enum RimOp { RO_QOLD, RO_DT = 5, RO_E = 6, RO_D = 6, RO_VIS = 11, RO_N = 15 };
constexpr size_t RIM_SMEM = sizeof(StageSmem) + sizeof(double) * RO_N * NTHREADS;

__device__ __forceinline__ void put_slot(StageSlots& S, int s, const Prim& p, double h) {
    S.uv[s] = make_double2(p.u, p.v);
    S.rp[s] = make_double2(p.rho, p.p);
    S.hr[s] = make_double2(h, p.ri);
    S.qm[s] = p.qm;
}

// A cell's slot from its state; returns the cell's T (read for the cell alone).
__device__ __forceinline__ double put_cell_slot(const Params& P, StageSlots& S, int s, const double q[5]) {
    Prim p;
    primitive(P, q[0], q[1], q[2], q[3], q[4], p);
    put_slot(S, s, p, q[3] + p.p);
    return kept(p.t);
}

// The slot of halo position h: a cell's from its state q, a ghost's (and, where it borders a
// cell of the tile, its flux through their face) from its parent's state q; opp(double[5])
// gives the state of the parent's opposite neighbour.
template <class Opp>
__device__ __forceinline__ void put_halo_slot(const Params& P, const Mesh& M, StageSlots& S, const HaloPos& h,
                                              const GhostSite& site, const double q[5], Opp opp) {
    Prim p;
    primitive(P, q[0], q[1], q[2], q[3], q[4], p);
    if (h.kind == 0) {
        put_slot(S, h.li * SW + h.lj, p, q[3] + p.p);
        return;
    }
    Prim gh;
    ghost_prim(P, M, site, h.g, p,
               [&](Prim& o) {
                   double c[5];
                   opp(c);
                   primitive(P, c[0], c[1], c[2], c[3], c[4], o);
               }, gh);
    put_slot(S, h.li * SW + h.lj, gh, 0.0);
    const bool row = h.kind == 1 || h.kind == 3;  // ghosts beside the tile's rows
    const int at = (row ? h.li : h.lj) - 1;
    if (at >= 0 && at < (row ? TI : TJ)) {
        const int f = (h.kind == 1 ? 0 : h.kind == 3 ? TI : h.kind == 4 ? 2 * TI : 2 * TI + TJ) + at;
#pragma unroll
        for (int m = 0; m < 5; m++) S.gf[m][f] = gh.f[m] * site.psx + gh.g[m] * site.psy;
    }
}

// The update operands of one cell: Q_old, the frozen terms VIS + D and DT.
struct StageOps {
    double qold[5], e[5], dt;
};

// Residual, source and update of the thread's cell (i, j) of a tile from the tile's slots,
// its nodes, the cells' static coefficients and `ops(StageOps&)`, which is called last and
// may wait for the update operands.
template <class Ops>
__device__ __forceinline__ void stage_cell(const Params& P, const Mesh& M, const StageArgs& A, const StageSlots& S,
                                           const double* nodes, const double* coef, bool inner, int i, int j,
                                           double own_t, Ops ops, double dv[5]) {
    const size_t ncell = (size_t)M.ni * M.nj;
    const int tj = threadIdx.x, ti = threadIdx.y, tid = ti * TJ + tj;
    const size_t cell = (size_t)i * M.nj + j;
    const int c = (ti + 1) * SW + (tj + 1);
    const int nb[4] = {c - 1, c + SW, c + 1, c - SW};  // NC1..NC4
    const double* X0 = nodes + ti * SNW + tj;  // node 1 of the cell
    const double* Y0 = X0 + SNN;
    const double X[4] = {X0[0], X0[SNW], X0[SNW + 1], X0[1]};
    const double Y[4] = {Y0[0], Y0[SNW], Y0[SNW + 1], Y0[1]};

    // inviscid residual (residual.f90:23-62): half the sum over the faces of the cell's own
    // flux and the neighbour's; the own flux meets the sum of the face vectors
    double R[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    {
        double SX[4], SY[4];
#pragma unroll
        for (int k = 0; k < 4; k++) face_vector(P.iaxis, k + 1, X, Y, SX[k], SY[k]);
        auto add = [&](int s, double sx, double sy) {
            const double2 uv = S.uv[s], rp = S.rp[s], hr = S.hr[s];
            const double vn = uv.x * sx + uv.y * sy;
            const double m = rp.x * vn;
            R[0] = R[0] + m;
            R[1] = fma(m, uv.x, fma(rp.y, sx, R[1]));
            R[2] = fma(m, uv.y, fma(rp.y, sy, R[2]));
            R[3] = fma(hr.x, vn, R[3]);
            R[4] = fma(m, hr.y, R[4]);
        };
        add(c, (SX[0] + SX[2]) + (SX[1] + SX[3]), (SY[0] + SY[2]) + (SY[1] + SY[3]));
        const bool gh[4] = {j == 0, i == M.ni - 1, j == M.nj - 1, i == 0};
        const int gs[4] = {ti, 2 * TI + TJ + tj, TI + ti, 2 * TI + tj};
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (!inner && gh[k]) {
#pragma unroll
                for (int m = 0; m < 5; m++) R[m] = R[m] + S.gf[m][gs[k]];
            } else {
                add(nb[k], SX[k], SY[k]);
            }
        }
    }

    // source terms (source_terms.f90:24-104)
    double src3, src5;
    {
        const double* G = coef + tid;
        SrcIn s;
        s.ga = G[ST_GA * NTHREADS]; s.gb = G[ST_GB * NTHREADS];
        s.gc = G[ST_GC * NTHREADS]; s.gd = G[ST_GD * NTHREADS];
        const double2 ua = S.uv[nb[0]], ub = S.uv[nb[1]], uc = S.uv[nb[2]], ud = S.uv[nb[3]];
        s.ua = ua.x; s.ub = ub.x; s.uc = uc.x; s.ud = ud.x;
        s.va = ua.y; s.vb = ub.y; s.vc = uc.y; s.vd = ud.y;
        s.ra = S.hr[nb[0]].y; s.rb = S.hr[nb[1]].y; s.rc = S.hr[nb[2]].y; s.rd = S.hr[nb[3]].y;
        s.qa = S.qm[nb[0]]; s.qb = S.qm[nb[1]]; s.qc = S.qm[nb[2]]; s.qd = S.qm[nb[3]];
        const double YCCI = (Y[0] + Y[1] + Y[2] + Y[3]) * 0.25;
        source_terms(P, s, S.rp[c].x, S.hr[c].y, own_t, S.rp[c].y, S.uv[c].y, YCCI, G[ST_RYCC * NTHREADS], src3, src5);
    }

    // update (residual.f90:67-83), the sources per volume
    const double RVOL = coef[ST_RVOL * NTHREADS + tid];
    StageOps o;
    ops(o);
    const double aDT = A.alpha * o.dt;
    double Cn[5];
    const double* Co = o.qold;
    Cn[0] = Co[0] - aDT * (RVOL * (HALF * R[0] - o.e[0]));
    Cn[1] = Co[1] - aDT * (RVOL * (HALF * R[1] - o.e[1]));
    Cn[2] = Co[2] - aDT * fma(RVOL, HALF * R[2] - o.e[2], -src3);
    Cn[3] = Co[3] - aDT * (RVOL * (HALF * R[3] - o.e[3]));
    Cn[4] = Co[4] - aDT * CFLTURB * fma(RVOL, HALF * R[4] - o.e[4], -src5);
    Cn[4] = Cn[0] * dmax1(P.rtol, quot(Cn[4], Cn[0]));
#pragma unroll
    for (int m = 0; m < 5; m++) A.qout[m * ncell + cell] = Cn[m];
    if (A.status) {
        bool bad = false;
#pragma unroll
        for (int m = 0; m < 5; m++) bad |= !isfinite(Cn[m]);
        if (bad) atomicOr(A.status, 1u);
    }
#pragma unroll
    for (int m = 0; m < 5; m++) dv[m] = fabs(Co[m] - Cn[m]);
}

// The frozen terms VIS + D of a cell, by stage 1; D and VIS read from planes `dst` apart.
__device__ __forceinline__ void frozen_terms(const StageArgs& A, size_t ncell, size_t cell, const double* dp,
                                             const double* vp, size_t dst, double e[5]) {
    double d[5], v[4];
#pragma unroll
    for (int m = 0; m < 5; m++) d[m] = dp[m * dst];
#pragma unroll
    for (int m = 0; m < 4; m++) v[m] = vp[m * dst];
    e[0] = d[0];
#pragma unroll
    for (int m = 1; m < 5; m++) e[m] = v[m - 1] + d[m];
    if (A.eout) {
#pragma unroll
        for (int m = 0; m < 5; m++) A.eout[m * ncell + cell] = e[m];
    }
}

// max |COLD - C| per component: warp max, then one atomic per warp on the ordered bit
// pattern (non-negative doubles order like their bits)
__device__ __forceinline__ void stage_cdiff(const StageArgs& A, const double dv[5]) {
#pragma unroll
    for (int m = 0; m < 5; m++) {
        double v = dv[m];
        for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
        if ((threadIdx.x & 31) == 0) atomicMax(&A.cdiff[m], (unsigned long long)__double_as_longlong(v));
    }
}

// One RK stage (turbnstwod.f90:204-227, boundary.f90:24-48, source_terms.f90:24-104,
// residual.f90:23-83) on a TI x TJ tile with its halo staged in shared memory.  RIM: the block
// has RIM_ROWS more rows of threads, which evaluate the halo.  The result: tile_copy_wait.
template <bool RIM>
__device__ __forceinline__ bool stage_tile(const Params& P, const Mesh& M, const StageArgs& A, int bx, int by) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    StageSmem& S = *reinterpret_cast<StageSmem*>(smem_raw);
    const size_t ncell = (size_t)M.ni * M.nj;
    const int j0 = bx * TJ, i0 = by * TI;
    const int tj = threadIdx.x, ti = threadIdx.y;
    const int tid = ti * TJ + tj;
    pdl_trigger();
    // the static block is written by nothing: its copy overlaps the previous kernel's tail
    if (tid == 0) {
        bulk_barrier_init(&S.bar);
        const size_t tile = (size_t)by * ((M.nj + TJ - 1) / TJ) + bx;
        bulk_copy_start(S.st, M.stile + tile * STILE, STILE * sizeof(double), &S.bar);
    }
    // a tile whose halo holds no ghost (and which is full) needs no classification
    const bool inner = i0 > 0 && j0 > 0 && i0 + TI < M.ni && j0 + TJ < M.nj;
    const int i = i0 + ti, j = j0 + tj;
    const bool valid = (!RIM || ti < TI) && i < M.ni && j < M.nj;
    const int rt = RIM ? tid - NTHREADS : tid;  // the thread's place on the ring
    // the ring around the tile's cells; a ghost's type and geometry are static too
    const int ri = inner ? TI : min(TI, M.ni - i0), rj = inner ? TJ : min(TJ, M.nj - j0);
    HaloPos h;
    h.kind = -1;
    GhostSite site{0, 0.0, 0.0, 0.0, 0.0};
    if (rt >= 0 && rt < 2 * (ri + rj + 2)) {
        int li, lj;
        ring_slot(rt, ri, rj, li, lj);
        h = halo_pos(M, inner, i0, j0, li, lj);
        if (h.kind > 0) site = ghost_site(M, h.g);
    }
    pdl_wait();
    __syncthreads();
    auto load = [&](int ci, int cj, double q[5]) {
        const double* p = A.qin + ((size_t)ci * M.nj + cj);
#pragma unroll
        for (int m = 0; m < 5; m++) q[m] = p[m * ncell];
    };
    // own cell (its T kept) and ring slot, both states on their way first
    double qo[5], qr[5], own_t = 0.0;
    if (valid) load(i, j, qo);
    if (h.kind >= 0) load(h.ci, h.cj, qr);
    double* op = reinterpret_cast<double*>(smem_raw + sizeof(StageSmem)) + tid;
    if (RIM && valid) {
        const size_t cell = (size_t)i * M.nj + j;
        auto fetch = [&](int at, int n, const double* src) {
#pragma unroll
            for (int m = 0; m < n; m++) copy_async(op + (at + m) * NTHREADS, src + m * ncell + cell);
        };
        fetch(RO_QOLD, 5, A.qold);
        if (P.local) fetch(RO_DT, 1, A.dt);
        if (A.e) {
            fetch(RO_E, 5, A.e);
        } else {
            fetch(RO_D, 5, A.d);
            fetch(RO_VIS, 4, A.vis);
        }
    }
    if (valid) own_t = put_cell_slot(P, S.w, (ti + 1) * SW + tj + 1, qo);
    if (h.kind >= 0) put_halo_slot(P, M, S.w, h, site, qr, [&](double c[5]) { load(h.ci + h.oi, h.cj + h.oj, c); });
    const bool arrived = tile_copy_wait(&S.bar, A.error);
    double dv[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (valid) {
        const size_t cell = (size_t)i * M.nj + j;
        stage_cell(P, M, A, S.w, S.st, S.st + 2 * SNN, inner, i, j, own_t,
                   [&](StageOps& o) {
                       if (RIM) copies_wait();
#pragma unroll
                       for (int m = 0; m < 5; m++)
                           o.qold[m] = RIM ? op[(RO_QOLD + m) * NTHREADS] : A.qold[m * ncell + cell];
                       o.dt = !P.local ? *A.dtmin : RIM ? op[RO_DT * NTHREADS] : A.dt[cell];
                       if (A.e) {
#pragma unroll
                           for (int m = 0; m < 5; m++) o.e[m] = RIM ? op[(RO_E + m) * NTHREADS] : A.e[m * ncell + cell];
                       } else if (RIM) {
                           frozen_terms(A, ncell, cell, op + RO_D * NTHREADS, op + RO_VIS * NTHREADS, NTHREADS, o.e);
                       } else {
                           frozen_terms(A, ncell, cell, A.d + cell, A.vis + cell, ncell, o.e);
                       }
                   }, dv);
    }
    if (A.cdiff) stage_cdiff(A, dv);
    return arrived;
}

// Specialised on the residual monitor, so the CDIFF reduction is compiled only where it
// runs, and on the extra rows of threads.
template <int MONITOR, bool RIM>
__global__ void __launch_bounds__(NTHREADS + (RIM ? TJ * RIM_ROWS : 0), RIM ? RIM_MINB : TNS_PER_SM(TNS_STAGE_MINB))
k_stage(Params P, Mesh M, StageArgs A) {
    StageArgs Ac = A;
    if (!MONITOR) Ac.cdiff = nullptr;
    stage_tile<RIM>(P, M, Ac, blockIdx.x, blockIdx.y);
}

// A stage of a large mesh, by resident blocks that walk its tiles (tile t, t + grid, ...)
// with the data of the next tile on its way through the TMA engine while they compute:
//   a: the stage input's halo box (rows i0-1 .. i0+TI, columns j0-2 .. j0+TJ+1: one column
//      early so that the box starts at a multiple of 16 bytes; positions outside the mesh
//      arrive as zeros), asked for as soon as the tile before has formed its slots;
//   b: the tile's static block, and
//   c: Q_old, the frozen terms and DT of its cells (FIRST: D, VIS and DT), asked for when the
//      tile before is done and needed when this one's slots are formed, and at its very end.
// The copies take the global-load latency (4.7 of 11.6 stall cycles an instruction in the
// kernel above, half of its time) out of the warps; a tile's buffers fit three times into an
// SM because VIS + D is one array (and stage 1's Q_old is its input, read again from global
// memory), so 24 warps stay resident at 80 registers (with D and VIS apart and two blocks an SM
// it was no faster than the plain kernel).  What bounds it now: issue (0.5 an SM quarter a cycle
// under 24 warps) and the launch.  1024 x 384 nozzle-plume, a FP64 iteration: 0.153 ms with the
// plain kernel in all stages, 0.138 ms with this one; 2048 x 768 port 0.647 -> 0.565 ms; stage 1
// by it as well 0.1179 -> 0.1161 ms.  It needs more tiles than the plain kernel has resident
// blocks (at 384 tiles the two take the same 42 us an iteration) and rows and arrays that TMA can
// address.
constexpr int QH = TI + 2, QW = TJ + 4;  // halo box
static_assert(QW % 2 == 0 && STILE % 2 == 0, "box rows and static blocks are multiples of 16 bytes");

// Planes of the update operands
// (stage 1: VIS, D and DT; its Q_old is its input, and read again from global memory)
enum StageOp { SO_QOLD, SO_VIS = 0, SO_E = 5, SO_DT = 10, SO_N };

struct StagePipeSmem {
    // (128-byte aligned destinations first)
    double q[(5 * QH * QW + 15) / 16 * 16];
    double op[SO_N][NTHREADS];
    double st[STILE];
    StageSlots w;
    unsigned long long bar_a, bar_b, bar_c;
};

struct StageMaps {
    CUtensorMap q, qold, e, dt;
};

template <int MONITOR, bool FIRST>
__global__ void __launch_bounds__(NTHREADS, TNS_PER_SM(TNS_STAGE_MINB))
k_stage_pipe(Params P, Mesh M, StageArgs A, int ntiles, const __grid_constant__ StageMaps maps) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const unsigned skew = (128u - ((unsigned)__cvta_generic_to_shared(smem_raw) & 127u)) & 127u;
    StagePipeSmem& W = *reinterpret_cast<StagePipeSmem*>(smem_raw + skew);
    StageSlots& S = W.w;
    const int ntj = (M.nj + TJ - 1) / TJ;
    const int tj = threadIdx.x, ti = threadIdx.y, tid = ti * TJ + tj;
    // tile t: row t / ntj, its column shifted by the row so that a block whose stride is a
    // multiple of ntj does not meet the same (boundary) column every time
    auto row_of = [&](int t) { return t / ntj; };
    auto col_of = [&](int t) { return (t % ntj + t / ntj) % ntj; };
    auto fetch_a = [&](int t) {
        barrier_expect(&W.bar_a, sizeof(double) * 5 * QH * QW);
        tensor_copy_3d(W.q, &maps.q, col_of(t) * TJ - 2, row_of(t) * TI - 1, 0, &W.bar_a);
    };
    auto fetch_b = [&](int t) {
        const size_t tile = (size_t)row_of(t) * ntj + col_of(t);
        bulk_copy_start(W.st, M.stile + tile * STILE, sizeof(double) * STILE, &W.bar_b);
    };
    auto fetch_c = [&](int t) {
        const int j0 = col_of(t) * TJ, i0 = row_of(t) * TI;
        barrier_expect(&W.bar_c, sizeof(double) * ((FIRST ? 9 : 10) + (P.local ? 1 : 0)) * NTHREADS);
        tensor_copy_3d(W.op[SO_E], &maps.e, j0, i0, 0, &W.bar_c);
        tensor_copy_3d(W.op[SO_QOLD], &maps.qold, j0, i0, 0, &W.bar_c);
        if (P.local) tensor_copy_3d(W.op[SO_DT], &maps.dt, j0, i0, 0, &W.bar_c);
    };
    if (tid == 0) {
        bulk_barrier_init(&W.bar_a);
        bulk_barrier_init(&W.bar_b);
        bulk_barrier_init(&W.bar_c);
        fetch_b(blockIdx.x);  // static: before the previous kernel is done
    }
    pdl_wait();
    if (tid == 0) {
        fetch_a(blockIdx.x);
        fetch_c(blockIdx.x);
    }
    __syncthreads();  // the barriers are set up
    unsigned parity = 0;
    bool ok = true;
    double dv[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, parity ^= 1) {
        const int i0 = row_of(t) * TI, j0 = col_of(t) * TJ;
        const int i = i0 + ti, j = j0 + tj;
        const bool valid = i < M.ni && j < M.nj;
        const bool inner = i0 > 0 && j0 > 0 && i0 + TI < M.ni && j0 + TJ < M.nj;
        auto box = [&](int ci, int cj, double q[5]) {
            const double* b = W.q + (ci - i0 + 1) * QW + (cj - j0 + 2);
#pragma unroll
            for (int m = 0; m < 5; m++) q[m] = b[m * QH * QW];
        };
        ok = bulk_wait(&W.bar_a, parity) && ok;
        double own_t = 0.0;
        if (valid) {
            double q[5];
            box(i, j, q);
            own_t = put_cell_slot(P, S, (ti + 1) * SW + tj + 1, q);
        }
        const int ri = inner ? TI : min(TI, M.ni - i0), rj = inner ? TJ : min(TJ, M.nj - j0);
        if (tid < 2 * (ri + rj + 2)) {
            int li, lj;
            ring_slot(tid, ri, rj, li, lj);
            const HaloPos h = halo_pos(M, inner, i0, j0, li, lj);
            if (h.kind >= 0) {
                double q[5];
                box(h.ci, h.cj, q);
                GhostSite site{0, 0.0, 0.0, 0.0, 0.0};
                if (h.kind > 0) site = ghost_site(M, h.g);
                put_halo_slot(P, M, S, h, site, q, [&](double c[5]) { box(h.ci + h.oi, h.cj + h.oj, c); });
            }
        }
        ok = bulk_wait(&W.bar_b, parity) && ok;
        if (!__syncthreads_and(ok)) {
            // a copy did not complete: report it, give the copies in flight one more bounded
            // wait (they write this block's shared memory) and leave
            if (tid == 0) {
                atomicOr(A.error, 2u);
                bulk_wait(&W.bar_a, parity);
                bulk_wait(&W.bar_b, parity);
                bulk_wait(&W.bar_c, parity);
            }
            return;
        }
        const int next = t + gridDim.x;
        // the next kernel's blocks may start once all of these are on their last tile (asked
        // for at the start they take an SM's slots early: 0.122 -> 0.125 ms an iteration)
        if (next >= ntiles) pdl_trigger();
        if (tid == 0 && next < ntiles) fetch_a(next);
        if (valid) {
            double d[5];
            stage_cell(P, M, A, S, W.st, W.st + 2 * SNN, inner, i, j, own_t,
                       [&](StageOps& o) {
                           ok = bulk_wait(&W.bar_c, parity) && ok;
                           const size_t cell = (size_t)i * M.nj + j, ncell = (size_t)M.ni * M.nj;
#pragma unroll
                           for (int m = 0; m < 5; m++)
                               o.qold[m] = FIRST ? A.qold[m * ncell + cell] : W.op[SO_QOLD + m][tid];
                           if (FIRST) {
                               frozen_terms(A, ncell, cell, &W.op[SO_E][tid], &W.op[SO_VIS][tid], NTHREADS, o.e);
                           } else {
#pragma unroll
                               for (int m = 0; m < 5; m++) o.e[m] = W.op[SO_E + m][tid];
                           }
                           o.dt = P.local ? W.op[SO_DT][tid] : *A.dtmin;
                       }, d);
            if (MONITOR) {
#pragma unroll
                for (int m = 0; m < 5; m++) dv[m] = fmax(dv[m], d[m]);
            }
        }
        ok = bulk_wait(&W.bar_c, parity) && ok;  // (threads without a cell, too)
        __syncthreads();
        if (tid == 0 && next < ntiles) {
            fetch_b(next);
            fetch_c(next);
        }
    }
    if (!ok) {  // the last tile's operands
        atomicOr(A.error, 2u);
        bulk_wait(&W.bar_c, parity ^ 1);
    }
    if (MONITOR && A.cdiff) stage_cdiff(A, dv);
}

// ---------------------------------------------------------------- viscous kernel

size_t visc_smem_bytes() { return sizeof(ViscSmem<double>); }

template <bool RIM>
__device__ __forceinline__ bool viscous_tile_f64(const Params& P, const Mesh& M, const double* __restrict__ q,
                                                 double* __restrict__ vis, unsigned int* error, int bx, int by) {
    return viscous_tile<RIM, double>(P, M, q, vis, error, bx, by,
                                     [&](const FaceVals& f, double sx, double sy, double ga, double gb, double gc,
                                         double gd, double ry, double out[4]) {
                                         viscous_face(P, f, sx, sy, ga, gb, gc, gd, ry, out);
                                     });
}

template <bool RIM>
__global__ void __launch_bounds__(NTHREADS + (RIM ? TJ * RIM_ROWS : 0), RIM ? RIM_MINB : TNS_PER_SM(TNS_VISC_MINB))
k_viscous(Params P, Mesh M, const double* __restrict__ q, double* __restrict__ vis, unsigned int* error) {
    viscous_tile_f64<RIM>(P, M, q, vis, error, blockIdx.x, blockIdx.y);
}

// --------------------------------------------------------- dissipation kernel

size_t diss_smem_bytes() { return sizeof(DissSmem<double>); }

__device__ __forceinline__ void dissipation_tile_f64(const Params& P, const Mesh& M, const DissArgs<double>& A, int bx,
                                                     int by) {
    dissipation_tile(P, M, A, bx, by, [](const double*) {});
}

__global__ void __launch_bounds__(NTHREADS, TNS_PER_SM(TNS_DISS_MINB))
k_dissipation(Params P, Mesh M, DissArgs<double> A) {
    dissipation_tile_f64(P, M, A, blockIdx.x, blockIdx.y);
}

// ------------------------------------------------------------- time step min

// The time step of up to STEP_UNROLL cells a thread, a block apart: all their loads are on
// their way before the first is used (a grid of one load round at a time was bound by their
// latency).
constexpr int STEP_UNROLL = 4;
template <class Store>
__device__ __forceinline__ double step_min(const Params& P, const double* __restrict__ q,
                                           const double* __restrict__ cfldl, long long ncell, long long first,
                                           long long stride, double mn, Store store) {
    for (; first < ncell; first += STEP_UNROLL * stride) {
        double c[STEP_UNROLL][5];
#pragma unroll
        for (int k = 0; k < STEP_UNROLL; k++) {
            const long long i = first + k * stride;
            if (i < ncell) {
#pragma unroll
                for (int m = 0; m < 4; m++) c[k][m] = q[m * ncell + i];
                c[k][4] = cfldl[i];
            }
        }
#pragma unroll
        for (int k = 0; k < STEP_UNROLL; k++) {
            const long long i = first + k * stride;
            if (i < ncell) {
                const double v = local_dt(P, c[k][0], c[k][1], c[k][2], c[k][3], c[k][4]);
                store(i, v);
                mn = dmin1(mn, v);
            }
        }
    }
    return mn;
}

// Minimum over the grid: a partial per block, and the block that finishes last reduces them
// with all its threads (one thread reading them in turn took most of the kernel: 65 -> 21 us
// for the time step of 1.57 M cells).  `partial`: one double per block; `counter`: zero on
// entry, left at zero.
__device__ __forceinline__ void grid_min(double mn, double* partial, unsigned int* counter, double* dtmin) {
    __shared__ double wmin[8];
    __shared__ bool last;
    auto block_min = [&](double v) {
        for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
        if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = v;
        __syncthreads();
        v = wmin[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) v = fmin(v, wmin[w]);
        return v;
    };
    const double b = block_min(mn);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = b;
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double v = 100000.0;
    for (unsigned int k = threadIdx.x; k < gridDim.x; k += blockDim.x) v = fmin(v, ((volatile double*)partial)[k]);
    v = block_min(v);
    if (threadIdx.x == 0) {
        *dtmin = v;
        *counter = 0u;
    }
}

__global__ void __launch_bounds__(256)
k_dtmin(Params P, Mesh M, const double* __restrict__ q, double* partial, unsigned int* counter, double* dtmin) {
    const long long ncell = (long long)M.ni * M.nj;
    const double mn = step_min(P, q, M.cfldl, ncell, blockIdx.x * 256LL + threadIdx.x, gridDim.x * 256LL, 100000.0,
                               [](long long, double) {});
    grid_min(mn, partial, counter, dtmin);
}

// Variant of k_dtmin for caller-provided device buffers (tns_time_step_noalloc): also
// stores the per-cell DT, and reduces through the scratch the launcher is handed.
__global__ void __launch_bounds__(256)
k_time_step_scratch(Params P, const double* __restrict__ q, const double* __restrict__ cfldl,
                    long long ncell, double* __restrict__ dt, double* partial,
                    unsigned int* counter, double* dtmin) {
    const double mn = step_min(P, q, cfldl, ncell, blockIdx.x * 256LL + threadIdx.x, gridDim.x * 256LL, 100000.0,
                               [&](long long i, double v) { dt[i] = v; });
    grid_min(mn, partial, counter, dtmin);
}

// The same for a mesh that one cluster of blocks covers in a few rounds: the minimum goes through
// the cluster's shared memory, so no scratch, and no counter to clear in a launch of its own.
// Such calls were bound by the two launches: 5000 cells 8.1 -> 3.2 us on the device, 20,000 8.2 ->
// 5.5, and the host's part of a call 0.7 us less; from some 33,000 on (8.2 both ways) the larger
// grid is ahead.
__global__ void __cluster_dims__(STEP_CLUSTER, 1, 1) __launch_bounds__(256)
k_time_step_cluster(Params P, const double* __restrict__ q, const double* __restrict__ cfldl, long long ncell,
                    double* __restrict__ dt, double* dtmin) {
    __shared__ double wmin[8], bmin;
    double mn = step_min(P, q, cfldl, ncell, blockIdx.x * 256LL + threadIdx.x, STEP_CLUSTER * 256LL, 100000.0,
                         [&](long long i, double v) { dt[i] = v; });
    for (int o = 16; o > 0; o >>= 1) mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = mn;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) mn = fmin(mn, wmin[w]);
        bmin = mn;
    }
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    cluster.sync();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        for (int b = 1; b < STEP_CLUSTER; b++) mn = fmin(mn, *cluster.map_shared_rank(&bmin, b));
        *dtmin = mn;
    }
    cluster.sync();  // no block leaves before its minimum is read
}

void launch_time_step_cluster(const Params& P, const double* q, const double* cfldl, long long ncell, double* dt,
                              double* dtmin, cudaStream_t s) {
    k_time_step_cluster<<<STEP_CLUSTER, 256, 0, s>>>(P, q, cfldl, ncell, dt, dtmin);
}

void launch_time_step_scratch(const Params& P, const double* q, const double* cfldl,
                              long long ncell, double* dt, double* partial,
                              unsigned int* counter, double* dtmin, int nblocks,
                              cudaStream_t s) {
    k_time_step_scratch<<<nblocks, 256, 0, s>>>(P, q, cfldl, ncell, dt, partial, counter, dtmin);
}

// ------------------------------------------------------------ port mass flux

// One block per type-6 ghost (port_line, tns_tile.cuh).
__global__ void __launch_bounds__(GP_THREADS) k_gport(Params P, Mesh M, const double* __restrict__ q,
                                                      const int* ghosts, double* gport) {
    port_line(M, StateF64{q, (size_t)M.ni * M.nj}, ghosts, gport);
}

// ------------------------------------------------------ primitive output

// U, V, T, P of every cell and ghost computed from q (the last stage's input), the
// arrays COMPUTE_PRIMITIVE_VARS / APPLY_BOUNDARY leave behind.  Output layout:
// [4][ncell + nghost] with ghosts in side-array order.
__global__ void k_prim_out(Params P, Mesh M, const double* __restrict__ q, double* out) {
    const size_t ncell = (size_t)M.ni * M.nj;
    const size_t ng = M.nghosts(), ntot = ncell + ng;
    const size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (k >= ntot) return;
    Prim p;
    if (k < ncell) {
        cell_prim(P, q, ncell, k, p);
    } else {
        const int g = (int)(k - ncell);
        int side, along;
        if (g < M.ni) { side = 1; along = g; }
        else if (g < M.ni + M.nj) { side = 2; along = g - M.ni; }
        else if (g < 2 * M.ni + M.nj) { side = 3; along = g - M.ni - M.nj; }
        else { side = 4; along = g - 2 * M.ni - M.nj; }
        ghost_state(P, M, q, ncell, side, along, p);
    }
    out[k] = p.u;
    out[ntot + k] = p.v;
    out[2 * ntot + k] = p.t;
    out[3 * ntot + k] = p.p;
}

// ---------------------------------------------------------- post-processing

// POSTPROCESS node averages (solver_state.f90:237-281) of the [4][ncell+nghost] U,V,T,P
// array k_prim_out produced: cells in ascending id order, then the ghosts of the node
// in bc.in order, divided by their count.  Output [4][nnode] as (P, U, V, T).
__global__ void k_node_average(Mesh M, const double* __restrict__ prim, double* __restrict__ out) {
    const size_t ncell = (size_t)M.ni * M.nj, ntot = ncell + M.nghosts();
    const size_t nnode = (size_t)(M.ni + 1) * (M.nj + 1);
    const size_t n = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (n >= nnode) return;
    const int a = (int)(n / (M.nj + 1)), b = (int)(n % (M.nj + 1));
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    int cnt = 0, ng = 0;
    size_t gk[2] = {0, 0};
    int gr[2] = {0, 0};
    for (int k = 0; k < 4; k++) {
        const int pi = a - 1 + (k >> 1), pj = b - 1 + (k & 1);
        int along = 0;
        const int kind = classify(M, pi, pj, along);
        if (kind == 0) {
            const size_t c = (size_t)pi * M.nj + pj;
            s[0] += prim[3 * ntot + c]; s[1] += prim[c]; s[2] += prim[ntot + c]; s[3] += prim[2 * ntot + c];
            cnt++;
        } else if (kind > 0) {
            const int g = M.ghost_index(kind, along);
            gk[ng] = ncell + g;
            gr[ng] = M.grank[g];
            ng++;
        }
    }
    if (ng == 2 && gr[1] < gr[0]) { const size_t t = gk[0]; gk[0] = gk[1]; gk[1] = t; }
    for (int k = 0; k < ng; k++) {
        const size_t c = gk[k];
        s[0] += prim[3 * ntot + c]; s[1] += prim[c]; s[2] += prim[ntot + c]; s[3] += prim[2 * ntot + c];
        cnt++;
    }
    const double d = (double)cnt;
#pragma unroll
    for (int f = 0; f < 4; f++) out[f * nnode + n] = s[f] / d;
}

// Boundary-face sums over the ghosts whose BC type / side match (0 = any), with the face
// state (parent + ghost)/2.  mode 0: [0] sum P*SX, [1] sum P*SY, [2] sum RHO*(U*SX+V*SY),
// [3] sum |S|; mode 1: [0] sum P0*|MDOT|, [1] sum |MDOT| with the face's total pressure
// P0 = P (1 + (GAMA-1)/2 M^2)^(GAMA/(GAMA-1)), M^2 = (U^2+V^2)/(GAMA RR T), and mass flux
// MDOT = RHO (U SX + V SY).  One warp per 32 faces; one atomicAdd per warp and quantity.
__global__ void k_boundary_sums(Params P, Mesh M, const double* __restrict__ prim, int type,
                                int side, int mode, double* __restrict__ out) {
    const size_t ncell = (size_t)M.ni * M.nj, ntot = ncell + M.nghosts();
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    if (g < M.nghosts()) {
        int sd, along;
        if (g < M.ni) { sd = 1; along = g; }
        else if (g < M.ni + M.nj) { sd = 2; along = g - M.ni; }
        else if (g < 2 * M.ni + M.nj) { sd = 3; along = g - M.ni - M.nj; }
        else { sd = 4; along = g - 2 * M.ni - M.nj; }
        if ((type == 0 || M.gtype[g] == type) && (side == 0 || sd == side)) {
            int ip, jp;
            if (sd == 1) { ip = along; jp = 0; }
            else if (sd == 2) { ip = M.ni - 1; jp = along; }
            else if (sd == 3) { ip = along; jp = M.nj - 1; }
            else { ip = 0; jp = along; }
            const size_t cp = (size_t)ip * M.nj + jp, cg = ncell + g;
            const size_t n1 = (size_t)ip * (M.nj + 1) + jp;
            const double X[4] = {M.x[n1], M.x[n1 + M.nj + 1], M.x[n1 + M.nj + 2], M.x[n1 + 1]};
            const double Y[4] = {M.y[n1], M.y[n1 + M.nj + 1], M.y[n1 + M.nj + 2], M.y[n1 + 1]};
            double sx, sy;
            face_vector(P.iaxis, sd, X, Y, sx, sy);
            const double u = 0.5 * (prim[cp] + prim[cg]), vv = 0.5 * (prim[ntot + cp] + prim[ntot + cg]);
            face_sums(P, mode, u, vv, prim[2 * ntot + cp], prim[2 * ntot + cg], prim[3 * ntot + cp],
                      prim[3 * ntot + cg], sx, sy, v);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        double x = v[q];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0 && x != 0.0) atomicAdd(&out[q], x);
    }
}

// Face state (parent + ghost)/2 of every ghost in device order: out [5][nghosts] = U, V,
// P, RHO (the average of P/(RR*T) on both sides), T.
__global__ void k_face_states(Params P, Mesh M, const double* __restrict__ prim, double* __restrict__ out) {
    const size_t ncell = (size_t)M.ni * M.nj, ng = M.nghosts(), ntot = ncell + ng;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= (int)ng) return;
    int sd, along;
    if (g < M.ni) { sd = 1; along = g; }
    else if (g < M.ni + M.nj) { sd = 2; along = g - M.ni; }
    else if (g < 2 * M.ni + M.nj) { sd = 3; along = g - M.ni - M.nj; }
    else { sd = 4; along = g - 2 * M.ni - M.nj; }
    int ip, jp;
    if (sd == 1) { ip = along; jp = 0; }
    else if (sd == 2) { ip = M.ni - 1; jp = along; }
    else if (sd == 3) { ip = along; jp = M.nj - 1; }
    else { ip = 0; jp = along; }
    const size_t cp = (size_t)ip * M.nj + jp, cg = ncell + g;
    const double tp = prim[2 * ntot + cp], tgh = prim[2 * ntot + cg];
    const double pp = prim[3 * ntot + cp], pgh = prim[3 * ntot + cg];
    out[g] = 0.5 * (prim[cp] + prim[cg]);
    out[ng + g] = 0.5 * (prim[ntot + cp] + prim[ntot + cg]);
    out[2 * ng + g] = 0.5 * (pp + pgh);
    out[3 * ng + g] = 0.5 * (pp / (P.rr * tp) + pgh / (P.rr * tgh));
    out[4 * ng + g] = 0.5 * (tp + tgh);
}

void launch_face_states(const Params& P, const Mesh& M, const double* prim, double* out, cudaStream_t s) {
    k_face_states<<<(M.nghosts() + 255) / 256, 256, 0, s>>>(P, M, prim, out);
}

// ------------------------------------------------------------ batched kernels

// One launch per kernel advances every active case of a batch; block b works on tile
// tiles[b] = (case, tile j, tile i) with its case's parameters and buffers.
__global__ void __launch_bounds__(NTHREADS, TNS_PER_SM(TNS_DISS_MINB))
k_dissipation_batch(const BatchCase* __restrict__ cases, const int4* __restrict__ tiles,
                    const int* __restrict__ active) {
    const int4 t = tiles[blockIdx.x];
    if (!active[t.x]) return;  // whole block: before any barrier
    const BatchCase& c = cases[t.x];
    dissipation_tile_f64(c.P, c.M, c.diss, t.y, t.z);
}

__global__ void __launch_bounds__(NTHREADS, TNS_PER_SM(TNS_VISC_BATCH_MINB))
k_viscous_batch(const BatchCase* __restrict__ cases, const int4* __restrict__ tiles, const int* __restrict__ active) {
    const int4 t = tiles[blockIdx.x];
    if (!active[t.x]) return;
    const BatchCase& c = cases[t.x];
    viscous_tile_f64<false>(c.P, c.M, c.q, c.vis, c.stage[0][0].error, t.y, t.z);
}

__global__ void __launch_bounds__(NTHREADS, TNS_PER_SM(TNS_STAGE_BATCH_MINB))
k_stage_batch(const BatchCase* __restrict__ cases, const int4* __restrict__ tiles, const int* __restrict__ active,
              int stage, int monitor) {
    const int4 t = tiles[blockIdx.x];
    if (!active[t.x]) return;
    const BatchCase& c = cases[t.x];
#if TNS_BATCH_SMEM_ARGS
    // the case's arguments copied into shared memory (raw storage, never constructed):
    // loads from constant shared addresses instead of through the descriptor pointer
    __shared__ __align__(16) unsigned char sargs[sizeof(Params) + sizeof(Mesh) + sizeof(StageArgs)];
    Params& sP = *reinterpret_cast<Params*>(sargs);
    Mesh& sM = *reinterpret_cast<Mesh*>(sargs + sizeof(Params));
    StageArgs& sA = *reinterpret_cast<StageArgs*>(sargs + sizeof(Params) + sizeof(Mesh));
    {
        const int tid = threadIdx.y * TJ + threadIdx.x;
        copy_words(&sP, &c.P, sizeof(Params), tid);
        copy_words(&sM, &c.M, sizeof(Mesh), tid);
        copy_words(&sA, &c.stage[monitor][stage], sizeof(StageArgs), tid);
        __syncthreads();
    }
    stage_tile<false>(sP, sM, sA, t.y, t.z);
#else
    stage_tile<false>(c.P, c.M, c.stage[monitor][stage], t.y, t.z);
#endif
}

// Persistent batched iterations (schedule 3): one cooperative launch advances every
// active case by `iters` unmonitored RK4 iterations.  Its blocks walk the tile table
// phase by phase -- dissipation and viscous flux together (both read Q_old only and
// write disjoint arrays), then the four stages -- with a grid barrier between phases
// (bounded waits: a barrier that gives up sets error bit 2 and the kernel returns).  A
// block that finishes a tile synchronises before the next, whose static-block copy
// reuses the tile's shared memory and barrier; one whose copy did not arrive leaves (the
// others then give up at the grid barrier).  Cases need LOCAL=1 and no type-6 port
// (those add per-case reductions between the phases).
#ifndef TNS_PERSIST_MINB
#define TNS_PERSIST_MINB 3
#endif
__global__ void __launch_bounds__(NTHREADS, TNS_PER_SM(TNS_PERSIST_MINB))
k_batch_persistent(const BatchCase* __restrict__ cases, const int4* __restrict__ tiles,
                   const int* __restrict__ active, int ntiles, int iters, unsigned int* bar,
                   unsigned int* error) {
    for (int it = 0; it < iters; it++) {
        for (int ph = 0; ph < 5; ph++) {
            const int nwork = ph == 0 ? 2 * ntiles : ntiles;
            for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
                const int4 t = tiles[w % ntiles];
                bool ok = true;
                if (active[t.x]) {
                    const BatchCase& c = cases[t.x];
                    if (ph == 0 && w < ntiles) dissipation_tile_f64(c.P, c.M, c.diss, t.y, t.z);
                    else if (ph == 0) ok = viscous_tile_f64<false>(c.P, c.M, c.q, c.vis, c.stage[0][0].error, t.y, t.z);
                    else ok = stage_tile<false>(c.P, c.M, c.stage[0][ph - 1], t.y, t.z);
                }
                async_proxy_fence();
                if (!__syncthreads_and(ok)) return;  // the whole block
            }
            if (!grid_barrier(bar, bar + 1)) {
                if (threadIdx.x == 0 && threadIdx.y == 0) atomicOr(error, 4u);
                return;
            }
        }
    }
}

// ---------------------------------------------------------------- math check

// Evaluates one of the FP64 helpers the kernels use, elementwise, for testing their
// accuracy: fn 0 = pow06(a), 1 = tanh_ratio(a, b), 2 = expm1_nonneg(a).
__global__ void k_debug_math(int fn, long long n, const double* __restrict__ a, const double* __restrict__ b,
                             double* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = fn == 0 ? pow06(a[i]) : (fn == 1 ? tanh_ratio(a[i], b[i]) : expm1_nonneg(a[i]));
}

void launch_debug_math(int fn, long long n, const double* a, const double* b, double* out, cudaStream_t s) {
    const long long blocks = (n + 255) / 256;
    if (blocks > 0) k_debug_math<<<(unsigned)blocks, 256, 0, s>>>(fn, n, a, b, out);
}

// ------------------------------------------------------------------ launchers

static dim3 tile_grid(const Mesh& M) { return dim3((M.nj + TJ - 1) / TJ, (M.ni + TI - 1) / TI); }

// SMs of the current device, and the pipelined stage's resident blocks on all of them.
int sm_count() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 148;
    return n;
}
constexpr size_t PIPE_SMEM = sizeof(StagePipeSmem) + 128;  // (the kernel aligns its boxes to 128 bytes)
static int pipe_grid() {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_stage_pipe<0, false>, NTHREADS, PIPE_SMEM) !=
        cudaSuccess)
        return 0;
    return per_sm * sm_count();
}

// The driver's tensor-map encoder, looked up once through the runtime.
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
                cudaSuccess || q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

// Tensor map of an array [planes][NI][NJ] with boxes [planes][rows][cols]; false where TMA
// cannot address it: NJ odd (rows not a multiple of 16 bytes) or the array not 16-byte
// aligned.
static bool plane_map(const Mesh& M, const double* a, int planes, int rows, int cols, CUtensorMap* map) {
    const PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
    if (!enc || M.nj % 2 != 0 || (reinterpret_cast<uintptr_t>(a) & 15) != 0) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)M.nj, (cuuint64_t)M.ni, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {(cuuint64_t)M.nj * sizeof(double), (cuuint64_t)M.ni * M.nj * sizeof(double)};
    const cuuint32_t box[3] = {(cuuint32_t)cols, (cuuint32_t)rows, (cuuint32_t)planes};
    const cuuint32_t elem[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double*>(a), dims, strides, box, elem,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
static bool stage_maps(const Params& P, const Mesh& M, const StageArgs& A, StageMaps* m) {
    const bool first = !A.e;
    const double* e = first ? A.d : A.e;
    return plane_map(M, A.qin, 5, QH, QW, &m->q) &&
           (first ? plane_map(M, A.vis, 4, TI, TJ, &m->qold) : plane_map(M, A.qold, 5, TI, TJ, &m->qold)) &&
           plane_map(M, e, 5, TI, TJ, &m->e) && plane_map(M, P.local ? A.dt : e, 1, TI, TJ, &m->dt);
}

cudaError_t configure_kernels() {
    cudaError_t e;
    for (auto k : {k_stage<0, false>, k_stage<1, false>, k_stage<0, true>, k_stage<1, true>}) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RIM_SMEM);
        if (e != cudaSuccess) return e;
    }
    for (auto k : {k_stage_pipe<0, false>, k_stage_pipe<1, false>, k_stage_pipe<0, true>}) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PIPE_SMEM);
        if (e != cudaSuccess) return e;
    }
    for (auto k : {k_viscous<false>, k_viscous<true>}) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)visc_smem_bytes());
        if (e != cudaSuccess) return e;
    }
    e = cudaFuncSetAttribute(k_dissipation, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)diss_smem_bytes());
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_dissipation_batch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)diss_smem_bytes());
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_viscous_batch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)visc_smem_bytes());
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_batch_persistent, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)persistent_smem_bytes(false));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_stage_batch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)stage_smem_bytes());
}

size_t persistent_smem_bytes(bool mixed) {
    if (mixed) return std::max(stage_mx_smem_bytes(), std::max(visc_mx_smem_bytes(), diss_mx_smem_bytes()));
    return std::max(stage_smem_bytes(), std::max(visc_smem_bytes(), diss_smem_bytes()));
}

int persistent_grid(bool mixed, int ntiles) {
    int per_sm = 0, grid = 0;
    if (mixed) {
        persistent_kernel_mx(ntiles, &grid);
        return grid;
    }
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_persistent, NTHREADS,
                                                      persistent_smem_bytes(mixed)) != cudaSuccess)
        return 0;
    return per_sm * sm_count();
}

cudaError_t launch_persistent(bool mixed, const BatchCase* cases, const int4* tiles, const int* active,
                              int ntiles, int iters, int parity, unsigned int* bar, unsigned int* error,
                              cudaStream_t s) {
    int grid = 0;
    const void* k = mixed ? persistent_kernel_mx(ntiles, &grid) : (const void*)k_batch_persistent;
    grid = std::min(mixed ? grid : persistent_grid(false, ntiles), 2 * ntiles);
    const dim3 blk(TJ, TI);
    if (mixed) {  // (its tile table holds active cases alone)
        void* args[] = {(void*)&cases, (void*)&tiles,  (void*)&ntiles, (void*)&iters,
                        (void*)&parity, (void*)&bar, (void*)&error};
        return cudaLaunchCooperativeKernel(k, dim3(grid), blk, args, persistent_smem_bytes(true), s);
    }
    void* args[] = {(void*)&cases, (void*)&tiles, (void*)&active, (void*)&ntiles, (void*)&iters, (void*)&bar,
                    (void*)&error};
    return cudaLaunchCooperativeKernel(k, dim3(grid), blk, args, persistent_smem_bytes(false), s);
}

void launch_batch_f64(const BatchCase* cases, const int4* tiles, const int* active, int ntiles,
                      int kernel, int stage, int monitor, cudaStream_t s) {
    const dim3 blk(TJ, TI);
    if (kernel == 0)
        launch_tile(k_dissipation_batch, dim3(ntiles), blk, diss_smem_bytes(), s, cases, tiles, active);
    else if (kernel == 1)
        launch_tile(k_viscous_batch, dim3(ntiles), dim3(TJ, TI), visc_smem_bytes(), s, cases, tiles, active);
    else
        launch_tile(k_stage_batch, dim3(ntiles), blk, stage_smem_bytes(), s, cases, tiles, active, stage, monitor);
}

// A state between the caller's numbering and the device's.  The host loop it replaces took a
// cache miss a value: 98,304 cells up and down, 0.9 ms of a 3.2 ms pass.
template <bool TO_DEVICE>
__global__ void __launch_bounds__(256) k_renumber(const int* __restrict__ cell_of, const double* __restrict__ src,
                                                  double* __restrict__ dst, size_t n) {
    const size_t k = blockIdx.x * (size_t)256 + threadIdx.x;
    if (k >= n) return;
    const size_t c = (size_t)cell_of[k];
#pragma unroll
    for (int m = 0; m < 5; m++) {
        if (TO_DEVICE) dst[m * n + k] = src[m * n + c];
        else dst[m * n + c] = src[m * n + k];
    }
}

void launch_renumber(const int* cell_of, const double* src, double* dst, size_t ncell, bool to_device,
                     cudaStream_t s) {
    const unsigned grid = (unsigned)((ncell + 255) / 256);
    if (to_device) k_renumber<true><<<grid, 256, 0, s>>>(cell_of, src, dst, ncell);
    else k_renumber<false><<<grid, 256, 0, s>>>(cell_of, src, dst, ncell);
}

void launch_dissipation(const Params& P, const Mesh& M, const double* q, double* d, double* dt,
                        const double* dtmin, cudaStream_t s) {
    DissArgs<double> A{q, d, dt, dtmin};
    launch_tile(k_dissipation, tile_grid(M), dim3(TJ, TI), diss_smem_bytes(), s, P, M, A);
}

void launch_viscous(const Params& P, const Mesh& M, const double* q, double* vis, unsigned int* error,
                    cudaStream_t s, int beside) {
    const dim3 grid = tile_grid(M);
    // the rim rows shorten one tile's chain (115 x 50 nozzle: 22.8 -> 22.2 us an iteration,
    // 192 x 64: 24.2 -> 22.2) but leave room for two blocks an SM instead of three (400 x 160,
    // 250 tiles: 28.0 -> 29.9)
    if ((int)(grid.x * grid.y) + beside <= VISC_RIM_PER_SM * sm_count())
        launch_tile(k_viscous<true>, grid, dim3(TJ, TI + RIM_ROWS), visc_smem_bytes(), s, P, M, q, vis, error);
    else
        launch_tile(k_viscous<false>, grid, dim3(TJ, TI), visc_smem_bytes(), s, P, M, q, vis, error);
}

void launch_stage(const Params& P, const Mesh& M, const double* qin, const double* qold,
                  double* qout, const double* d, const double* vis, const double* dt,
                  const double* dtmin, int stage, double* e, unsigned long long* cdiff,
                  unsigned int* status, unsigned int* error, cudaStream_t s, int beside) {
    const StageArgs A{qin, qold, qout, d, vis, dt, dtmin, RK_ALPHA[stage], stage ? e : nullptr, stage ? nullptr : e,
                      cdiff, status, error};
    const dim3 grid = tile_grid(M);
    const int ntiles = grid.x * grid.y;
    StageMaps maps;
    const int pipe = (A.e || !cdiff) && ntiles > TNS_PER_SM(TNS_STAGE_MINB) * sm_count() ? pipe_grid() : 0;
    if (pipe > 0 && pipe <= ntiles && stage_maps(P, M, A, &maps)) {
        launch_tile(!A.e ? k_stage_pipe<0, true> : cdiff ? k_stage_pipe<1, false> : k_stage_pipe<0, false>, dim3(pipe),
                    dim3(TJ, TI), PIPE_SMEM, s, P, M, A, ntiles, maps);
        return;
    }
    // the rim rows while every tile has its own resident block of that size (at 8 rows a tile; for
    // other heights see tns_tile.cuh): 115 x 50 nozzle,
    // an iteration, 22.7 -> 22.2 us (20.6 with the operands fetched early); 400 x 160 ramp (250
    // tiles) 31.2 -> 28.0.  The tiles of
    // other cases in flight beside this mesh count too: their warps fill the gaps, and the
    // larger blocks would only displace them (16 ramp cases on branch streams, 20 iterations:
    // 6.05 ms with the rim rows, 5.28 without; 4 cases 1.63 and 1.50)
    if (ntiles + beside <= STAGE_RIM_PER_SM * sm_count())
        launch_tile(cdiff ? k_stage<1, true> : k_stage<0, true>, grid, dim3(TJ, TI + RIM_ROWS), RIM_SMEM, s, P, M, A);
    else
        launch_tile(cdiff ? k_stage<1, false> : k_stage<0, false>, grid, dim3(TJ, TI), stage_smem_bytes(), s, P, M, A);
}

int dtmin_blocks(const Mesh& M) {
    const long long ncell = (long long)M.ni * M.nj;
    long long b = (ncell + 255) / 256;
    return (int)(b < 1184 ? b : 1184);  // 148 SMs x 8
}

void launch_dtmin(const Params& P, const Mesh& M, const double* q, double* partial,
                  unsigned int* counter, double* dtmin, cudaStream_t s) {
    k_dtmin<<<dtmin_blocks(M), 256, 0, s>>>(P, M, q, partial, counter, dtmin);
}

void launch_gport(const Params& P, const Mesh& M, const double* q, const int* ghosts, int nport,
                  double* gport, cudaStream_t s) {
    if (nport <= 0) return;
    launch_tile(k_gport, dim3(nport), dim3(GP_THREADS), 0, s, P, M, q, ghosts, gport);
}

void launch_node_average(const Mesh& M, const double* prim, double* out, cudaStream_t s) {
    const size_t nnode = (size_t)(M.ni + 1) * (M.nj + 1);
    k_node_average<<<(unsigned)((nnode + 255) / 256), 256, 0, s>>>(M, prim, out);
}

void launch_boundary_sums(const Params& P, const Mesh& M, const double* prim, int type, int side,
                          int mode, double* out, cudaStream_t s) {
    k_boundary_sums<<<(M.nghosts() + 255) / 256, 256, 0, s>>>(P, M, prim, type, side, mode, out);
}

void launch_prim_out(const Params& P, const Mesh& M, const double* q, double* out,
                     cudaStream_t s) {
    const size_t ntot = (size_t)M.ni * M.nj + M.nghosts();
    k_prim_out<<<(unsigned)((ntot + 255) / 256), 256, 0, s>>>(P, M, q, out);
}

}  // namespace tns
