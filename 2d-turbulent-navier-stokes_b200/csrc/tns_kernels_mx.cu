// tns_kernels_mx.cu -- mixed FP32/FP64 kernels of one RK4 iteration.
//
// What stays FP64: the state Q (and every stage state COLD + dQ), each stage tile's
// reference state with its primitives and fluxes, ghost states, the viscous and
// dissipation kernels' primitives and pressures, the differences of nearly equal
// quantities there (gradient stencils, node averages, sensors, Laplacians, VOL/DT until
// each is rounded once), the part of the flux residual that cancels (the reference flux
// times the closed-contour sum of S, and VOL/YCC times the reference pressure), the sums
// of a cell's viscous face fluxes, 1/YAVG, the state accumulation and the residual
// monitor.  The geometry is computed in FP64 on the host; face vectors, gradient
// coefficients, 1/VOL, VOL and 1/YCC are rounded once from there.  What is FP32: the
// stage increments dQ, the dissipation D, the viscous flux VIS, VIS + D and DT as stored,
// the stage slots as deviations from the tile reference (primitives, fluxes and the
// source stencils), and the source / viscous arithmetic with its transcendentals
// (T**0.6, tanh, sqrt).
//
// Working with deviations instead of values keeps the FP32 rounding of the residual
// proportional to the flow's variation inside a tile rather than to the pressure and
// total-enthalpy levels, so the iteration can still converge by RTRED=1e-5 and more.
#include <algorithm>

#include "tns_device.cuh"
#include "tns_kernels.h"
#include "tns_mx.cuh"
#include "tns_tile.cuh"
#include "tns_batch.cuh"
#include "tns_diss.cuh"
#include "tns_visc.cuh"

namespace tns {

// ------------------------------------------------------------------ stage kernel

// Each thread forms its own cell's slot and keeps that cell's T, RHO and P - Pref (read for
// the cell alone) in registers; the first threads (with RIM, threads of their own) form the
// halo ring (tns_tile.cuh).
// What bounds it: issue (0.55 - 0.6 an SM quarter a cycle) and the wait of a tile's other warps
// for the three that form the ring.  A cell takes 826 instructions, 945 before its geometry was
// rounded once on the host, its slots packed into 16-byte words, each neighbour's flux met its
// face vector alone and VIS + D became one array: 384 x 1024 nozzle-plume, an iteration, 130 ->
// 116 us.  A mesh with fewer tiles than resident blocks waits for one tile's latency instead:
// extra rows of threads for the ring, with the ghosts' static records and both states asked for
// first, took 200 x 90 from 42.0 to 27.6 us and 96 x 32 from 33.4 to 25.6.  (Without RIM the
// early loads only cost registers: 200 x 66 cases of a batch 5.1 against 5.0 ms.  The static
// block read straight into registers instead of shared memory: 163 -> 175 us.)
struct StageSmemMx {
    double st[MXTILE];         // the tile's static block (tns_tile.cuh), one bulk copy
    float4 a[NSLOT], b[NSLOT], c[NSLOT];  // slots (SlotsMx)
    float q[NSLOT];
    TileRefMx ref;           // the tile's reference state (written by the dissipation kernel)
    unsigned long long bar;  // completion of the static block's copy
};

size_t stage_mx_smem_bytes() { return sizeof(StageSmemMx); }

#ifndef TNS_STAGE_MX_MINB
#define TNS_STAGE_MX_MINB 4
#endif
// the batched kernels at 4 blocks/SM as the single-case ones (the stage kernel with its
// arguments in shared memory, TNS_BATCH_SMEM_ARGS)
#ifndef TNS_STAGE_MX_BATCH_MINB
#define TNS_STAGE_MX_BATCH_MINB 4
#endif
#ifndef TNS_VISC_MX_MINB
#define TNS_VISC_MX_MINB 4  // 64 registers with small spills beat 80 registers at 3 blocks/SM
#endif
#ifndef TNS_VISC_MX_BATCH_MINB
#define TNS_VISC_MX_BATCH_MINB 4
#endif
// One stage on tile (bx, by) of a mesh; the single-case and the batched kernels wrap it.
// RIM: the block has RIM_ROWS more rows of threads, which form the halo.  LATE: the halo's places
// are looked up after the own slots (they cost registers until then).  The result: tile_copy_wait.
template <bool RIM, bool LATE = false>
__device__ __forceinline__ bool stage_mx_tile(const Params& P, const Mesh& M, const StageArgsMx& A,
                                              int bx, int by) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    StageSmemMx& S = *reinterpret_cast<StageSmemMx*>(smem_raw);
    const SlotsMx W{S.a, S.b, S.c, S.q};
    const size_t ncell = (size_t)M.ni * M.nj;
    const int j0 = bx * TJ, i0 = by * TI;
    const int tj = threadIdx.x, ti = threadIdx.y;
    const int tid = ti * TJ + tj;
    const size_t tile = (size_t)by * ((M.nj + TJ - 1) / TJ) + bx;
    pdl_trigger();
    // the static block is written by nothing: its copy overlaps the previous kernel's tail
    if (tid == 0) {
        bulk_barrier_init(&S.bar);
        bulk_copy_start(S.st, M.stile + tile * MXTILE, sizeof(double) * (P.iaxis == 1 ? MXTILE : MX_VR * NTHREADS),
                        &S.bar);
    }
    const bool inner = i0 > 0 && j0 > 0 && i0 + TI < M.ni && j0 + TJ < M.nj;
    const int i = i0 + ti, j = j0 + tj;
    const bool valid = (!RIM || ti < TI) && i < M.ni && j < M.nj;
    HaloPos h;
    h.kind = -1;
    GhostSite site{0, 0.0, 0.0, 0.0, 0.0};
    const int rt = RIM ? tid - NTHREADS : tid;  // the thread's place on the ring
    const int ri = inner ? TI : min(TI, M.ni - i0), rj = inner ? TJ : min(TJ, M.nj - j0);
    auto place = [&]() {
        if (rt >= 0 && rt < 2 * (ri + rj + 2)) {
            int li, lj;
            ring_slot(rt, ri, rj, li, lj);
            h = halo_pos(M, inner, i0, j0, li, lj);
            if (h.kind > 0) site = ghost_site(M, h.g);
        }
    };
    if (!LATE) place();
    pdl_wait();
    // a cell's COLD and stage increment
    auto load = [&](int ci, int cj, double q[5], float d[5]) {
        const size_t at = (size_t)ci * M.nj + cj;
#pragma unroll
        for (int m = 0; m < 5; m++) q[m] = A.cold[m * ncell + at];
#pragma unroll
        for (int m = 0; m < 5; m++) d[m] = A.dqin ? A.dqin[m * ncell + at] : 0.0f;
    };
    double qo[5], qr[5];
    float dqo[5], dqr[5];
    if (valid) load(i, j, qo, dqo);
    if (RIM && h.kind >= 0) load(h.ci, h.cj, qr, dqr);
    if (tid < TREF_WORDS)
        reinterpret_cast<unsigned long long*>(&S.ref)[tid] =
            reinterpret_cast<const unsigned long long*>(M.tref + tile)[tid];
    __syncthreads();
    auto cell_slot = [&](int s, const double q[5], const float dq[5], SlotMx& o) {
        float d[5];
#pragma unroll
        for (int m = 0; m < 5; m++) d[m] = (float)(q[m] - S.ref.c[m]) + dq[m];
        slot_dev_mx(P, S.ref, d[0], d[1], d[2], d[3], d[4], o);
        W.put(s, o);
    };
    float3 own = make_float3(0.0f, 0.0f, 0.0f);
    if (valid) {
        SlotMx o;
        cell_slot((ti + 1) * SW + tj + 1, qo, dqo, o);
        own = o.own;
    }
    if (LATE) place();
    if (!RIM && h.kind >= 0) load(h.ci, h.cj, qr, dqr);
    if (h.kind == 0) {
        SlotMx o;
        cell_slot(h.li * SW + h.lj, qr, dqr, o);
    } else if (h.kind > 0) {
        // a ghost's BC state in FP64
        auto prim = [&](const double q[5], const float dq[5], Prim& p) {
            primitive(P, q[0] + (double)dq[0], q[1] + (double)dq[1], q[2] + (double)dq[2], q[3] + (double)dq[3],
                      q[4] + (double)dq[4], p);
        };
        Prim par, gh;
        prim(qr, dqr, par);
        ghost_prim(P, M, site, h.g, par,
                   [&](Prim& o) {
                       load(h.ci + h.oi, h.cj + h.oj, qr, dqr);
                       prim(qr, dqr, o);
                   }, gh);
        SlotMx o;
        slot_ghost_mx(S.ref, gh, o);
        W.put(h.li * SW + h.lj, o);
    }
    const bool arrived = tile_copy_wait(&S.bar, A.error);
    double dv[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (valid) {
        const int c = (ti + 1) * SW + (tj + 1);
        const int nb[4] = {c - 1, c + SW, c + 1, c - SW};
        const float4* g = reinterpret_cast<const float4*>(S.st) + tid;
        const double* g8 = S.st + tid;
        const GeoMx G{g[0], g[NTHREADS], g[2 * NTHREADS], g[3 * NTHREADS], g8[MX_SUMX * NTHREADS],
                      g8[MX_SUMY * NTHREADS], P.iaxis == 1 ? g8[MX_VR * NTHREADS] : 0.0};
        const size_t cell = (size_t)i * M.nj + j;
        stage_cell_mx(P, S.ref, A, ncell, cell, W, c, nb, G, own,
                      [&](float v[4]) {
#pragma unroll
                          for (int m = 0; m < 4; m++) v[m] = A.vis[m * ncell + cell];
                      }, dv);
    }
    if (A.cdiff) stage_cdiff_mx(A, dv);
    return arrived;
}

// Specialised on the residual monitor, so the CDIFF reduction is compiled only where it
// runs, and on the extra rows of threads.
template <int MONITOR, bool RIM>
__global__ void __launch_bounds__(NTHREADS + (RIM ? TJ * RIM_ROWS : 0), RIM ? RIM_MINB : TNS_PER_SM(TNS_STAGE_MX_MINB))
k_stage_mx(Params P, Mesh M, StageArgsMx A) {
    StageArgsMx Ac = A;
    if (!MONITOR) Ac.cdiff = nullptr;
    stage_mx_tile<RIM>(P, M, Ac, blockIdx.x, blockIdx.y);
}

// ---------------------------------------------------------------- viscous kernel

size_t visc_mx_smem_bytes() { return sizeof(ViscSmem<float>); }
// (four blocks of the largest phase leave the persistent kernel a fifth of an SM's 228 KB as L1)
static_assert(TI != 8 || 4 * std::max(sizeof(ViscSmem<float>), sizeof(StageSmemMx)) <= 183 * 1024,
              "shared memory of a mixed tile");

// One face of viscous.f90:130-217: FP64 stencil differences, FP32 rest.
__device__ __forceinline__ void viscous_face_mx(const Params& P, const FaceVals& f, float sx, float sy, float ga,
                                                float gb, float gc, float gd, double ryavg, float out[4]) {
    const float duac = (float)(f.ua - f.uc), dubd = (float)(f.ub - f.ud);
    const float dvac = (float)(f.va - f.vc), dvbd = (float)(f.vb - f.vd);
    const float dtac = (float)(f.ta - f.tc), dtbd = (float)(f.tb - f.td);
    const float drac = (float)(f.ra - f.rc), drbd = (float)(f.rb - f.rd);
    const float DUX = duac * ga + dubd * gb, DUY = duac * gc + dubd * gd;
    const float DVX = dvac * ga + dvbd * gb, DVY = dvac * gc + dvbd * gd;
    const float DTX = dtac * ga + dtbd * gb, DTY = dtac * gc + dtbd * gd;
    const float DRX = drac * ga + drbd * gb, DRY = drac * gc + drbd * gd;
    const double vsum = f.va + f.vb + f.vc + f.vd;
    const float UAVG = (float)(QUARTER * (f.ua + f.ub + f.uc + f.ud));
    const float VAVG = (float)(QUARTER * vsum);
    const float TAVG = (float)(QUARTER * (f.ta + f.tb + f.tc + f.td));
    const float RHOAVG = (float)(QUARTER * (f.rhoa + f.rhob + f.rhoc + f.rhod));
    const float RAVG = (float)(QUARTER * (f.ra + f.rb + f.rc + f.rd));
    float DIVVEL;
    if (P.iaxis == 1) {
        const float VBYY = (ryavg == 0.0) ? DVY : (float)(QUARTER * vsum * ryavg);
        DIVVEL = DUX + DVY + VBYY;
    } else {
        DIVVEL = DUX + DVY;
    }
    const float AMU = (float)P.suth_amol * pow06f(TAVG);
    const float AK = AMU * (float)P.cp_pr;
    const float CHI = RHOAVG * RAVG / (AMU * (float)CMU);
    const float chi2 = CHI * CHI;
    const float FMU = tanh_f32((float)ALPHA_T * chi2) / tanh_f32((float)BETA_T * chi2);
    const float AMUT = RHOAVG * RAVG * FMU;
    const float AKT = AMUT * (float)P.cp_prt;
    const float AMUEFF = AMU + AMUT;
    const float AKEFF = AK + AKT;
    const float DIV23 = (float)P.div23;
    const float TXX = AMUEFF * (DUX + DUX - DIV23 * DIVVEL);
    const float TYY = AMUEFF * (DVY + DVY - DIV23 * DIVVEL);
    const float TXY = AMUEFF * (DUY + DVX);
    const float QXX = UAVG * TXX + VAVG * TXY + AKEFF * DTX;
    const float QYY = UAVG * TXY + VAVG * TYY + AKEFF * DTY;
    out[0] = TXX * sx + TXY * sy;
    out[1] = TXY * sx + TYY * sy;
    out[2] = QXX * sx + QYY * sy;
    out[3] = AMUEFF * DRX * sx + AMUEFF * DRY * sy;
}

template <bool RIM>
__device__ __forceinline__ bool viscous_mx_tile(const Params& P, const Mesh& M, const double* __restrict__ q,
                                                float* __restrict__ vis, unsigned int* error, int bx, int by) {
    return viscous_tile<RIM, float>(P, M, q, vis, error, bx, by,
                                    [&](const FaceVals& f, float sx, float sy, float ga, float gb, float gc, float gd,
                                        double ry, float out[4]) {
                                        viscous_face_mx(P, f, sx, sy, ga, gb, gc, gd, ry, out);
                                    });
}

template <bool RIM>
__global__ void __launch_bounds__(NTHREADS + (RIM ? TJ * RIM_ROWS : 0), RIM ? RIM_MINB : TNS_PER_SM(TNS_VISC_MX_MINB))
k_viscous_mx(Params P, Mesh M, const double* __restrict__ q, float* __restrict__ vis, unsigned int* error) {
    viscous_mx_tile<RIM>(P, M, q, vis, error, blockIdx.x, blockIdx.y);
}

// ------------------------------------------------------------ dissipation kernel

size_t diss_mx_smem_bytes() { return sizeof(DissSmem<float>); }

__device__ __forceinline__ void dissipation_mx_tile(const Params& P, const Mesh& M, const double* __restrict__ q,
                                                    float* __restrict__ dout, float* __restrict__ dtout,
                                                    const double* __restrict__ dtmin, int bx, int by) {
    // with the tile's reference state for this iteration's stages
    dissipation_tile(P, M, DissArgs<float>{q, dout, dtout, dtmin}, bx, by, [&](const double* c) {
        make_tile_ref(P, c, M.tref[(size_t)by * ((M.nj + TJ - 1) / TJ) + bx]);
    });
}

__global__ void __launch_bounds__(NTHREADS, TNS_PER_SM(TNS_DISS_MX_MINB))
k_dissipation_mx(Params P, Mesh M, const double* __restrict__ q, float* __restrict__ dout, float* __restrict__ dtout,
                 const double* __restrict__ dtmin) {
    dissipation_mx_tile(P, M, q, dout, dtout, dtmin, blockIdx.x, blockIdx.y);
}

// ------------------------------------------------------------ port mass flux

__global__ void __launch_bounds__(GP_THREADS) k_gport_mx(Params P, Mesh M, const double* __restrict__ cold,
                                                         const float* __restrict__ dq, const int* ghosts,
                                                         double* gport) {
    port_line(M, StateMixed{cold, dq, (size_t)M.ni * M.nj}, ghosts, gport);
}

// ------------------------------------------------------ primitive output

__global__ void k_prim_out_mx(Params P, Mesh M, const double* __restrict__ cold,
                              const float* __restrict__ dq, double* out) {
    const size_t ncell = (size_t)M.ni * M.nj;
    const size_t ng = M.nghosts(), ntot = ncell + ng;
    const size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (k >= ntot) return;
    const StateMixed st{cold, dq, ncell};
    Prim p;
    if (k < ncell) {
        cell_prim(P, st, k, p);
    } else {
        const int g = (int)(k - ncell);
        int side, along;
        if (g < M.ni) { side = 1; along = g; }
        else if (g < M.ni + M.nj) { side = 2; along = g - M.ni; }
        else if (g < 2 * M.ni + M.nj) { side = 3; along = g - M.ni - M.nj; }
        else { side = 4; along = g - 2 * M.ni - M.nj; }
        ghost_state(P, M, st, side, along, p);
    }
    out[k] = p.u;
    out[ntot + k] = p.v;
    out[2 * ntot + k] = p.t;
    out[3 * ntot + k] = p.p;
}

// ------------------------------------------------------------ batched kernels

// Mixed-path batch: `parity` selects which of qa / qa2 holds each active case's state
// (all active cases advance together, so they share it).
__global__ void __launch_bounds__(NTHREADS, TNS_PER_SM(TNS_DISS_MX_MINB))
k_dissipation_mx_batch(const BatchCase* __restrict__ cases, const int4* __restrict__ tiles,
                       const int* __restrict__ active, int parity) {
    const int4 t = tiles[blockIdx.x];
    if (!active[t.x]) return;  // whole block: before any barrier
    const BatchCase& c = cases[t.x];
    dissipation_mx_tile(c.P, c.M, c.qmx[parity], c.df, c.dtf, c.dtmin, t.y, t.z);
}

__global__ void __launch_bounds__(NTHREADS, TNS_PER_SM(TNS_VISC_MX_BATCH_MINB))
k_viscous_mx_batch(const BatchCase* __restrict__ cases, const int4* __restrict__ tiles,
                   const int* __restrict__ active, int parity) {
    const int4 t = tiles[blockIdx.x];
    if (!active[t.x]) return;
    const BatchCase& c = cases[t.x];
    viscous_mx_tile<false>(c.P, c.M, c.qmx[parity], c.visf, c.stage_mx[0][0][0].error, t.y, t.z);
}

// A stage on a tile of a batch's case, its arguments in shared memory: constant-address loads
// instead of loads through a descriptor pointer held in registers.
__device__ __forceinline__ bool stage_mx_batch_tile(const BatchCase& c, const StageArgsMx& args, int bx, int by) {
#if TNS_BATCH_SMEM_ARGS
    // (raw storage: the structs are copied in, never constructed)
    __shared__ __align__(16) unsigned char sargs[sizeof(Params) + sizeof(Mesh) + sizeof(StageArgsMx)];
    Params& sP = *reinterpret_cast<Params*>(sargs);
    Mesh& sM = *reinterpret_cast<Mesh*>(sargs + sizeof(Params));
    StageArgsMx& sA = *reinterpret_cast<StageArgsMx*>(sargs + sizeof(Params) + sizeof(Mesh));
    const int tid = threadIdx.y * TJ + threadIdx.x;
    copy_words(&sP, &c.P, sizeof(Params), tid);
    copy_words(&sM, &c.M, sizeof(Mesh), tid);
    copy_words(&sA, &args, sizeof(StageArgsMx), tid);
    __syncthreads();
    return stage_mx_tile<false>(sP, sM, sA, bx, by);
#else
    return stage_mx_tile<false>(c.P, c.M, args, bx, by);
#endif
}

__global__ void __launch_bounds__(NTHREADS, TNS_PER_SM(TNS_STAGE_MX_BATCH_MINB))
k_stage_mx_batch(const BatchCase* __restrict__ cases, const int4* __restrict__ tiles, const int* __restrict__ active,
                 int parity, int stage, int monitor) {
    const int4 t = tiles[blockIdx.x];
    if (!active[t.x]) return;
    const BatchCase& c = cases[t.x];
    stage_mx_batch_tile(c, c.stage_mx[parity][monitor][stage], t.y, t.z);
}

// Persistent batched iterations of the mixed path (schedule 3), as k_batch_persistent:
// the state parity alternates from `parity` with every iteration.  A case's arguments stay in
// shared memory until a tile of another case comes.  The two pre-passes of a tile follow one
// another in one block, which finds the state in L1, where every block gets a tile that way.
// Two register budgets, PER_SM blocks of eight rows an SM: a tile's chain is shorter with 80
// registers, and with 64 more tiles are under way; the launcher takes the first where it needs no
// more rounds over the tiles (692 tiles, 20 iterations: 2.36 -> 1.93 ms; 9500 tiles, which it takes
// at 64, 19.2 with 64 and 20.8 with 80).  Arguments copied for every stage tile, and all
// dissipation tiles before the first viscous one: 1.34 ms for 1 case of 224 tiles, 19.4 for 64
// cases; now 1.15 and 18.5.
template <int PER_SM>
__global__ void __launch_bounds__(NTHREADS, TNS_PER_SM(PER_SM))
k_batch_persistent_mx(const BatchCase* __restrict__ cases, const int4* __restrict__ tiles, int ntiles, int iters,
                      int parity0, unsigned int* bar, unsigned int* error) {
    // (raw storage: the structs are copied in, never constructed)
    __shared__ __align__(16) unsigned char sargs[sizeof(Params) + sizeof(Mesh) + sizeof(StageArgsMx)];
    Params& sP = *reinterpret_cast<Params*>(sargs);
    Mesh& sM = *reinterpret_cast<Mesh*>(sargs + sizeof(Params));
    StageArgsMx& sA = *reinterpret_cast<StageArgsMx*>(sargs + sizeof(Params) + sizeof(Mesh));
    const bool pairs = ntiles >= (int)gridDim.x;
    int held = -1;  // the case whose Params and Mesh are in shared memory
    for (int it = 0; it < iters; it++) {
        const int parity = parity0 ^ (it & 1);
        for (int ph = 0; ph < 5; ph++) {
            // pre-passes (ph 0): dissipation of tile k is item 2 k, its viscous flux 2 k + 1, taken
            // in pairs, or apart (the viscous tiles then go to other blocks than the dissipation's)
            const bool two = ph == 0 && pairs;
            const int nwork = ph == 0 ? 2 * ntiles : ntiles;
            int args = -1;  // the case whose stage arguments are
            for (int w = two ? 2 * blockIdx.x : blockIdx.x; w < nwork;
                 w += !two ? gridDim.x : w & 1 ? 2 * gridDim.x - 1 : 1) {
                const int4 t = tiles[two ? w >> 1 : w < ntiles ? w : w - ntiles];
                const BatchCase& c = cases[t.x];
                if (t.x != args) {
                    const int tid = threadIdx.y * TJ + threadIdx.x;
                    if (t.x != held) {
                        copy_words(&sP, &c.P, sizeof(Params), tid);
                        copy_words(&sM, &c.M, sizeof(Mesh), tid);
                        held = t.x;
                    }
                    if (ph) copy_words(&sA, &c.stage_mx[parity][0][ph - 1], sizeof(StageArgsMx), tid);
                    args = t.x;
                    __syncthreads();
                }
                bool ok = true;
                if (ph)
                    ok = stage_mx_tile<false, true>(sP, sM, sA, t.y, t.z);
                else if (two ? w & 1 : w >= ntiles)
                    ok = viscous_mx_tile<false>(sP, sM, c.qmx[parity], c.visf, c.stage_mx[0][0][0].error, t.y, t.z);
                else
                    dissipation_mx_tile(sP, sM, c.qmx[parity], c.df, c.dtf, c.dtmin, t.y, t.z);
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

// The kernel for a batch of ntiles tiles, and its resident blocks on the device (0: none).
const void* persistent_kernel_mx(int ntiles, int* grid) {
    const void* k[2] = {(const void*)k_batch_persistent_mx<3>, (const void*)k_batch_persistent_mx<4>};
    int g[2];
    for (int v = 0; v < 2; v++) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k[v], NTHREADS, persistent_smem_bytes(true)) !=
            cudaSuccess)
            per_sm = 0;
        g[v] = per_sm * sm_count();
    }
    const int v = g[0] > 0 && (g[1] <= 0 || (ntiles + g[0] - 1) / g[0] <= (ntiles + g[1] - 1) / g[1]) ? 0 : 1;
    *grid = g[v];
    return k[v];
}

// ------------------------------------------------------------------ launchers

static dim3 tile_grid_mx(const Mesh& M) { return dim3((M.nj + TJ - 1) / TJ, (M.ni + TI - 1) / TI); }

cudaError_t configure_kernels_mx() {
    cudaError_t e;
    for (auto k : {k_stage_mx<0, false>, k_stage_mx<1, false>, k_stage_mx<0, true>, k_stage_mx<1, true>}) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)stage_mx_smem_bytes());
        if (e != cudaSuccess) return e;
    }
    e = cudaFuncSetAttribute(k_dissipation_mx, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)diss_mx_smem_bytes());
    if (e != cudaSuccess) return e;
    for (auto k : {k_viscous_mx<false>, k_viscous_mx<true>}) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)visc_mx_smem_bytes());
        if (e != cudaSuccess) return e;
    }
    e = cudaFuncSetAttribute(k_dissipation_mx_batch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)diss_mx_smem_bytes());
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_viscous_mx_batch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)visc_mx_smem_bytes());
    if (e != cudaSuccess) return e;
    for (auto k : {k_batch_persistent_mx<3>, k_batch_persistent_mx<4>}) {
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)persistent_smem_bytes(true));
        if (e != cudaSuccess) return e;
    }
    return cudaFuncSetAttribute(k_stage_mx_batch, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)stage_mx_smem_bytes());
}

void launch_batch_mx(const BatchCase* cases, const int4* tiles, const int* active, int ntiles,
                     int kernel, int parity, int stage, int monitor, cudaStream_t s) {
    const dim3 blk(TJ, TI);
    if (kernel == 0)
        launch_tile(k_dissipation_mx_batch, dim3(ntiles), blk, diss_mx_smem_bytes(), s, cases, tiles, active, parity);
    else if (kernel == 1)
        launch_tile(k_viscous_mx_batch, dim3(ntiles), dim3(TJ, TI), visc_mx_smem_bytes(), s, cases, tiles, active,
                    parity);
    else
        launch_tile(k_stage_mx_batch, dim3(ntiles), blk, stage_mx_smem_bytes(), s, cases, tiles, active, parity, stage,
                    monitor);
}

void launch_dissipation_mx(const Params& P, const Mesh& M, const double* q, float* d, float* dt,
                            const double* dtmin, cudaStream_t s) {
    launch_tile(k_dissipation_mx, tile_grid_mx(M), dim3(TJ, TI), diss_mx_smem_bytes(), s, P, M, q, d, dt, dtmin);
}

void launch_viscous_mx(const Params& P, const Mesh& M, const double* q, float* vis, unsigned int* error,
                       cudaStream_t s, int beside) {
    const dim3 grid = tile_grid_mx(M);
    // the rim rows by the FP64 kernel's rule
    if ((int)(grid.x * grid.y) + beside <= VISC_RIM_PER_SM * sm_count())
        launch_tile(k_viscous_mx<true>, grid, dim3(TJ, TI + RIM_ROWS), visc_mx_smem_bytes(), s, P, M, q, vis, error);
    else
        launch_tile(k_viscous_mx<false>, grid, dim3(TJ, TI), visc_mx_smem_bytes(), s, P, M, q, vis, error);
}

void launch_stage_mx(const Params& P, const Mesh& M, const double* cold, const float* dqin,
                     float* dqout, double* qout, const float* d, const float* vis, float* e, const float* dt,
                     const double* dtmin, double alpha, unsigned long long* cdiff,
                     unsigned int* status, unsigned int* error, cudaStream_t s, int beside) {
    const StageArgsMx A{cold, dqin, dqout, qout, d, vis, dt, dtmin, (float)alpha, dqin ? e : nullptr,
                        dqin ? nullptr : e, cdiff, status, error};
    const dim3 grid = tile_grid_mx(M);
    // the rim rows by the FP64 stage's rule, which here follows the tile height (tns_tile.cuh)
    if ((int)(grid.x * grid.y) + beside <= STAGE_MX_RIM_PER_SM * sm_count())
        launch_tile(cdiff ? k_stage_mx<1, true> : k_stage_mx<0, true>, grid, dim3(TJ, TI + RIM_ROWS),
                    stage_mx_smem_bytes(), s, P, M, A);
    else
        launch_tile(cdiff ? k_stage_mx<1, false> : k_stage_mx<0, false>, grid, dim3(TJ, TI), stage_mx_smem_bytes(), s,
                    P, M, A);
}

void launch_gport_mx(const Params& P, const Mesh& M, const double* cold, const float* dq,
                     const int* ghosts, int nport, double* gport, cudaStream_t s) {
    if (nport <= 0) return;
    launch_tile(k_gport_mx, dim3(nport), dim3(GP_THREADS), 0, s, P, M, cold, dq, ghosts, gport);
}

void launch_prim_out_mx(const Params& P, const Mesh& M, const double* cold, const float* dq,
                        double* out, cudaStream_t s) {
    const size_t ntot = (size_t)M.ni * M.nj + M.nghosts();
    k_prim_out_mx<<<(unsigned)((ntot + 255) / 256), 256, 0, s>>>(P, M, cold, dq, out);
}

}  // namespace tns
