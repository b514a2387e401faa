// tns_unstructured_mx.cu -- the mixed FP32/FP64 RK stage on a general quadrilateral mesh.
//
// The general path's chunks (tns_unstructured.cu: 256 consecutive cells in Hilbert
// order and their halo) with the mixed path's arithmetic (tns_kernels_mx.cu): FP64 state
// COLD plus FP32 stage increments dQ; each chunk's slots formed in FP32 as deviations
// from a FP64 reference state, the first cell of the chunk's COLD (tns_mx.cuh); the flux
// residual in FP32 over the flux deviations plus the reference flux times the sum of the
// face vectors in FP64; source terms in FP32; D, VIS, DT stored in FP32.  Compiled, like
// tns_kernels_mx.cu, with FP32 division and square root to 2 ulp and FP32 denormals
// flushed.
#include "tns_batch.cuh"
#include "tns_handle.h"
#include "tns_mx.cuh"
#include "tns_tile.cuh"
#include "tns_umesh.h"

namespace tns {

constexpr size_t SLOTS_AT = (sizeof(TileRefMx) + 15) / 16 * 16;

// Chunk slots in shared memory (SlotsMx): (UT + hmax) of three 16-byte words and |V| - ref,
// after the chunk's reference state.
size_t u_chunk_mx_smem_bytes(const UMesh& M) {
    return SLOTS_AT + (3 * sizeof(float4) + sizeof(float)) * ((size_t)UT + M.hmax);
}

// One mixed RK stage of one chunk (source_terms.f90:24-104, residual.f90:23-83): stage
// input COLD + dQin (dQin null in stage 1); stages 1-3 write dQout, stage 4 the state qout.
// Latency bound: the halo's slot numbers load before the previous kernel has ended, the cell's
// packed geometry and local slots while the halo is formed (renumbered 256 x 96 ramp, 20
// iterations with the transfers: 1.19 -> 1.08 ms; the halo's states loaded early too cost
// registers: 1.11).
#ifndef TNS_U_CHUNK_MX_MINB
// Blocks per SM the register budget is sized for; measured on a renumbered 1024 x 384
// nozzle-plume (B200, one mixed iteration): 4 -> 0.248 ms, 3 -> 0.264 ms, 5 -> 0.257 ms.
#define TNS_U_CHUNK_MX_MINB 4
#endif
__global__ void __launch_bounds__(UT, TNS_U_CHUNK_MX_MINB) k_u_stage_chunk_mx(Params P, UMesh M, StageArgsMx A,
                                                                            const double* __restrict__ vf,
                                                                            float* vis) {
    extern __shared__ __align__(16) unsigned char usm_raw[];
    TileRefMx& R = *reinterpret_cast<TileRefMx*>(usm_raw);
    const int ns = UT + M.hmax;
    float4* slots = reinterpret_cast<float4*>(usm_raw + SLOTS_AT);
    const SlotsMx W{slots, slots + ns, slots + 2 * ns, reinterpret_cast<float*>(slots + 3 * ns)};
    const int ne = M.ne, t = threadIdx.x;
    const size_t n = (size_t)ne;
    const int c0 = blockIdx.x * UT, I = c0 + t;
    const int h0 = M.cptr[blockIdx.x], nh = M.cptr[blockIdx.x + 1] - h0;
    pdl_trigger();
    // a halo slot's cell, or the ghost's parent
    int hs = -1, hc = 0;
    auto halo = [&](int h) {
        hs = M.cslot[h0 + h];
        hc = hs < ne ? hs : M.gpar[hs - ne];
    };
    if (t < nh) halo(t);
    pdl_wait();
    auto load = [&](int c, double q[5], float d[5]) {
#pragma unroll
        for (int m = 0; m < 5; m++) q[m] = A.cold[m * n + c];
#pragma unroll
        for (int m = 0; m < 5; m++) d[m] = A.dqin ? A.dqin[m * n + c] : 0.0f;
    };
    double qo[5];
    float dqo[5];
    if (I < ne) load(I, qo, dqo);
    // the chunk's reference state: its first cell's COLD (the same in all four stages)
    if (t == 0) make_tile_ref(P, qo, R);
    __syncthreads();
    auto cell_slot = [&](int s, const double q[5], const float dq[5], SlotMx& o) {
        float d[5];
#pragma unroll
        for (int m = 0; m < 5; m++) d[m] = (float)(q[m] - R.c[m]) + dq[m];
        slot_dev_mx(P, R, d[0], d[1], d[2], d[3], d[4], o);
        W.put(s, o);
    };
    float3 own = make_float3(0.0f, 0.0f, 0.0f);
    if (I < ne) {
        SlotMx o;
        cell_slot(t, qo, dqo, o);
        own = o.own;
    }
    for (int h = t; h < nh; h += UT) {
        if (h != t) halo(h);
        double qr[5];
        float dqr[5];
        load(hc, qr, dqr);
        SlotMx o;
        if (hs < ne) {
            cell_slot(UT + h, qr, dqr, o);
            continue;
        }
        // a ghost's BC state in FP64
        auto prim = [&](const double q[5], const float dq[5], Prim& p) {
            primitive(P, q[0] + (double)dq[0], q[1] + (double)dq[1], q[2] + (double)dq[2], q[3] + (double)dq[3],
                      q[4] + (double)dq[4], p);
        };
        const int L = hs - ne, type = M.gtype[L];
        Prim pa, op, p;
        prim(qr, dqr, pa);
        if (type == 3) {
            load(M.gopp[L], qr, dqr);
            prim(qr, dqr, op);
        } else {
            op = pa;
        }
        boundary_ghost(P, type, pa, op, M.gsx[L], M.gsy[L], M.gyc[L], M.cg[UCG_YCC * ne + hc],
                       type == 6 ? M.gport[L] : 0.0, M.ginj[L], p);
        slot_ghost_mx(R, p, o);
        W.put(UT + h, o);
    }
    // the cell's geometry and local slots arrive while the halo is formed
    GeoMx G;
    int nb[4];
    if (I < ne) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int l = M.lnb[k * ne + I];
            nb[k] = l < 0 ? ~l : l;
        }
        const float4* g = reinterpret_cast<const float4*>(M.gmx) + I;
        const double* g8 = M.gmx + 8 * n + I;
        G = GeoMx{g[0], g[n], g[2 * n], g[3 * n], g8[0], g8[n], P.iaxis == 1 ? g8[2 * n] : 0.0};
    }
    __syncthreads();
    double dv[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    if (I < ne)
        stage_cell_mx(P, R, A, n, (size_t)I, W, t, nb, G, own,
                      [&](float v[4]) {
                          double s[4];
                          u_gather_faces(M, vf, I, s);
#pragma unroll
                          for (int m = 0; m < 4; m++) vis[m * n + I] = v[m] = (float)s[m];
                      }, dv);
    if (A.cdiff) stage_cdiff_mx(A, dv);
}

void launch_u_stage_chunk_mx(const Params& P, const UMesh& M, const StageArgsMx& A, const double* vf, float* vis,
                             cudaStream_t s) {
    launch_tile(k_u_stage_chunk_mx, dim3(M.nchunk), dim3(UT), u_chunk_mx_smem_bytes(M), s, P, M, A, vf, vis);
}

cudaError_t configure_u_chunk_mx(const UMesh& M) {
    return cudaFuncSetAttribute(k_u_stage_chunk_mx, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)u_chunk_mx_smem_bytes(M));
}

}  // namespace tns
