// tns_tile.cuh -- tile geometry and the helpers every tile kernel shares: bulk copies,
// programmatic dependent launch, halo classification, primitive variables of a cell, and the
// ghost state of a halo position (BC of boundary.f90:24-327 from the parent and its opposite
// neighbour).
#pragma once

#include <utility>

#include <cuda.h>

#include "tns_device.cuh"

namespace tns {

#ifndef TNS_TI
#define TNS_TI 8
#endif
#ifndef TNS_STAGE_MINB
#define TNS_STAGE_MINB 3
#endif
#ifndef TNS_STAGE_BATCH_MINB
#define TNS_STAGE_BATCH_MINB 3  // with its arguments in shared memory (tns_batch.cuh)
#endif
#ifndef TNS_VISC_MINB
#define TNS_VISC_MINB 3  // 80 registers: 3 blocks/SM beat 2 blocks without the cap
#endif
#ifndef TNS_STAGE_RIM_PER_SM
#define TNS_STAGE_RIM_PER_SM 2
#endif
#ifndef TNS_VISC_RIM_PER_SM
#define TNS_VISC_RIM_PER_SM 1
#endif
#ifndef TNS_VISC_BATCH_MINB
#define TNS_VISC_BATCH_MINB 1  // descriptor-fed arguments spill at 3 blocks/SM
#endif
#ifndef TNS_DISS_MINB
#define TNS_DISS_MINB 4
#endif
#ifndef TNS_DISS_MX_MINB
#define TNS_DISS_MX_MINB 4
#endif
// Resident blocks per SM of a kernel tuned at TI = 8, for the compiled TI: the same
// threads per SM at every tile height.
#define TNS_PER_SM(n) ((n) * 8 / TNS_TI > 0 ? (n) * 8 / TNS_TI : 1)
constexpr int TJ = 32;      // tile extent along j (contiguous in memory)
constexpr int GP_THREADS = 128;  // threads per port line of the type-6 port-flux kernels
constexpr int TI = TNS_TI;  // tile extent along i
constexpr int NTHREADS = TJ * TI;
// Tiles an SM, in all meshes in flight, up to which the stage and viscous kernels take blocks with
// extra rows of threads for a tile's rim (RIM_ROWS), at 8 rows a tile see launch_stage and
// launch_viscous.  The mixed stage's line moves with the tile height, as its blocks' residency
// does (16 rows, 200 tiles: 44.1 us an iteration with the extra rows, 38.5 without; 4 rows, 560
// tiles: 28.3 with, 31.6 without).  The others' does not: the FP64 stage's early operands outweigh
// a second round of blocks (16 rows, 200 tiles: 48.4 with, 50.8 without), and the viscous blocks
// soon lack shared memory (4 rows, 280 tiles: 31.5 with, 27.2 without).
constexpr int STAGE_RIM_PER_SM = TNS_STAGE_RIM_PER_SM;
constexpr int STAGE_MX_RIM_PER_SM = TNS_PER_SM(TNS_STAGE_RIM_PER_SM);
constexpr int VISC_RIM_PER_SM = TNS_VISC_RIM_PER_SM;
constexpr int RIM_MINB = TNS_PER_SM(2);  // resident blocks an SM the register budget of such a kernel is for
// Halo-1 slot grid (TI+2) x (TJ+2).
constexpr int SW = TJ + 2;
constexpr int NSLOT = (TI + 2) * SW;
// The halo ring of the slot grid, 2 (TI + 2) + 2 TJ + 4 positions as ring slots r:
// position (li, lj) of r runs along the first and last slot rows, then along the first
// and last slot columns between them.
constexpr int NRING = 2 * SW + 2 * TI;
__device__ __forceinline__ void ring_slot(int r, int& li, int& lj) {
    if (r < SW) { li = 0; lj = r; }
    else if (r < 2 * SW) { li = TI + 1; lj = r - SW; }
    else if (r < 2 * SW + TI) { li = 1 + r - 2 * SW; lj = 0; }
    else { li = 1 + r - 2 * SW - TI; lj = SW - 1; }
}
// The same around the first ri x rj cells of a tile that the mesh's edge cuts short,
// 2 (ri + rj + 2) positions.
__device__ __forceinline__ void ring_slot(int r, int ri, int rj, int& li, int& lj) {
    const int w = rj + 2;
    if (r < w) { li = 0; lj = r; }
    else if (r < 2 * w) { li = ri + 1; lj = r - w; }
    else if (r < 2 * w + ri) { li = 1 + r - 2 * w; lj = 0; }
    else { li = 1 + r - 2 * w - ri; lj = w - 1; }
}
// Rows of threads a block can have on top of one per cell: they take the halo ring (and the
// other work a tile has on its rim) while the cells' threads evaluate their own.
constexpr int RIM_ROWS = (NRING + TJ - 1) / TJ;
constexpr int AW = TJ + 1;  // node-average grid (TI+1) x (TJ+1)
constexpr int NAVG = (TI + 1) * AW;

// Static block of one stage tile (tile (bx, by) at M.stile + (by * ntiles_j + bx) * STILE),
// built on the host: the nodes of the tile's cells, (i0..i0+TI) x (j0..j0+TJ), x then y
// (index la * SNW + lb), then per cell (index ti * TJ + tj) the source-gradient
// coefficients GA..GD, 1/VOL and 1/YCC (see source_terms).  Positions outside the mesh
// hold zeros.  A multiple of 16 bytes, so a tile's block is one bulk copy.
constexpr int SNW = TJ + 1;
constexpr int SNN = (TI + 1) * SNW;
enum StageTileField { ST_GA, ST_GB, ST_GC, ST_GD, ST_RVOL, ST_RYCC, ST_NF };
constexpr int STILE = 2 * SNN + ST_NF * TI * TJ;
static_assert(STILE % 2 == 0, "a stage tile block must be a multiple of 16 bytes");

// The mixed stage's static block of a tile instead (MXTILE doubles a tile): per cell (index
// ti * TJ + tj) the four 16-byte FP32 words of GeoMx (tns_mx.cuh), a plane each, then the
// FP64 sums of the face vectors and VOL/YCC; a plane mesh leaves the last one out of the copy.
enum MixedTilePlane { MX_SUMX = 8, MX_SUMY, MX_VR, MX_N };  // in planes of doubles
constexpr int MXTILE = MX_N * TI * TJ;

// Faces of a tile: i-faces (between cells (i-1, j) and (i, j)) for i in i0..i0+TI, j-faces
// (between (i, j-1) and (i, j)) for j in j0..j0+TJ; and the tile's static face geometry
// (tile (bx, by) at M.vtile + (by * ntiles_j + bx) * VTILE), [FG_N][NVF], i-face (la, lb) at
// la * TJ + lb, j-face (la, lb) at NIF + la * (TJ + 1) + lb.  On mixed-precision handles (VTILE_MX
// doubles a tile) the face vectors and gradient coefficients are floats, rounded on the host as
// the kernel would at their use, and the last row, 1/YAVG, doubles.
constexpr int NIF = (TI + 1) * TJ;
constexpr int NJF = TI * (TJ + 1);
constexpr int NVF = NIF + NJF;
constexpr int VTILE = FG_N * NVF;
constexpr int VTILE_MX = FG_RYAVG * NVF / 2 + NVF;
static_assert(NVF % 4 == 0, "rows of the face geometry are multiples of 16 bytes");

// Programmatic dependent launch: a tile kernel lets the next kernel in the stream start
// as soon as all its blocks are running (pdl_trigger), and waits for the previous one
// to finish, with its memory visible, before it touches data that kernel produced
// (pdl_wait).  Static data, which nothing writes, may load before the wait.  Both are
// no-ops when the kernel was not launched with the attribute.
#ifndef TNS_PDL
#define TNS_PDL 1
#endif
__device__ __forceinline__ void pdl_trigger() {
#if TNS_PDL
    asm volatile("griddepcontrol.launch_dependents;");
#endif
}
__device__ __forceinline__ void pdl_wait() {
#if TNS_PDL
    asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
}

// One-shot bulk copy global -> shared through the TMA engine, completed on an mbarrier
// (cp.async.bulk with mbarrier::complete_tx).  Both addresses 16-byte aligned, bytes a
// multiple of 16.  bulk_copy_start: one thread, after it initialised the barrier
// (bulk_barrier_init); the block's other threads may wait on it after a __syncthreads.
__device__ __forceinline__ void bulk_barrier_init(unsigned long long* bar) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(a) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // without this fence the copy engine may complete a copy on a barrier it does not see
    // initialised yet, and the wait never ends
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// Its shared memory is ordinary memory again.  One thread, when no thread and no copy uses the
// barrier any more.
__device__ __forceinline__ void bulk_barrier_end(unsigned long long* bar) {
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"((unsigned)__cvta_generic_to_shared(bar)) : "memory");
}
// Per-thread copies of 4 or 8 bytes global -> shared that need no registers on the way; the
// thread that issued them waits for all of its own (copies_wait).
template <class T>
__device__ __forceinline__ void copy_async(T* dst, const T* src) {
    static_assert(sizeof(T) == 4 || sizeof(T) == 8, "sizes cp.async takes");
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"((int)sizeof(T)) : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// barrier_expect: the phase completes when `bytes` of copies have arrived.
__device__ __forceinline__ void barrier_expect(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;"
                 ::"r"((unsigned)__cvta_generic_to_shared(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
    const unsigned b = (unsigned)__cvta_generic_to_shared(bar);
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(d), "l"(src), "r"(bytes), "r"(b) : "memory");
}
__device__ __forceinline__ void bulk_copy_start(void* dst, const void* src, unsigned bytes,
                                                unsigned long long* bar) {
    barrier_expect(bar, bytes);
    bulk_copy(dst, src, bytes, bar);
}
// Tiled tensor copy global -> shared (cp.async.bulk.tensor, 3-D, no multicast): the box of
// `map` at element coordinates (x, y, z), x the innermost; x * element size a multiple of 16
// bytes; the shared destination 128-byte aligned; out-of-range elements arrive as zeros and
// count.  `map` is the address of a __grid_constant__ kernel parameter.
__device__ __forceinline__ void tensor_copy_3d(void* dst, const CUtensorMap* map, int x, int y, int z,
                                               unsigned long long* bar) {
    const unsigned b = (unsigned)__cvta_generic_to_shared(bar);
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(d), "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(b)
                 : "memory");
}
// Waits for the barrier's phase of the given parity with a bounded number of polls; false if
// the copy did not complete in that many (the caller reports it and skips the tile).
__device__ __forceinline__ bool bulk_wait(unsigned long long* bar, unsigned parity = 0, int max_polls = 1 << 20) {
    const unsigned b = (unsigned)__cvta_generic_to_shared(bar);
    for (int k = 0; k < max_polls; k++) {
        unsigned done;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(b), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

// A tile's wait for its static copy, and the block barrier its threads need there anyway.  Each
// thread counts its own polls, so around the limit some see the copy and some do not.  None
// leaves by itself (it would miss the block's later barriers, and in a kernel that loops over
// tiles run one barrier ahead of the others into the next tile's buffers): a thread that gives up
// reports it (bit 1 of *error, which ends the run with an error), gives the copy, which writes this
// block's shared memory, one more bounded wait, and goes through the tile with what is there --
// geometry, no indices.  The result says whether the copy arrived; a kernel that loops over tiles
// votes on it before the next.  After the barrier no thread looks at the copy's barrier any more
// and it is taken down: such a kernel writes other data over its place and sets one up there
// again, neither of which a live barrier allows.  (A vote in place of this barrier cost 1 % of an
// iteration on small meshes.)
__device__ __forceinline__ bool tile_copy_wait(unsigned long long* bar, unsigned int* error) {
    bool arrived = bulk_wait(bar);
    if (!arrived) {
        atomicOr(error, 2u);
        arrived = bulk_wait(bar);
    }
    __syncthreads();
    if (arrived && threadIdx.x == 0 && threadIdx.y == 0) bulk_barrier_end(bar);
    return arrived;
}

// Orders this thread's shared-memory accesses before later bulk copies into them (issued after
// a block barrier), for kernels whose tiles reuse one buffer.
__device__ __forceinline__ void async_proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Grid-wide barrier of a cooperative launch (every block resident): an arrival counter
// and a generation word in global memory, both zero before the launch.  The last block
// to arrive resets the counter and advances the generation; the others poll the
// generation at most max_polls times.  Returns false when the wait gave up (the caller
// reports it and leaves the kernel).
__device__ __forceinline__ bool grid_barrier(unsigned int* count, unsigned int* gen, int max_polls = 1 << 22) {
    __shared__ int passed;
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        const unsigned int g = *(volatile unsigned int*)gen;
        __threadfence();
        const unsigned int nb = gridDim.x * gridDim.y;
        if (atomicAdd(count, 1u) == nb - 1) {
            atomicExch(count, 0u);
            __threadfence();
            atomicAdd(gen, 1u);
            passed = 1;
        } else {
            int k = 0;
            while (*(volatile unsigned int*)gen == g && k < max_polls) {
                __nanosleep(64);
                k++;
            }
            passed = *(volatile unsigned int*)gen != g;
        }
        __threadfence();
    }
    __syncthreads();
    return passed != 0;
}

// Launch of a tile kernel that may overlap its predecessor's tail (see pdl_wait).
template <class... Exp, class... Act>
inline cudaError_t launch_tile(void (*kernel)(Exp...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                               Act&&... args) {
#if TNS_PDL
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Act>(args)...);
#else
    kernel<<<grid, block, smem, s>>>(std::forward<Act>(args)...);
    return cudaGetLastError();
#endif
}

// How a kernel reads the conservative state of cell c: FP64 array, or FP64 COLD plus an
// FP32 stage increment (the mixed-precision path).
struct StateF64 {
    const double* __restrict__ q;
    size_t n;
    __device__ __forceinline__ double c(int m, size_t cell) const { return q[m * n + cell]; }
};
struct StateMixed {
    const double* __restrict__ cold;
    const float* __restrict__ dq;  // null in stage 1 (state = COLD)
    size_t n;
    __device__ __forceinline__ double c(int m, size_t cell) const {
        const double v = cold[m * n + cell];
        return dq ? v + (double)dq[m * n + cell] : v;
    }
};

template <class St>
__device__ __forceinline__ void cell_prim(const Params& P, const St& st, size_t c, Prim& p) {
    primitive(P, st.c(0, c), st.c(1, c), st.c(2, c), st.c(3, c), st.c(4, c), p);
}

__device__ __forceinline__ void cell_prim(const Params& P, const double* __restrict__ q, size_t ncell,
                                          size_t c, Prim& p) {
    cell_prim(P, StateF64{q, ncell}, c, p);
}

// Classifies halo position (i, j): 0 = cell, 1..4 = ghost on that side, -1 = unused.
__device__ __forceinline__ int classify(const Mesh& M, int i, int j, int& along) {
    const bool in_i = i >= 0 && i < M.ni, in_j = j >= 0 && j < M.nj;
    if (in_i && in_j) return 0;
    if (in_i && j == -1) { along = i; return 1; }
    if (in_j && i == M.ni) { along = j; return 2; }
    if (in_i && j == M.nj) { along = i; return 3; }
    if (in_j && i == -1) { along = j; return 4; }
    return -1;
}

// The boundary code of node (a, b), 0 inside the mesh (see Mesh::bnode).
__device__ __forceinline__ int node_code(const Mesh& M, int a, int b) {
    if (b == 0 && a <= M.ni) return M.bnode[a];
    if (b == M.nj && a <= M.ni) return M.bnode[M.ni + 1 + a];
    if (a == 0 && b < M.nj) return M.bnode[2 * (M.ni + 1) + b];
    if (a == M.ni && b < M.nj) return M.bnode[2 * (M.ni + 1) + M.nj + 1 + b];
    return 0;
}

// What a ghost's state depends on besides its parent: its BC type and static geometry
// (written by nothing while kernels run), loaded ahead of the states.
struct GhostSite {
    int type;
    double psx, psy, ycg, ycp;
};
__device__ __forceinline__ GhostSite ghost_site(const Mesh& M, int g) {
    const GhostRec r = M.grec[g];
    return GhostSite{M.gtype[g], r.psx, r.psy, r.ycg, r.ycp};
}

// A halo position (li, lj) of a tile: what is there (classify), for a ghost its index, and
// the cell its state comes from: the cell itself or the ghost's parent, whose neighbour
// opposite the ghost is at (ci + oi, cj + oj).
struct HaloPos {
    int li, lj, kind, g, ci, cj, oi, oj;
};
__device__ __forceinline__ HaloPos halo_pos(const Mesh& M, bool inner, int i0, int j0, int li, int lj) {
    HaloPos h{li, lj, 0, 0, i0 - 1 + li, j0 - 1 + lj, 0, 0};
    if (inner) return h;
    int along = 0;
    h.kind = classify(M, h.ci, h.cj, along);
    if (h.kind > 0) {
        h.g = M.ghost_index(h.kind, along);
        h.oi = h.kind == 2 ? -1 : h.kind == 4 ? 1 : 0;
        h.oj = h.kind == 3 ? -1 : h.kind == 1 ? 1 : 0;
        h.ci += h.oi;  // the parent lies where the opposite neighbour is seen from the ghost
        h.cj += h.oj;
    }
    return h;
}

// BC state of a ghost from its parent's primitives; opp(Prim&) gives those of the parent's
// opposite neighbour (type 3 alone reads them).
template <class Opp>
__device__ __forceinline__ void ghost_prim(const Params& P, const Mesh& M, const GhostSite& s, int g, const Prim& par,
                                           Opp opp, Prim& gh) {
    Prim o = par;
    if (s.type == 3) opp(o);
    double gport = 0.0, inj = 1.0;
    if (s.type == 6) {
        gport = M.gport[g];
        inj = M.ginj[g];
    }
    boundary_ghost(P, s.type, par, o, s.psx, s.psy, s.ycg, s.ycp, gport, inj, gh);
}

// The same, with both cells read from the state `st`.
template <class St>
__device__ __forceinline__ void ghost_state(const Params& P, const Mesh& M, const St& st, int side, int along,
                                            Prim& gh) {
    const int g = M.ghost_index(side, along);
    const GhostSite s = ghost_site(M, g);
    const int ip = side == 2 ? M.ni - 1 : side == 4 ? 0 : along, jp = side == 1 ? 0 : side == 3 ? M.nj - 1 : along;
    const int oi = side == 2 ? -1 : side == 4 ? 1 : 0, oj = side == 3 ? -1 : side == 1 ? 1 : 0;
    Prim par;
    cell_prim(P, st, (size_t)ip * M.nj + jp, par);
    ghost_prim(P, M, s, g, par, [&](Prim& o) { cell_prim(P, st, (size_t)(ip + oi) * M.nj + jp + oj, o); }, gh);
}

__device__ __forceinline__ void ghost_state(const Params& P, const Mesh& M, const double* __restrict__ q,
                                            size_t ncell, int side, int along, Prim& gh) {
    ghost_state(P, M, StateF64{q, ncell}, side, along, gh);
}

// Port mass flux of type-6 ghost ghosts[blockIdx.x] by one block: the sum of C1*U*DELY(*YCC)
// along the mesh line through the parent, across to the opposite boundary (the repaired GPORT
// walk).  C1*U is C2, and DELY(*YCC) is a static weight per cell (M.wport; a line read from
// the other side has the opposite sign): 16 bytes a cell, several cells of a thread on their
// way at once, then a reduction in fixed order.  19 -> 9 us at 2048 lines of
// 768 cells; launched like the tile kernels, so that it and the stage after it start during
// the tail of the kernel before them.
template <class St>
__device__ __forceinline__ void port_line(const Mesh& M, const St& st, const int* ghosts, double* gport) {
    const int g = ghosts[blockIdx.x];
    int side, along;
    if (g < M.ni) { side = 1; along = g; }
    else if (g < M.ni + M.nj) { side = 2; along = g - M.ni; }
    else if (g < 2 * M.ni + M.nj) { side = 3; along = g - M.ni - M.nj; }
    else { side = 4; along = g - 2 * M.ni - M.nj; }
    const bool row = side == 1 || side == 3;  // a line along j
    const int len = row ? M.nj : M.ni;
    const double* w = row ? M.wport : M.wport_i;
    const size_t first = row ? (size_t)along * M.nj : along, step = row ? 1 : M.nj;
    pdl_trigger();
    pdl_wait();
    double sum = 0.0;
#pragma unroll 4
    for (int k = threadIdx.x; k < len; k += GP_THREADS) {
        const size_t c = first + k * step;
        sum += st.c(1, c) * w[c];
    }
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    __shared__ double part[GP_THREADS / 32];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = part[0];
#pragma unroll
        for (int k = 1; k < GP_THREADS / 32; k++) t += part[k];
        gport[g] = side == 1 || side == 4 ? -t : t;
    }
}

}  // namespace tns
