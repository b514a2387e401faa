// tns_visc.cuh -- the frozen viscous flux VIS of Q_old (viscous.f90:29-217) on one tile, for
// the FP64 and the mixed kernels: the tile's slots (primitives of its cells, its halo and
// its ghosts), the nodal averages, then each face once; a cell adds its four faces in order
// 1..4, negating the two that were evaluated in the neighbour's orientation.
//
// The face geometry (vector, diamond-gradient coefficients, 1/YAVG: 31 KB a tile, mixed 18) is static:
// one bulk copy per tile, started before the previous kernel has ended.  Each face's flux
// then takes the place of its own geometry, which only the thread that evaluates it reads.
// Boundary nodes find the visit order and the types of their two ghosts in a static code
// instead of through the bc.in line numbers.  What bounds it: instruction issue (a face is
// some 200 instructions) on large meshes, the chain slots -> nodes -> faces of one tile on
// small ones.  Against the same kernel with face rows read from global memory, classified
// halo and nodes everywhere and bc.in lines looked up per boundary node: 38.9 -> 32.7 us
// (1024 x 384), 121 -> 97 us (2048 x 768, a FP64 iteration 0.565 -> 0.535 ms); 115 x 50, an
// iteration: 27.4 -> 25.3 us.
#pragma once

#include "tns_tile.cuh"

namespace tns {

// One tile's shared memory; G: type of the face vectors, gradient coefficients and face fluxes.
// On the mixed path that is float, 43 KB a tile instead of 56: the persistent batch kernel has four
// blocks an SM with its largest phase's shared memory, and lives on the L1 that is left (with 56 KB
// a block in place of 36 an earlier form of it went from 20.1 to 23.4 ms; 64 ramp cases, 20
// iterations).  Those 64 cases: 21.3 -> 19.2 ms, by tile-table launches 17.0 -> 15.2, on branch
// streams 14.3 -> 13.0.
template <class G>
struct ViscSmem {
    G fg[FG_RYAVG][NVF];                   // face geometry, then the fluxes of VIS 0..3
    double ry[NVF];                        // 1/YAVG (axisymmetric meshes)
    double2 uv[NSLOT], tr[NSLOT];          // slots: (U, V), (T, RHO)
    double2 auv[NAVG + 1], atr[NAVG + 1];  // nodal averages
    double ri[NSLOT], ar[NAVG + 1];        // C5/C1 of both
    unsigned long long bar;
};

// The values of one face's four points: A = the cell (slot sa), C = its neighbour (slot sc),
// B, D = the face's nodes ab, ad.
template <class G>
__device__ __forceinline__ void face_values(const ViscSmem<G>& S, int sa, int sc, int ab, int ad, FaceVals& f) {
    double2 v;
    v = S.uv[sa]; f.ua = v.x; f.va = v.y;
    v = S.uv[sc]; f.uc = v.x; f.vc = v.y;
    v = S.auv[ab]; f.ub = v.x; f.vb = v.y;
    v = S.auv[ad]; f.ud = v.x; f.vd = v.y;
    v = S.tr[sa]; f.ta = v.x; f.rhoa = v.y;
    v = S.tr[sc]; f.tc = v.x; f.rhoc = v.y;
    v = S.atr[ab]; f.tb = v.x; f.rhob = v.y;
    v = S.atr[ad]; f.td = v.x; f.rhod = v.y;
    f.ra = S.ri[sa]; f.rc = S.ri[sc]; f.rb = S.ar[ab]; f.rd = S.ar[ad];
}

// face(FaceVals, G sx, sy, ga, gb, gc, gd, double ryavg, G out[4]) evaluates one face's flux.
// The result: tile_copy_wait.  RIM: the block has
// RIM_ROWS more rows of threads, which take the halo, the nodes and the faces beyond the
// cells' own.
template <bool RIM, class G, class OutT, class Face>
__device__ __forceinline__ bool viscous_tile(const Params& P, const Mesh& M, const double* __restrict__ q,
                                             OutT* __restrict__ vis, unsigned int* error, int bx, int by, Face face) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ViscSmem<G>& S = *reinterpret_cast<ViscSmem<G>*>(smem_raw);
    constexpr int BLOCK = sizeof(G) == sizeof(double) ? VTILE : VTILE_MX;
    const size_t ncell = (size_t)M.ni * M.nj;
    const int j0 = bx * TJ, i0 = by * TI;
    const int tj = threadIdx.x, ti = threadIdx.y, tid = ti * TJ + tj;
    pdl_trigger();
    if (tid == 0) {
        bulk_barrier_init(&S.bar);
        const size_t tile = (size_t)by * ((M.nj + TJ - 1) / TJ) + bx;
        bulk_copy_start(S.fg, M.vtile + tile * BLOCK, sizeof(S.fg) + (P.iaxis == 1 ? sizeof(S.ry) : 0), &S.bar);
    }
    const bool inner = i0 > 0 && j0 > 0 && i0 + TI < M.ni && j0 + TJ < M.nj;
    const int i = i0 + ti, j = j0 + tj;
    const bool mine = !RIM || ti < TI;  // the thread has a cell's place
    const bool valid = mine && i < M.ni && j < M.nj;
    const int rt = RIM ? tid - NTHREADS : tid;  // the thread's place on the rim
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
    // nodes: the thread's own (ti, tj), and of the last row and column one more for the first
    // threads; the codes of those on the boundary
    const int xa = rt < AW ? TI : rt - AW, xb = rt < AW ? rt : TJ;
    const bool extra = rt >= 0 && rt < AW + TI;
    int code0 = 0, code1 = 0;
    if (!inner) {
        if (mine) code0 = node_code(M, i, j);
        if (extra) code1 = node_code(M, i0 + xa, j0 + xb);
    }
    pdl_wait();
    __syncthreads();
    auto load = [&](int ci, int cj, double c[5]) {
        const double* p = q + ((size_t)ci * M.nj + cj);
#pragma unroll
        for (int m = 0; m < 5; m++) c[m] = p[m * ncell];
    };
    auto put = [&](int s, const Prim& p) {
        S.uv[s] = make_double2(p.u, p.v);
        S.tr[s] = make_double2(p.t, p.rho);
        S.ri[s] = p.ri;
    };
    {
        double qo[5], qr[5];
        if (valid) load(i, j, qo);
        if (h.kind >= 0) load(h.ci, h.cj, qr);
        Prim p;
        if (valid) {
            primitive(P, qo[0], qo[1], qo[2], qo[3], qo[4], p);
            put((ti + 1) * SW + tj + 1, p);
        }
        if (h.kind >= 0) {
            primitive(P, qr[0], qr[1], qr[2], qr[3], qr[4], p);
            if (h.kind > 0) {
                Prim gh;
                ghost_prim(P, M, site, h.g, p,
                           [&](Prim& o) {
                               double c[5];
                               load(h.ci + h.oi, h.cj + h.oj, c);
                               primitive(P, c[0], c[1], c[2], c[3], c[4], o);
                           }, gh);
                put(h.li * SW + h.lj, gh);
            } else {
                put(h.li * SW + h.lj, p);
            }
        }
    }
    __syncthreads();
    // nodal averages (viscous.f90:40-59,77-124): the four surrounding positions in ascending
    // cell-id order, then the ghosts in bc.in order
    auto node = [&](int la, int lb, int code) {
        const int s0 = la * SW + lb;
        double2 uv, tr;
        double rn;
        double idf = 0.25;
        if (code == 0) {
            const double2 a = S.uv[s0], b = S.uv[s0 + 1], c = S.uv[s0 + SW], d = S.uv[s0 + SW + 1];
            uv = make_double2(a.x + b.x + c.x + d.x, a.y + b.y + c.y + d.y);
            const double2 e = S.tr[s0], f = S.tr[s0 + 1], g = S.tr[s0 + SW], k = S.tr[s0 + SW + 1];
            tr = make_double2(e.x + f.x + g.x + k.x, e.y + f.y + g.y + k.y);
            rn = S.ri[s0] + S.ri[s0 + 1] + S.ri[s0 + SW] + S.ri[s0 + SW + 1];
        } else {
            const int a = i0 + la, b = j0 + lb;
            uv = make_double2(0.0, 0.0);
            tr = uv;
            rn = 0.0;
            int gs[2] = {0, 0}, ng = 0, cnt = 2;  // both ghosts count
            auto take = [&](int s) {
                uv.x += S.uv[s].x;
                uv.y += S.uv[s].y;
                tr.x += S.tr[s].x;
                tr.y += S.tr[s].y;
                rn += S.ri[s];
            };
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int pi = a - 1 + (k >> 1), pj = b - 1 + (k & 1), s = s0 + (k >> 1) * SW + (k & 1);
                const bool in_i = pi >= 0 && pi < M.ni, in_j = pj >= 0 && pj < M.nj;
                if (in_i && in_j) {
                    take(s);
                    cnt++;
                } else if (in_i || in_j) {
                    if (ng == 0) gs[0] = s;
                    else gs[1] = s;
                    ng++;
                }
            }
#pragma unroll
            for (int k = 0; k < 2; k++) {
                take(k == (code >> 6 & 1) ? gs[0] : gs[1]);
                const int type = code >> (3 * k) & 7;
                if (type == 4 || type == 5) uv.y = 0.0;
                if (type == 5) {
                    uv.x = 0.0;
                    rn = P.rtol_rtred;
                }
            }
            if (cnt != 4) idf = 1.0 / (double)cnt;
        }
        const int s = la * AW + lb;
        S.auv[s] = make_double2(uv.x * idf, uv.y * idf);
        S.atr[s] = make_double2(tr.x * idf, tr.y * idf);
        S.ar[s] = dmax1(P.rtol, rn * idf);
    };
    if (mine && i <= M.ni && j <= M.nj) node(ti, tj, code0);
    if (extra && i0 + xa <= M.ni && j0 + xb <= M.nj) node(xa, xb, code1);
    const bool arrived = tile_copy_wait(&S.bar, error);
    auto eval = [&](int f, int sa, int sc, int ab, int ad) {
        FaceVals v;
        face_values(S, sa, sc, ab, ad, v);
        G out[4];
        face(v, S.fg[FG_SX][f], S.fg[FG_SY][f], S.fg[FG_GA][f], S.fg[FG_GB][f], S.fg[FG_GC][f], S.fg[FG_GD][f],
             P.iaxis == 1 ? S.ry[f] : 0.0, out);
#pragma unroll
        for (int k = 0; k < 4; k++) S.fg[k][f] = out[k];
    };
    // a thread's i-face (between cells (i-1, j) and (i, j)), its j-face (between (i, j-1) and
    // (i, j)), then the last row of i-faces and the last column of j-faces
#pragma unroll 1
    for (int r = mine ? 0 : 2; r < 3; r++) {
        int la = ti, lb = tj;
        bool iface = r == 0;
        if (r == 2) {
            iface = rt < TJ;
            la = iface ? TI : rt - TJ;
            lb = iface ? rt : TJ;
            if (rt < 0 || rt >= TJ + TI) break;
        }
        const int fi = i0 + la, fj = j0 + lb;
        if (iface ? fi > M.ni || fj >= M.nj : fi >= M.ni || fj > M.nj) continue;
        const int s = (la + 1) * SW + lb + 1, n = la * AW + lb;  // cell (fi, fj), node (fi, fj)
        const int sb = iface ? s - SW : s - 1, nb = iface ? n + 1 : n + AW;
        // orientation of the cell before the face (as its face 2 or 3), on the first row or
        // column of the mesh of the cell behind it (its face 4 or 1)
        const bool flip = iface ? fi == 0 : fj == 0;
        const bool rev = flip == iface;  // i-faces: B = n, D = n + 1; j-faces the other way
        eval(iface ? la * TJ + lb : NIF + la * AW + lb, flip ? s : sb, flip ? sb : s, rev ? nb : n, rev ? n : nb);
    }
    __syncthreads();
    if (!valid) return arrived;
    const size_t cell = (size_t)i * M.nj + j;
    const int f1 = NIF + ti * AW + tj, f4 = ti * TJ + tj;  // j-face j, i-face i
    const double s1 = (j == 0) ? 1.0 : -1.0, s4 = (i == 0) ? 1.0 : -1.0;
#pragma unroll
    for (int k = 0; k < 4; k++)
        vis[k * ncell + cell] =
            (OutT)(((s1 * (double)S.fg[k][f1] + (double)S.fg[k][f4 + TJ]) + (double)S.fg[k][f1 + 1]) +
                   s4 * (double)S.fg[k][f4]);
    return arrived;
}

}  // namespace tns
