// tns_api.cu -- host runtime behind the C ABI of include/tnsgpu.h.
//
// tns_create validates the Fortran arrays, finds the structured i x j block the cells
// form (faces 1..4 = j-, i+, j+, i- as the reference's generators number them), and
// lays the mesh out on the device in (i, j) order with the ghosts in four side arrays.
// tns_run replays one RK4 iteration (turbnstwod.f90:95-168) as a CUDA graph.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "tns_handle.h"
#include "tns_params.h"
#include "tns_mx.cuh"
#include "tns_tile.cuh"
#include "tns_umesh.h"

using tns::make_params;

namespace {

int build_mesh(tns_handle* h, const tns_mesh* m) {
    const int ne = m->neles, ng = m->nghosts, nn = m->nods;
    if (ne <= 0 || nn <= 0 || ng < 0 || !m->x || !m->y || !m->nod || !m->nc1 || !m->nc2 ||
        !m->nc3 || !m->nc4 || (ng > 0 && (!m->nparent || !m->nghost || !m->ntype || !m->nside)))
        return h->fail(TNS_ERR_ARG, "tns_create: missing mesh arrays or sizes");
    if (m->ld_nod < ne) return h->fail(TNS_ERR_ARG, "tns_create: ld_nod < NELES");
    const int* ncs[4] = {m->nc1, m->nc2, m->nc3, m->nc4};
    auto NOD = [&](int cell0, int k) { return m->nod[(size_t)k * m->ld_nod + cell0]; };
    // ghost lines
    std::unordered_map<int, int> line_of;
    line_of.reserve((size_t)ng * 2 + 1);
    int maxid = ne;
    for (int L = 0; L < ng; L++) {
        const int gid = m->nghost[L], par = m->nparent[L], ty = m->ntype[L], sd = m->nside[L];
        if (gid >= 1 && gid <= ne)
            return h->fail(TNS_ERR_MESH, "bc.in line %d: ghost id %d collides with a cell", L + 1, gid);
        if (gid < 1) return h->fail(TNS_ERR_MESH, "bc.in line %d: bad ghost id %d", L + 1, gid);
        if (!line_of.emplace(gid, L).second)
            return h->fail(TNS_ERR_MESH, "bc.in line %d: ghost id %d repeated", L + 1, gid);
        if (par < 1 || par > ne)
            return h->fail(TNS_ERR_MESH, "bc.in line %d: parent %d out of range", L + 1, par);
        if (sd < 1 || sd > 4) return h->fail(TNS_ERR_MESH, "bc.in line %d: side %d", L + 1, sd);
        if (ty < 2 || ty > 7)
            return h->fail(TNS_ERR_MESH, "bc.in line %d: BC type %d is not one of 2..7", L + 1, ty);
        if (ncs[sd - 1][par - 1] != gid)
            return h->fail(TNS_ERR_MESH, "bc.in line %d: NC%d(%d)=%d is not ghost %d", L + 1, sd,
                           par, ncs[sd - 1][par - 1], gid);
        maxid = std::max(maxid, gid);
    }
    for (int c = 0; c < ne; c++)
        for (int k = 0; k < 4; k++) {
            const int v = ncs[k][c];
            if (v >= 1 && v <= ne) continue;
            auto it = line_of.find(v);
            if (it == line_of.end())
                return h->fail(TNS_ERR_MESH, "cell %d face %d: neighbour %d is neither a cell nor a ghost",
                               c + 1, k + 1, v);
            const int L = it->second;
            if (m->nparent[L] != c + 1 || m->nside[L] != k + 1)
                return h->fail(TNS_ERR_MESH, "ghost %d is referenced by cell %d face %d but belongs to cell %d side %d",
                               v, c + 1, k + 1, m->nparent[L], m->nside[L]);
            const int n1 = NOD(c, k);
            (void)n1;
        }
    for (int c = 0; c < ne; c++)
        for (int k = 0; k < 4; k++) {
            const int v = NOD(c, k);
            if (v < 1 || v > nn) return h->fail(TNS_ERR_MESH, "cell %d node %d: id %d out of range", c + 1, k + 1, v);
        }
    auto is_cell = [&](int v) { return v >= 1 && v <= ne; };
    // corner cell: ghosts on faces 1 and 4
    int corner = -1, ncorner = 0;
    for (int c = 0; c < ne; c++)
        if (!is_cell(m->nc1[c]) && !is_cell(m->nc4[c])) { corner = c; ncorner++; }
    if (ncorner != 1)
        return h->fail(TNS_ERR_UNSUPPORTED,
                       "mesh is not one structured i x j block (%d cells with ghosts on faces 1 and 4)", ncorner);
    int nj = 1, ni = 1;
    for (int c = corner; is_cell(m->nc3[c]); c = m->nc3[c] - 1) {
        if (++nj > ne) return h->fail(TNS_ERR_UNSUPPORTED, "face-3 walk does not end");
    }
    for (int c = corner; is_cell(m->nc2[c]); c = m->nc2[c] - 1) {
        if (++ni > ne) return h->fail(TNS_ERR_UNSUPPORTED, "face-2 walk does not end");
    }
    if ((long long)ni * nj != ne)
        return h->fail(TNS_ERR_UNSUPPORTED, "mesh is not one structured block (%d x %d != %d cells)", ni, nj, ne);
    if (ni < 2 || nj < 2) return h->fail(TNS_ERR_UNSUPPORTED, "need at least 2 x 2 cells (got %d x %d)", ni, nj);
    std::vector<int> cell_of((size_t)ne, -1), seen((size_t)ne, 0);
    int start = corner;
    for (int i = 0; i < ni; i++) {
        int c = start;
        for (int j = 0; j < nj; j++) {
            if (c < 0 || c >= ne || seen[c])
                return h->fail(TNS_ERR_UNSUPPORTED, "cells do not form an i x j block (at %d,%d)", i, j);
            seen[c] = 1;
            cell_of[(size_t)i * nj + j] = c;
            if (j + 1 < nj) c = is_cell(m->nc3[c]) ? m->nc3[c] - 1 : -1;
        }
        if (i + 1 < ni) start = is_cell(m->nc2[start]) ? m->nc2[start] - 1 : -1;
    }
    // adjacency and node consistency
    std::vector<int> node_of((size_t)(ni + 1) * (nj + 1), 0);
    auto set_node = [&](int a, int b, int id) {
        int& slot = node_of[(size_t)a * (nj + 1) + b];
        if (slot == 0) slot = id;
        return slot == id;
    };
    for (int i = 0; i < ni; i++)
        for (int j = 0; j < nj; j++) {
            const int c = cell_of[(size_t)i * nj + j];
            const int want[4] = {j > 0 ? cell_of[(size_t)i * nj + j - 1] + 1 : 0,
                                 i + 1 < ni ? cell_of[(size_t)(i + 1) * nj + j] + 1 : 0,
                                 j + 1 < nj ? cell_of[(size_t)i * nj + j + 1] + 1 : 0,
                                 i > 0 ? cell_of[(size_t)(i - 1) * nj + j] + 1 : 0};
            for (int k = 0; k < 4; k++) {
                const int v = ncs[k][c];
                if (want[k] ? v != want[k] : is_cell(v))
                    return h->fail(TNS_ERR_UNSUPPORTED, "cell %d face %d breaks the i x j block", c + 1, k + 1);
            }
            if (!set_node(i, j, NOD(c, 0)) || !set_node(i + 1, j, NOD(c, 1)) ||
                !set_node(i + 1, j + 1, NOD(c, 2)) || !set_node(i, j + 1, NOD(c, 3)))
                return h->fail(TNS_ERR_UNSUPPORTED, "cell %d: nodes are not shared as in an i x j block", c + 1);
        }
    h->ni = ni; h->nj = nj; h->neles = ne; h->nods = nn; h->nghosts = ng; h->maxid = maxid;
    h->identity = true;
    for (int k = 0; k < ne; k++)
        if (cell_of[k] != k) { h->identity = false; break; }
    h->cell_of.swap(cell_of);

    // device-order host arrays
    const size_t nnode = (size_t)(ni + 1) * (nj + 1), ncell = (size_t)ne;
    const int ngs = 2 * (ni + nj);
    if (ngs != ng)
        return h->fail(TNS_ERR_MESH, "expected %d ghosts for a %d x %d block, bc.in has %d", ngs, ni, nj, ng);
    std::vector<double> X(nnode), Y(nnode), cfldl(ncell), gxc(ngs), gyc(ngs), ginj(ngs, 1.0);
    std::vector<int> gtype(ngs), grank(ngs);
    for (size_t a = 0; a < nnode; a++) {
        X[a] = m->x[node_of[a] - 1];
        Y[a] = m->y[node_of[a] - 1];
    }
    h->M.ni = ni;
    h->M.nj = nj;
    h->ghost_line.assign(ngs, -1);
    h->ghost_id.assign(ng, 0);
    for (int L = 0; L < ng; L++) h->ghost_id[L] = m->nghost[L];
    for (int i = 0; i < ni; i++)
        for (int j = 0; j < nj; j++) {
            const size_t k = (size_t)i * nj + j;
            const int c = h->cell_of[k];
            const size_t n1 = (size_t)i * (nj + 1) + j;
            const double X1 = X[n1], X2 = X[n1 + nj + 1], X3 = X[n1 + nj + 2], X4 = X[n1 + 1];
            const double Y1 = Y[n1], Y2 = Y[n1 + nj + 1], Y3 = Y[n1 + nj + 2], Y4 = Y[n1 + 1];
            // a cell the scheme would divide by: non-finite corners or zero volume
            // (geometry.f90:75-103 takes |VOL| and would carry a zero into DT/VOL)
            if (!(std::isfinite(X1) && std::isfinite(X2) && std::isfinite(X3) && std::isfinite(X4) &&
                  std::isfinite(Y1) && std::isfinite(Y2) && std::isfinite(Y3) && std::isfinite(Y4)))
                return h->fail(TNS_ERR_MESH, "cell %d has a non-finite node coordinate", c + 1);
            double vol = 0.5 * ((X3 - X1) * (Y4 - Y2) - (X4 - X2) * (Y3 - Y1));
            if (h->P.iaxis == 1) vol = vol * ((Y1 + Y2 + Y3 + Y4) * 0.25);
            if (vol == 0.0)
                return h->fail(TNS_ERR_MESH, "cell %d has zero volume (collapsed or on the axis)", c + 1);
            // geometry.f90:70-74
            const double DL12 = std::sqrt((X1 - X2) * (X1 - X2) + (Y1 - Y2) * (Y1 - Y2));
            const double DL23 = std::sqrt((X2 - X3) * (X2 - X3) + (Y2 - Y3) * (Y2 - Y3));
            const double DL34 = std::sqrt((X3 - X4) * (X3 - X4) + (Y3 - Y4) * (Y3 - Y4));
            const double DL41 = std::sqrt((X4 - X1) * (X4 - X1) + (Y4 - Y1) * (Y4 - Y1));
            const double DL = std::min(std::min(std::min(DL12, DL23), DL34), DL41);
            cfldl[k] = h->P.cfl * DL;
            const double xcc = (X1 + X2 + X3 + X4) * 0.25, ycc = (Y1 + Y2 + Y3 + Y4) * 0.25;
            for (int s = 1; s <= 4; s++) {
                const bool bnd = (s == 1 && j == 0) || (s == 2 && i == ni - 1) ||
                                 (s == 3 && j == nj - 1) || (s == 4 && i == 0);
                if (!bnd) continue;
                const int g = h->M.ghost_index(s, (s == 1 || s == 3) ? i : j);
                const int L = line_of.at(ncs[s - 1][c]);
                h->ghost_line[g] = L;
                gtype[g] = m->ntype[L];
                grank[g] = L;
                // geometry.f90:114-142
                double xf, yf;
                if (s == 1) { xf = 0.5 * (X1 + X2); yf = 0.5 * (Y1 + Y2); }
                else if (s == 2) { xf = 0.5 * (X2 + X3); yf = 0.5 * (Y2 + Y3); }
                else if (s == 3) { xf = 0.5 * (X3 + X4); yf = 0.5 * (Y3 + Y4); }
                else { xf = 0.5 * (X4 + X1); yf = 0.5 * (Y4 + Y1); }
                gxc[g] = 2.0 * xf - xcc;
                gyc[g] = 2.0 * yf - ycc;
                if (gtype[g] == 6) h->port_ghosts.push_back(g);
            }
        }
    for (int g = 0; g < ngs; g++)
        if (h->ghost_line[g] < 0) return h->fail(TNS_ERR_MESH, "boundary face %d has no bc.in line", g);
    h->hX.swap(X); h->hY.swap(Y); h->hcfldl.swap(cfldl); h->hgxc.swap(gxc); h->hgyc.swap(gyc);
    h->hginj.swap(ginj); h->hgtype.swap(gtype); h->hgrank.swap(grank);
    h->node_of.swap(node_of);
    return TNS_OK;
}

// Static geometry of the tile kernels, from the device-order node and ghost-centroid
// arrays with the reference's formulas (geometry.f90:55-149; the gradients of
// source_terms.f90:24-60 and viscous.f90:130-180): VOL per cell, the tiles' static blocks of
// the stage and viscous kernels (tns_tile.cuh) and the boundary nodes' codes.
void build_geometry(tns_handle* h) {
    using namespace tns;
    const int ni = h->ni, nj = h->nj, iaxis = h->P.iaxis;
    const std::vector<double>&X = h->hX, &Y = h->hY;
    auto node = [&](int a, int b, double& x, double& y) {
        const size_t n = (size_t)a * (nj + 1) + b;
        x = X[n];
        y = Y[n];
    };
    // centroid of halo position (i, j): a cell from its corners, a ghost mirrored
    auto centroid = [&](int i, int j, double& x, double& y) {
        if (i >= 0 && i < ni && j >= 0 && j < nj) {
            const size_t n1 = (size_t)i * (nj + 1) + j;
            x = (X[n1] + X[n1 + nj + 1] + X[n1 + nj + 2] + X[n1 + 1]) * 0.25;
            y = (Y[n1] + Y[n1 + nj + 1] + Y[n1 + nj + 2] + Y[n1 + 1]) * 0.25;
            return;
        }
        const int g = j == -1 ? h->M.ghost_index(1, i) : i == ni ? h->M.ghost_index(2, j)
                    : j == nj ? h->M.ghost_index(3, i) : h->M.ghost_index(4, j);
        x = h->hgxc[g];
        y = h->hgyc[g];
    };
    // coefficients of the difference gradient over points a, b, c, d
    auto grad = [](double xa, double ya, double xb, double yb, double xc, double yc, double xd,
                   double yd, double* out, size_t stride) {
        const double ybd = yb - yd, yac = ya - yc, xbd = xb - xd, xac = xa - xc;
        const double iDNR = 1.0 / (xac * ybd - xbd * yac);
        out[0] = ybd * iDNR;
        out[stride] = -yac * iDNR;
        out[2 * stride] = -xbd * iDNR;
        out[3 * stride] = xac * iDNR;
    };
    const size_t nc = (size_t)ni * nj;
    h->hcvol.assign(nc, 0.0);
    const int ntj = (nj + TJ - 1) / TJ, nti = (ni + TI - 1) / TI;
    const bool mixed = h->precision == 1;  // (its stage has its own static block)
    const size_t tile = mixed ? MXTILE : STILE;
    h->hstile.assign((size_t)ntj * nti * tile, 0.0);
    for (int i = 0; i < ni; i++)
        for (int j = 0; j < nj; j++) {
            const size_t k = (size_t)i * nj + j;
            double* blk = &h->hstile[((size_t)(i / TI) * ntj + j / TJ) * tile];
            const int at = i % TI * TJ + j % TJ, gc = 2 * SNN + at;
            double xa, ya, xb, yb, xc, yc, xd, yd;
            centroid(i, j - 1, xa, ya);  // NC1..NC4
            centroid(i + 1, j, xb, yb);
            centroid(i, j + 1, xc, yc);
            centroid(i - 1, j, xd, yd);
            double g[4];
            grad(xa, ya, xb, yb, xc, yc, xd, yd, g, 1);
            const size_t n1 = (size_t)i * (nj + 1) + j;
            const double Xc[4] = {X[n1], X[n1 + nj + 1], X[n1 + nj + 2], X[n1 + 1]};
            const double Yc[4] = {Y[n1], Y[n1 + nj + 1], Y[n1 + nj + 2], Y[n1 + 1]};
            const double ycc = (Yc[0] + Yc[1] + Yc[2] + Yc[3]) * 0.25;
            const double vol = cell_volume(iaxis, Xc, Yc, ycc);
            h->hcvol[k] = vol;
            if (mixed) {
                double sx[4], sy[4];
                for (int f = 0; f < 4; f++) face_vector(iaxis, f + 1, Xc, Yc, sx[f], sy[f]);
                GeoMx m;
                geo_mx(iaxis, sx, sy, g, vol, ycc, m);
                float4* f4 = reinterpret_cast<float4*>(blk) + at;
                f4[0] = m.s01;
                f4[TI * TJ] = m.s23;
                f4[2 * TI * TJ] = m.g;
                f4[3 * TI * TJ] = m.w;
                blk[MX_SUMX * TI * TJ + at] = m.sumx;
                blk[MX_SUMY * TI * TJ + at] = m.sumy;
                blk[MX_VR * TI * TJ + at] = m.vr;
                continue;
            }
            for (int f = 0; f < 4; f++) blk[gc + (ST_GA + f) * TI * TJ] = g[f];
            blk[gc + ST_RVOL * TI * TJ] = 1.0 / vol;
            blk[gc + ST_RYCC * TI * TJ] = 1.0 / ycc;
        }
    for (int a = 0; !mixed && a <= ni; a++)  // nodes of each tile's cells; shared rows go to both tiles
        for (int b = 0; b <= nj; b++)
            for (int bi = std::max(0, (a - 1) / TI); bi <= std::min(nti - 1, a / TI); bi++)
                for (int bj = std::max(0, (b - 1) / TJ); bj <= std::min(ntj - 1, b / TJ); bj++) {
                    const int la = a - bi * TI, lb = b - bj * TJ;
                    if (la < 0 || la > TI || lb < 0 || lb > TJ) continue;
                    double* blk = &h->hstile[((size_t)bi * ntj + bj) * STILE];
                    node(a, b, blk[la * SNW + lb], blk[SNN + la * SNW + lb]);
                }
    // one face: A = the evaluating cell, C = the neighbour, B, D = the face's nodes
    auto face = [&](double* fg, int ia, int ja, int ic, int jc, int ib, int jb, int id, int jd) {
        double xa, ya, xc, yc, xb, yb, xd, yd;
        centroid(ia, ja, xa, ya);
        centroid(ic, jc, xc, yc);
        node(ib, jb, xb, yb);
        node(id, jd, xd, yd);
        if (iaxis == 1) {
            fg[FG_SX] = (yd - yb) * (yb + yd) * HALF;
            fg[FG_SY] = -(xd - xb) * (yb + yd) * HALF;
        } else {
            fg[FG_SX] = (yd - yb);
            fg[FG_SY] = -(xd - xb);
        }
        grad(xa, ya, xb, yb, xc, yc, xd, yd, &fg[FG_GA], 1);
        const double yavg = HALF * (yb + yd);
        fg[FG_RYAVG] = (iaxis == 1 && !(yavg < YAXIS_THRESH)) ? 1.0 / yavg : 0.0;
    };
    const size_t vt = mixed ? VTILE_MX : VTILE;
    h->hvtile.assign((size_t)ntj * nti * vt, 0.0);
    auto store = [&](const double* fg, int bi, int bj, int f) {
        double* blk = &h->hvtile[((size_t)bi * ntj + bj) * vt];
        if (mixed) {
            float* b4 = reinterpret_cast<float*>(blk);
            for (int k = 0; k < FG_RYAVG; k++) b4[(size_t)k * NVF + f] = (float)fg[k];
            blk[(size_t)FG_RYAVG * NVF / 2 + f] = fg[FG_RYAVG];
            return;
        }
        for (int k = 0; k < FG_N; k++) blk[(size_t)k * NVF + f] = fg[k];
    };
    double fg[FG_N];
    for (int i = 0; i <= ni; i++)
        for (int j = 0; j < nj; j++) {
            if (i == 0)  // face 4 of cell (0, j): B = node (0, j+1), D = node (0, j)
                face(fg, 0, j, -1, j, 0, j + 1, 0, j);
            else  // face 2 of cell (i-1, j): B = node (i, j), D = node (i, j+1)
                face(fg, i - 1, j, i, j, i, j, i, j + 1);
            const int lb = j % TJ;
            if (i < ni) store(fg, i / TI, j / TJ, i % TI * TJ + lb);
            // the first row of a tile is also the last of the one before it
            if (i > 0 && (i % TI == 0 || i == ni)) store(fg, (i - 1) / TI, j / TJ, ((i - 1) % TI + 1) * TJ + lb);
        }
    for (int i = 0; i < ni; i++)
        for (int j = 0; j <= nj; j++) {
            if (j == 0)  // face 1 of cell (i, 0): B = node (i, 0), D = node (i+1, 0)
                face(fg, i, 0, i, -1, i, 0, i + 1, 0);
            else  // face 3 of cell (i, j-1): B = node (i+1, j), D = node (i, j)
                face(fg, i, j - 1, i, j, i + 1, j, i, j);
            const int la = NIF + i % TI * (TJ + 1);
            if (j < nj) store(fg, i / TI, j / TJ, la + j % TJ);
            if (j > 0 && (j % TJ == 0 || j == nj)) store(fg, i / TI, (j - 1) / TJ, la + (j - 1) % TJ + 1);
        }
    // the boundary nodes' ghosts (Mesh::bnode)
    auto code = [&](int a, int b) {
        int g[2] = {0, 0}, n = 0;
        for (int k = 0; k < 4; k++) {
            const int pi = a - 1 + (k >> 1), pj = b - 1 + (k & 1);
            const bool in_i = pi >= 0 && pi < ni, in_j = pj >= 0 && pj < nj;
            if (in_i == in_j) continue;  // a cell, or no position
            g[n++] = in_i ? h->M.ghost_index(pj < 0 ? 1 : 3, pi) : h->M.ghost_index(pi < 0 ? 4 : 2, pj);
        }
        const bool swap = h->hgrank[g[1]] < h->hgrank[g[0]];
        return h->hgtype[g[swap ? 1 : 0]] | h->hgtype[g[swap ? 0 : 1]] << 3 | (swap ? 1 << 6 : 0);
    };
    h->hbnode.clear();
    for (int a = 0; a <= ni; a++) h->hbnode.push_back(code(a, 0));
    for (int a = 0; a <= ni; a++) h->hbnode.push_back(code(a, nj));
    for (int b = 0; b <= nj; b++) h->hbnode.push_back(code(0, b));
    for (int b = 0; b <= nj; b++) h->hbnode.push_back(code(ni, b));
}

// Device copy of the layout built by build_mesh.
int upload_mesh(tns_handle* h) {
    const size_t nnode = h->hX.size(), ncell = h->hcfldl.size(), ngs = h->hgxc.size();
    int rc;
    if ((rc = h->cuda(h->x.alloc(nnode), "cudaMalloc")) || (rc = h->cuda(h->y.alloc(nnode), "cudaMalloc")) ||
        (rc = h->cuda(h->cfldl.alloc(ncell), "cudaMalloc")) || (rc = h->cuda(h->gxc.alloc(ngs), "cudaMalloc")) ||
        (rc = h->cuda(h->gyc.alloc(ngs), "cudaMalloc")) || (rc = h->cuda(h->ginj.alloc(ngs), "cudaMalloc")) ||
        (rc = h->cuda(h->gport.alloc(ngs), "cudaMalloc")) || (rc = h->cuda(h->gtype.alloc(ngs), "cudaMalloc")) ||
        (rc = h->cuda(h->grank.alloc(ngs), "cudaMalloc")) ||
        (rc = h->cuda(h->ports.alloc(h->port_ghosts.size()), "cudaMalloc")))
        return rc;
    auto up = [&](void* dst, const void* src, size_t bytes) {
        return h->cuda(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice), "cudaMemcpy");
    };
    if ((rc = up(h->x.p, h->hX.data(), nnode * 8)) || (rc = up(h->y.p, h->hY.data(), nnode * 8)) ||
        (rc = up(h->cfldl.p, h->hcfldl.data(), ncell * 8)) ||
        (rc = up(h->gxc.p, h->hgxc.data(), ngs * 8)) || (rc = up(h->gyc.p, h->hgyc.data(), ngs * 8)) ||
        (rc = up(h->ginj.p, h->hginj.data(), ngs * 8)) ||
        (rc = up(h->gtype.p, h->hgtype.data(), ngs * 4)) ||
        (rc = up(h->grank.p, h->hgrank.data(), ngs * 4)))
        return rc;
    if (!h->port_ghosts.empty() &&
        (rc = up(h->ports.p, h->port_ghosts.data(), h->port_ghosts.size() * 4)))
        return rc;
    if ((rc = h->cuda(cudaMemset(h->gport.p, 0, ngs * 8), "cudaMemset"))) return rc;
    build_geometry(h);
    std::vector<double> vcfl(ncell);
    for (size_t k = 0; k < ncell; k++) vcfl[k] = h->hcvol[k] / h->hcfldl[k];
    if ((rc = h->cuda(h->cvol.alloc(h->hcvol.size()), "cudaMalloc")) ||
        (rc = h->cuda(h->vcfl.alloc(ncell), "cudaMalloc")) || (rc = up(h->vcfl.p, vcfl.data(), ncell * 8)) ||
        (rc = h->cuda(h->stile.alloc(h->hstile.size()), "cudaMalloc")) ||
        (rc = h->cuda(h->vtile.alloc(h->hvtile.size()), "cudaMalloc")) ||
        (rc = h->cuda(h->bnode.alloc(h->hbnode.size()), "cudaMalloc")) ||
        (rc = up(h->cvol.p, h->hcvol.data(), h->hcvol.size() * 8)) ||
        (rc = up(h->stile.p, h->hstile.data(), h->hstile.size() * 8)) ||
        (rc = up(h->vtile.p, h->hvtile.data(), h->hvtile.size() * 8)) ||
        (rc = up(h->bnode.p, h->hbnode.data(), h->hbnode.size() * 4)))
        return rc;
    // the host copies are not read again
    // weights of the port sums (boundary.f90:183-214), where there are ports along j or i
    if (!h->port_ghosts.empty()) {
        const int ni = h->ni, nj = h->nj;
        bool along_j = false, along_i = false;
        for (int g : h->port_ghosts) {
            const bool row = g < ni || (g >= ni + nj && g < 2 * ni + nj);
            along_j |= row;
            along_i |= !row;
        }
        std::vector<double> w(ncell);
        for (int dir = 0; dir < 2; dir++) {
            if (dir == 0 ? !along_j : !along_i) continue;
            for (int i = 0; i < ni; i++)
                for (int j = 0; j < nj; j++) {
                    const size_t n1 = (size_t)i * (nj + 1) + j;
                    const double y1 = h->hY[n1], y2 = h->hY[n1 + nj + 1], y3 = h->hY[n1 + nj + 2], y4 = h->hY[n1 + 1];
                    double v = dir == 0 ? tns::HALF * ((y3 + y4) - (y1 + y2)) : tns::HALF * ((y2 + y3) - (y1 + y4));
                    if (h->P.iaxis == 1) v = v * ((y1 + y2 + y3 + y4) * 0.25);
                    w[(size_t)i * nj + j] = v;
                }
            DevBuf<double>& d = dir == 0 ? h->wport : h->wport_i;
            if ((rc = h->cuda(d.alloc(ncell), "cudaMalloc")) || (rc = up(d.p, w.data(), ncell * 8))) return rc;
        }
    }
    // static ghost records
    {
        const int ni = h->ni, nj = h->nj;
        std::vector<tns::GhostRec> rec(ngs);
        for (int g = 0; g < (int)ngs; g++) {
            const int side = g < ni ? 1 : g < ni + nj ? 2 : g < 2 * ni + nj ? 3 : 4;
            const int along = side == 1 ? g : side == 2 ? g - ni : side == 3 ? g - ni - nj : g - 2 * ni - nj;
            const int ip = side == 2 ? ni - 1 : side == 4 ? 0 : along, jp = side == 1 ? 0 : side == 3 ? nj - 1 : along;
            const size_t n1 = (size_t)ip * (nj + 1) + jp;
            const double X[4] = {h->hX[n1], h->hX[n1 + nj + 1], h->hX[n1 + nj + 2], h->hX[n1 + 1]};
            const double Y[4] = {h->hY[n1], h->hY[n1 + nj + 1], h->hY[n1 + nj + 2], h->hY[n1 + 1]};
            tns::face_vector(h->P.iaxis, side, X, Y, rec[g].psx, rec[g].psy);
            rec[g].ycg = h->hgyc[g];
            rec[g].ycp = (Y[0] + Y[1] + Y[2] + Y[3]) * 0.25;
        }
        if ((rc = h->cuda(h->grec.alloc(ngs), "cudaMalloc")) ||
            (rc = up(h->grec.p, rec.data(), ngs * sizeof(tns::GhostRec))))
            return rc;
    }
    std::vector<double>().swap(h->hcvol);
    std::vector<double>().swap(h->hstile);
    std::vector<double>().swap(h->hvtile);
    Mesh& M = h->M;
    M.ni = h->ni; M.nj = h->nj; M.x = h->x.p; M.y = h->y.p; M.cfldl = h->cfldl.p; M.gtype = h->gtype.p;
    M.grank = h->grank.p; M.gxc = h->gxc.p; M.gyc = h->gyc.p; M.ginj = h->ginj.p;
    M.gport = h->gport.p;
    M.wport = h->wport.p;
    M.wport_i = h->wport_i.p;
    M.grec = h->grec.p;
    M.cvol = h->cvol.p;
    M.vcfl = h->vcfl.p;
    M.stile = h->stile.p;
    M.vtile = h->vtile.p;
    M.bnode = h->bnode.p;
    return TNS_OK;
}

int alloc_state(tns_handle* h) {
    const size_t nc = h->ncell();
    int rc;
    if (!h->identity &&
        ((rc = h->cuda(h->dcell_of.alloc(nc), "cudaMalloc")) || (rc = h->cuda(h->renum.alloc(5 * nc), "cudaMalloc")) ||
         (rc = h->cuda(cudaMemcpy(h->dcell_of.p, h->cell_of.data(), nc * sizeof(int), cudaMemcpyHostToDevice),
                       "cudaMemcpy"))))
        return rc;
    if (h->precision == 1) {
        if ((rc = h->cuda(h->qa.alloc(5 * nc), "cudaMalloc")) || (rc = h->cuda(h->qa2.alloc(5 * nc), "cudaMalloc")) ||
            (rc = h->cuda(h->dqb.alloc(5 * nc), "cudaMalloc")) || (rc = h->cuda(h->dqc.alloc(5 * nc), "cudaMalloc")) ||
            (rc = h->cuda(h->df.alloc(5 * nc), "cudaMalloc")) || (rc = h->cuda(h->visf.alloc(4 * nc), "cudaMalloc")) ||
            (rc = h->cuda(h->ef.alloc(4 * nc), "cudaMalloc")) || (rc = h->cuda(h->dtf.alloc(nc), "cudaMalloc")))
            return rc;
        if ((rc = h->cuda(cudaMemset(h->dtf.p, 0, nc * 4), "cudaMemset")) ||
            (rc = h->cuda(cudaMemset(h->visf.p, 0, 4 * nc * 4), "cudaMemset")))
            return rc;
        const size_t ntiles = (size_t)((h->nj + tns::TJ - 1) / tns::TJ) * ((h->ni + tns::TI - 1) / tns::TI);
        if ((rc = h->cuda(h->tref.alloc(ntiles * tns::TREF_WORDS), "cudaMalloc")) ||
            (rc = h->cuda(cudaMemset(h->tref.p, 0, ntiles * tns::TREF_WORDS * 8), "cudaMemset")))
            return rc;
        h->M.tref = reinterpret_cast<tns::TileRefMx*>(h->tref.p);
        // a general mesh's global time step (LOCAL=0) writes the FP64 per-cell DT
        if (h->unstructured && (rc = h->cuda(h->dt.alloc(nc), "cudaMalloc"))) return rc;
    } else if ((rc = h->cuda(h->qa.alloc(5 * nc), "cudaMalloc")) || (rc = h->cuda(h->qb.alloc(5 * nc), "cudaMalloc")) ||
               (rc = h->cuda(h->qc.alloc(5 * nc), "cudaMalloc")) || (rc = h->cuda(h->d.alloc(5 * nc), "cudaMalloc")) ||
               (rc = h->cuda(h->vis.alloc(4 * nc), "cudaMalloc")) || (rc = h->cuda(h->dt.alloc(nc), "cudaMalloc")) ||
               (rc = h->cuda(h->e.alloc(5 * nc), "cudaMalloc"))) {
        return rc;
    }
    if ((rc = h->cuda(h->dtmin.alloc(1), "cudaMalloc")) ||
        (rc = h->cuda(h->partial.alloc((size_t)tns::dtmin_blocks(h->M)), "cudaMalloc")) ||
        (rc = h->cuda(h->counter.alloc(1), "cudaMalloc")) || (rc = h->cuda(h->status.alloc(1), "cudaMalloc")) ||
        (rc = h->cuda(h->cdiff.alloc(5), "cudaMalloc")))
        return rc;
    if ((rc = h->cuda(cudaMemset(h->counter.p, 0, 4), "cudaMemset")) ||
        (rc = h->cuda(cudaMemset(h->status.p, 0, 4), "cudaMemset")))
        return rc;
    if (h->precision == 0 && ((rc = h->cuda(cudaMemset(h->dt.p, 0, nc * 8), "cudaMemset")) ||
                              (rc = h->cuda(cudaMemset(h->vis.p, 0, 4 * nc * 8), "cudaMemset"))))
        return rc;
    if ((rc = h->cuda(cudaMallocHost((void**)&h->status_host, sizeof(unsigned int)), "cudaMallocHost")))
        return rc;
    return h->cuda(cudaMallocHost((void**)&h->pinned, 5 * nc * sizeof(double)), "cudaMallocHost");
}

}  // namespace

namespace tns_rt {

// The two pre-passes of an iteration read only Q_old and write disjoint arrays: the
// dissipation (with DTMIN before it, LOCAL=0) on the side stream, the frozen viscous flux
// (with stage 1's port columns before it) on the main stream, joined before stage 1.
// With per-kernel profiling both run in order on the main stream.
template <class Diss, class Visc>
void prepass(tns_handle* h, Diss&& diss, Visc&& visc) {
    if (h->profile || !h->side) {
        diss(h->stream);
        visc(h->stream);
        return;
    }
    cudaEventRecord(h->fork, h->stream);
    cudaStreamWaitEvent(h->side, h->fork, 0);
    diss(h->side);
    visc(h->stream);
    cudaEventRecord(h->join, h->side);
    cudaStreamWaitEvent(h->stream, h->join, 0);
}

// One mixed-precision RK4 iteration from state buffer `in` to `out` (FP32 increments
// dQ_B, dQ_C between the stages).  The previous state survives in `in`, so the last
// stage's input (in + dQ_B) can be reconstructed for tns_download_primitives.
void enqueue_iteration_mx(tns_handle* h, bool monitor, double* A, double* Aout) {
    if (h->unstructured) {
        enqueue_iteration_u_mx(h, monitor, A, Aout);
        return;
    }
    const Params& P = h->P;
    const Mesh& M = h->M;
    const int np = (int)h->port_ghosts.size();
    static const double alpha[4] = {0.25, 1.0 / 3.0, 0.5, 1.0};
    const float* in[4] = {nullptr, h->dqb.p, h->dqc.p, h->dqb.p};
    float* out[4] = {h->dqb.p, h->dqc.p, h->dqb.p, nullptr};
    prepass(
        h,
        [&](cudaStream_t s) {
            if (!P.local)
                launch(h, K_DTMIN, [&] { tns::launch_dtmin(P, M, A, h->partial.p, h->counter.p, h->dtmin.p, s); });
            launch(h, K_DISS, [&] { tns::launch_dissipation_mx(P, M, A, h->df.p, h->dtf.p, h->dtmin.p, s); });
        },
        [&](cudaStream_t s) {
            if (np) launch(h, K_GPORT, [&] { tns::launch_gport_mx(P, M, A, in[0], h->ports.p, np, h->gport.p, s); });
            launch(h, K_VISC, [&] { tns::launch_viscous_mx(P, M, A, h->visf.p, h->status.p, s, h->beside); });
        });
    cudaStream_t s = h->stream;
    if (monitor) cudaMemsetAsync(h->cdiff.p, 0, 5 * sizeof(unsigned long long), s);
    for (int st = 0; st < 4; st++) {
        if (np && st > 0)
            launch(h, K_GPORT, [&] { tns::launch_gport_mx(P, M, A, in[st], h->ports.p, np, h->gport.p, s); });
        launch(h, K_STAGE, [&] {
            tns::launch_stage_mx(P, M, A, in[st], out[st], st == 3 ? Aout : nullptr, h->df.p, h->visf.p, h->ef.p,
                                 h->dtf.p, h->dtmin.p, alpha[st], (monitor && st == 3) ? h->cdiff.p : nullptr,
                                 st == 3 ? h->status.p : nullptr, h->status.p, s, h->beside);
        });
    }
}

// One RK4 iteration (turbnstwod.f90:97-168).  Buffers: A = state, B/C = stage scratch;
// stage 4 writes A in place (each cell reads only its own COLD there).
void enqueue_iteration_f64(tns_handle* h, bool monitor) {
    if (h->unstructured) {
        enqueue_iteration_u(h, monitor);
        return;
    }
    const Params& P = h->P;
    const Mesh& M = h->M;
    double *A = h->qa.p, *B = h->qb.p, *Cq = h->qc.p;
    const int np = (int)h->port_ghosts.size();
    const double* in[4] = {A, B, Cq, B};
    double* out[4] = {B, Cq, B, A};
    prepass(
        h,
        [&](cudaStream_t s) {
            if (!P.local)
                launch(h, K_DTMIN, [&] { tns::launch_dtmin(P, M, A, h->partial.p, h->counter.p, h->dtmin.p, s); });
            launch(h, K_DISS, [&] { tns::launch_dissipation(P, M, A, h->d.p, h->dt.p, h->dtmin.p, s); });
        },
        [&](cudaStream_t s) {
            // the frozen viscous flux of Q_old uses stage 1's boundary state (viscous.f90:29)
            if (np) launch(h, K_GPORT, [&] { tns::launch_gport(P, M, in[0], h->ports.p, np, h->gport.p, s); });
            launch(h, K_VISC, [&] { tns::launch_viscous(P, M, A, h->vis.p, h->status.p, s, h->beside); });
        });
    cudaStream_t s = h->stream;
    if (monitor) cudaMemsetAsync(h->cdiff.p, 0, 5 * sizeof(unsigned long long), s);
    for (int st = 0; st < 4; st++) {
        if (np && st > 0)
            launch(h, K_GPORT, [&] { tns::launch_gport(P, M, in[st], h->ports.p, np, h->gport.p, s); });
        launch(h, K_STAGE, [&] {
            tns::launch_stage(P, M, in[st], A, out[st], h->d.p, h->vis.p, h->dt.p, h->dtmin.p, st, h->e.p,
                              (monitor && st == 3) ? h->cdiff.p : nullptr,
                              st == 3 ? h->status.p : nullptr, h->status.p, s, h->beside);
        });
    }
}

}  // namespace tns_rt

extern "C" {

int tns_create(const tns_mesh* mesh, const tns_params* params, tns_handle** out) {
    if (!out) return TNS_ERR_ARG;
    *out = nullptr;
    if (!mesh || !params) return TNS_ERR_ARG;
    tns_handle* h = new tns_handle();
    *out = h;
    if (params->precision != 0 && params->precision != 1)
        return h->fail(TNS_ERR_ARG, "precision mode %d is not available (0 = FP64, 1 = mixed)", params->precision);
    h->precision = params->precision;
    if (!(params->gama > 1.0) || !(params->amol > 0.0) || !(params->cfl > 0.0))
        return h->fail(TNS_ERR_ARG, "GAMA must exceed 1, AMOL and CFL must be positive");
    h->P = make_params(*params);
    int rc;
    // host-side validation and layout first: mesh errors are reported without a GPU.  A
    // mesh that is not one structured block takes the general (gather) layout, FP64 only.
    rc = build_mesh(h, mesh);
    if (rc == TNS_ERR_UNSUPPORTED) rc = tns_rt::umesh_build(h, mesh);
    if (rc) return rc;
    if ((rc = h->cuda(cudaStreamCreateWithFlags(&h->own, cudaStreamNonBlocking), "cudaStreamCreate"))) return rc;
    h->stream = h->own;
    if ((rc = h->cuda(tns::configure_kernels(), "cudaFuncSetAttribute"))) return rc;
    if ((rc = h->cuda(tns::configure_kernels_mx(), "cudaFuncSetAttribute"))) return rc;
    if ((rc = h->unstructured ? tns_rt::umesh_upload(h) : upload_mesh(h))) return rc;
    if ((rc = alloc_state(h))) return rc;
    cudaEventCreate(&h->ev[0]);
    cudaEventCreate(&h->ev[1]);
    if ((rc = h->cuda(cudaStreamCreateWithFlags(&h->side, cudaStreamNonBlocking), "cudaStreamCreate")) ||
        (rc = h->cuda(cudaEventCreateWithFlags(&h->fork, cudaEventDisableTiming), "cudaEventCreate")) ||
        (rc = h->cuda(cudaEventCreateWithFlags(&h->join, cudaEventDisableTiming), "cudaEventCreate")))
        return rc;
    return TNS_OK;
}

int tns_set_injection_scale(tns_handle* h, const double* scale) {
    if (!h || !scale) return TNS_ERR_ARG;
    if (h->unstructured) return tns_rt::umesh_set_injection(h, scale);
    std::vector<double> g((size_t)h->M.nghosts(), 1.0);
    for (size_t k = 0; k < g.size(); k++) g[k] = scale[h->ghost_line[k]];
    return h->cuda(cudaMemcpy(h->ginj.p, g.data(), g.size() * 8, cudaMemcpyHostToDevice), "cudaMemcpy");
}

namespace {
bool page_locked(const void* p) {
    cudaPointerAttributes at;
    const bool ok = cudaPointerGetAttributes(&at, p) == cudaSuccess && at.type == cudaMemoryTypeHost;
    cudaGetLastError();
    return ok;
}

// The asynchronous transfers: one DMA per component on the handle's stream, page-locked
// caller arrays in the handle's own cell order only (no staging, no scatter).
int async_arrays_ok(tns_handle* h, const void* const* a, const char* who) {
    if (!h->identity)
        return h->fail(TNS_ERR_UNSUPPORTED, "%s: the mesh is renumbered on the device; use the synchronous call", who);
    for (int m = 0; m < 5; m++)
        if (!a[m] || !page_locked(a[m])) return h->fail(TNS_ERR_ARG, "%s: array %d is not page-locked", who, m + 1);
    return TNS_OK;
}
}  // namespace

int tns_upload_state_async(tns_handle* h, const double* c1, const double* c2, const double* c3,
                           const double* c4, const double* c5) {
    if (!h) return TNS_ERR_ARG;
    const double* src[5] = {c1, c2, c3, c4, c5};
    int rc;
    if ((rc = async_arrays_ok(h, reinterpret_cast<const void* const*>(src), "tns_upload_state_async"))) return rc;
    const size_t nc = h->ncell();
    for (int m = 0; m < 5; m++)
        if ((rc = h->cuda(cudaMemcpyAsync(h->state() + m * nc, src[m], nc * 8, cudaMemcpyHostToDevice, h->stream),
                          "cudaMemcpyAsync")))
            return rc;
    h->have_state = true;
    return TNS_OK;
}

int tns_download_state_async(tns_handle* h, double* c1, double* c2, double* c3, double* c4, double* c5) {
    if (!h) return TNS_ERR_ARG;
    if (!h->have_state) return h->fail(TNS_ERR_STATE, "tns_download_state_async: no state");
    double* dst[5] = {c1, c2, c3, c4, c5};
    int rc;
    if ((rc = async_arrays_ok(h, reinterpret_cast<const void* const*>(dst), "tns_download_state_async")))
        return rc;
    const size_t nc = h->ncell();
    for (int m = 0; m < 5; m++)
        if ((rc = h->cuda(cudaMemcpyAsync(dst[m], h->state() + m * nc, nc * 8, cudaMemcpyDeviceToHost, h->stream),
                          "cudaMemcpyAsync")))
            return rc;
    return TNS_OK;
}

int tns_upload_state(tns_handle* h, const double* c1, const double* c2, const double* c3,
                     const double* c4, const double* c5) {
    if (!h || !c1 || !c2 || !c3 || !c4 || !c5) return TNS_ERR_ARG;
    const size_t nc = h->ncell();
    const double* src[5] = {c1, c2, c3, c4, c5};
    int rc;
    // a state in the caller's own numbering is put in the device's order there
    double* dst = h->identity ? h->state() : h->renum.p;
    bool direct = true;
    for (int m = 0; m < 5 && direct; m++) direct = page_locked(src[m]);
    if (direct) {
        // page-locked caller arrays: one DMA per component, no staging copy
        for (int m = 0; m < 5; m++)
            if ((rc = h->cuda(cudaMemcpyAsync(dst + m * nc, src[m], nc * 8, cudaMemcpyHostToDevice, h->stream),
                              "cudaMemcpyAsync")))
                return rc;
    } else {
        for (int m = 0; m < 5; m++) std::memcpy(h->pinned + m * nc, src[m], nc * 8);
        if ((rc = h->cuda(cudaMemcpyAsync(dst, h->pinned, 5 * nc * 8, cudaMemcpyHostToDevice, h->stream),
                          "cudaMemcpyAsync")))
            return rc;
    }
    if (!h->identity) {
        tns::launch_renumber(h->dcell_of.p, dst, h->state(), nc, true, h->stream);
        if ((rc = h->cuda(cudaGetLastError(), "kernel launch"))) return rc;
    }
    rc = h->cuda(cudaStreamSynchronize(h->stream), "cudaStreamSynchronize");
    if (rc) return rc;
    h->have_state = true;
    return TNS_OK;
}

namespace {

// Enqueues one iteration of the handle's precision mode and advances the state buffer.
void enqueue_iteration(tns_handle* h, bool monitor) {
    if (h->precision == 1) {
        enqueue_iteration_mx(h, monitor, h->state(), h->other_state());
        h->cur ^= 1;
    } else {
        enqueue_iteration_f64(h, monitor);
    }
}

int capture(tns_handle* h, cudaGraphExec_t* exec, bool mixed, int parity, bool monitor = false, int iters = 1) {
    cudaGraph_t g;
    int rc;
    if ((rc = h->cuda(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal), "capture")))
        return rc;
    const long long before = h->launches;
    for (int k = 0; k < iters; k++) {
        if (mixed) {
            double* A = parity ^ (k & 1) ? h->qa2.p : h->qa.p;
            double* B = parity ^ (k & 1) ? h->qa.p : h->qa2.p;
            enqueue_iteration_mx(h, monitor, A, B);
        } else {
            enqueue_iteration_f64(h, monitor);
        }
    }
    h->per_iter = (h->launches - before) / iters;
    h->launches = before;
    if ((rc = h->cuda(cudaStreamEndCapture(h->stream, &g), "capture"))) return rc;
    rc = h->cuda(cudaGraphInstantiate(exec, g, 0), "cudaGraphInstantiate");
    cudaGraphDestroy(g);
    return rc;
}

// Captures one unmonitored iteration as a CUDA graph (once per handle; the mixed path
// needs one per state-buffer parity), and GRAPH_BLOCK of them as another.
int ensure_graph(tns_handle* h) {
    int rc;
    const bool mixed = h->precision == 1;
    for (int par = 0; par < (mixed ? 2 : 1); par++) {
        cudaGraphExec_t* g = mixed ? &h->graph_mx[par] : &h->graph;
        if (!*g && (rc = capture(h, g, mixed, par))) return rc;
    }
    return TNS_OK;
}
int ensure_block_graph(tns_handle* h) {
    const bool mixed = h->precision == 1;
    int rc;
    for (int par = 0; par < (mixed ? 2 : 1); par++)
        if (!h->graph_block[par] && (rc = capture(h, &h->graph_block[par], mixed, par, false, GRAPH_BLOCK))) return rc;
    return TNS_OK;
}

// One monitored iteration: a captured graph (memset of the CDIFF slots + the iteration),
// or direct launches when per-kernel profiling is on.
int enqueue_monitored(tns_handle* h) {
    if (h->profile) {
        enqueue_iteration(h, true);
        return TNS_OK;
    }
    int rc;
    cudaGraphExec_t* g = h->precision == 1 ? &h->graph_mon_mx[h->cur] : &h->graph_mon;
    if (!*g) {
        const long long per = h->per_iter;
        if ((rc = capture(h, g, h->precision == 1, h->cur, true))) return rc;
        h->per_iter_mon = h->per_iter;
        h->per_iter = per;
    }
    if ((rc = h->cuda(cudaGraphLaunch(*g, h->stream), "cudaGraphLaunch"))) return rc;
    if (h->precision == 1) h->cur ^= 1;
    h->launches += h->per_iter_mon;
    return TNS_OK;
}

int enqueue_plain(tns_handle* h, int niter) {
    int rc;
    if (h->profile) {
        for (int it = 0; it < niter; it++) enqueue_iteration(h, false);
        return TNS_OK;
    }
    if ((rc = ensure_graph(h))) return rc;
    int it = 0;
    if (niter >= GRAPH_BLOCK) {
        if ((rc = ensure_block_graph(h))) return rc;
        for (; it + GRAPH_BLOCK <= niter; it += GRAPH_BLOCK) {  // an even number: the parity stays
            if ((rc = h->cuda(cudaGraphLaunch(h->graph_block[h->precision == 1 ? h->cur : 0], h->stream),
                              "cudaGraphLaunch")))
                return rc;
            h->launches += GRAPH_BLOCK * h->per_iter;
        }
    }
    for (; it < niter; it++) {
        cudaGraphExec_t g = h->precision == 1 ? h->graph_mx[h->cur] : h->graph;
        if ((rc = h->cuda(cudaGraphLaunch(g, h->stream), "cudaGraphLaunch"))) return rc;
        if (h->precision == 1) h->cur ^= 1;
        h->launches += h->per_iter;
    }
    return TNS_OK;
}

int check_status(tns_handle* h) {
    int rc;
    if ((rc = h->cuda(cudaGetLastError(), "kernel launch"))) return rc;
    if ((rc = h->cuda(cudaMemcpyAsync(h->status_host, h->status.p, 4, cudaMemcpyDeviceToHost, h->stream),
                      "cudaMemcpyAsync")))
        return rc;
    if ((rc = h->cuda(cudaStreamSynchronize(h->stream), "cudaStreamSynchronize"))) return rc;
    if (h->cdiff_pending) {
        // the record of tns_enqueue_monitored has arrived: the floor tns_run applies
        for (int m = 0; m < 5; m++) {
            const double init = m < 4 ? 1.0e-10 : 1.0e-20;  // constants.f90:44-45
            const double v = h->cdiff_pending[m];
            h->cdiff_pending[m] = v >= init ? v : init;
        }
        h->cdiff_pending = nullptr;
    }
    if (*h->status_host & 1u) return h->fail(TNS_ERR_NONFINITE, "state became non-finite (NaN/Inf)");
    if (*h->status_host & 2u)
        return h->fail(TNS_ERR_CUDA, "a stage tile's static-data copy did not complete in its bounded wait");
    return TNS_OK;
}

}  // namespace

int tns_enqueue(tns_handle* h, int niter) {
    if (!h) return TNS_ERR_ARG;
    if (!h->have_state) return h->fail(TNS_ERR_STATE, "tns_enqueue: no state uploaded");
    if (niter <= 0) return TNS_OK;
    const int rc = enqueue_plain(h, niter);
    if (!rc) h->have_run = true;
    return rc;
}

int tns_prepare(tns_handle* h) {
    if (!h) return TNS_ERR_ARG;
    if (!h->have_state) return h->fail(TNS_ERR_STATE, "tns_prepare: no state uploaded");
    if (h->profile) return TNS_OK;
    int rc;
    if ((rc = ensure_graph(h)) || (rc = ensure_block_graph(h))) return rc;
    const long long per = h->per_iter;
    const bool mixed = h->precision == 1;
    for (int par = 0; par < (mixed ? 2 : 1); par++) {
        cudaGraphExec_t* g = mixed ? &h->graph_mon_mx[par] : &h->graph_mon;
        if (*g) continue;
        if ((rc = capture(h, g, mixed, par, true))) return rc;
        h->per_iter_mon = h->per_iter;
    }
    h->per_iter = per;
    return TNS_OK;
}

int tns_synchronize(tns_handle* h) {
    if (!h) return TNS_ERR_ARG;
    return check_status(h);
}

int tns_enqueue_monitored(tns_handle* h, double* cdiff) {
    if (!h || !cdiff) return TNS_ERR_ARG;
    if (!h->have_state) return h->fail(TNS_ERR_STATE, "tns_enqueue_monitored: no state uploaded");
    if (!page_locked(cdiff)) return h->fail(TNS_ERR_ARG, "tns_enqueue_monitored: cdiff is not page-locked");
    if (h->cdiff_pending)
        return h->fail(TNS_ERR_STATE, "tns_enqueue_monitored: the previous record was not synchronised");
    int rc;
    if ((rc = enqueue_monitored(h))) return rc;
    // the five maxima as IEEE bit patterns: a non-negative double orders like its bits
    if ((rc = h->cuda(cudaMemcpyAsync(cdiff, h->cdiff.p, 5 * sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                      h->stream), "cudaMemcpyAsync")))
        return rc;
    h->cdiff_pending = cdiff;
    h->have_run = true;
    return TNS_OK;
}

int tns_run(tns_handle* h, int niter, int monitor_every, double* cdiff_out, int max_records,
            int* n_records) {
    if (!h) return TNS_ERR_ARG;
    if (n_records) *n_records = 0;
    if (!h->have_state) return h->fail(TNS_ERR_STATE, "tns_run: no state uploaded");
    if (niter <= 0) return TNS_OK;
    int nrec = 0, rc;
    for (int it = 1; it <= niter;) {
        // run unmonitored iterations up to the next monitored one as one batch
        int next = (monitor_every > 0) ? ((it + monitor_every - 1) / monitor_every) * monitor_every
                                       : niter + 1;
        if (next > niter) next = niter + 1;
        if (next > it) {
            if ((rc = enqueue_plain(h, next - it))) return rc;
            it = next;
            if (it > niter) break;
        }
        if ((rc = enqueue_monitored(h))) return rc;  // iteration `it` is monitored
        {
            unsigned long long bits[5];
            if ((rc = h->cuda(cudaMemcpyAsync(bits, h->cdiff.p, sizeof bits, cudaMemcpyDeviceToHost, h->stream),
                              "cudaMemcpyAsync")))
                return rc;
            if ((rc = h->cuda(cudaStreamSynchronize(h->stream), "cudaStreamSynchronize"))) return rc;
            if (cdiff_out && nrec < max_records) {
                for (int m = 0; m < 5; m++) {
                    double v;
                    std::memcpy(&v, &bits[m], 8);
                    const double init = m < 4 ? 1.0e-10 : 1.0e-20;  // constants.f90:44-45
                    cdiff_out[nrec * 5 + m] = v >= init ? v : init;
                }
            }
            nrec++;
        }
        it++;
    }
    h->have_run = true;
    if (n_records) *n_records = std::min(nrec, max_records);
    return check_status(h);
}

int tns_download_state(tns_handle* h, double* c1, double* c2, double* c3, double* c4, double* c5) {
    if (!h || !c1 || !c2 || !c3 || !c4 || !c5) return TNS_ERR_ARG;
    if (!h->have_state) return h->fail(TNS_ERR_STATE, "tns_download_state: no state");
    const size_t nc = h->ncell();
    double* dst[5] = {c1, c2, c3, c4, c5};
    int rc;
    const double* src = h->state();
    if (!h->identity) {
        tns::launch_renumber(h->dcell_of.p, src, h->renum.p, nc, false, h->stream);
        if ((rc = h->cuda(cudaGetLastError(), "kernel launch"))) return rc;
        src = h->renum.p;
    }
    bool direct = true;
    for (int m = 0; m < 5 && direct; m++) direct = page_locked(dst[m]);
    if (direct) {
        // page-locked caller arrays: one DMA per component, no staging copy
        for (int m = 0; m < 5; m++)
            if ((rc = h->cuda(cudaMemcpyAsync(dst[m], src + m * nc, nc * 8, cudaMemcpyDeviceToHost, h->stream),
                              "cudaMemcpyAsync")))
                return rc;
        return h->cuda(cudaStreamSynchronize(h->stream), "cudaStreamSynchronize");
    }
    rc = h->cuda(cudaMemcpyAsync(h->pinned, src, 5 * nc * 8, cudaMemcpyDeviceToHost, h->stream), "cudaMemcpyAsync");
    if (rc || (rc = h->cuda(cudaStreamSynchronize(h->stream), "cudaStreamSynchronize"))) return rc;
    for (int m = 0; m < 5; m++) std::memcpy(dst[m], h->pinned + m * nc, nc * 8);
    return TNS_OK;
}

}  // extern "C"

namespace {
// U, V, T, P of the last stage's input for cells and ghosts into h->primout (device).
int fill_primitives(tns_handle* h) {
    if (h->unstructured) return tns_rt::umesh_primitives(h);
    const size_t nc = h->ncell(), ng = (size_t)h->M.nghosts(), nt = nc + ng;
    int rc;
    if (!h->primout.p && (rc = h->cuda(h->primout.alloc(4 * nt), "cudaMalloc"))) return rc;
    const int np = (int)h->port_ghosts.size();
    if (h->precision == 1) {
        // stage 4 read (previous state + dQ_B)
        if (np) tns::launch_gport_mx(h->P, h->M, h->other_state(), h->dqb.p, h->ports.p, np, h->gport.p, h->stream);
        tns::launch_prim_out_mx(h->P, h->M, h->other_state(), h->dqb.p, h->primout.p, h->stream);
    } else {
        // stage 4 read B: recompute its primitives and ghost states from B
        if (np) tns::launch_gport(h->P, h->M, h->qb.p, h->ports.p, np, h->gport.p, h->stream);
        tns::launch_prim_out(h->P, h->M, h->qb.p, h->primout.p, h->stream);
    }
    return h->cuda(cudaGetLastError(), "kernel launch");
}
}  // namespace

extern "C" {

int tns_download_primitives(tns_handle* h, double* u, double* v, double* t, double* p) {
    if (!h || !u || !v || !t || !p) return TNS_ERR_ARG;
    if (!h->have_run) return h->fail(TNS_ERR_STATE, "tns_download_primitives: no iteration has run");
    const size_t nc = h->ncell(), ng = h->unstructured ? (size_t)h->nghosts : (size_t)h->M.nghosts(), nt = nc + ng;
    int rc;
    if ((rc = fill_primitives(h))) return rc;
    std::vector<double> hb(4 * nt);
    rc = h->cuda(cudaMemcpyAsync(hb.data(), h->primout.p, 4 * nt * 8, cudaMemcpyDeviceToHost, h->stream),
                 "cudaMemcpyAsync");
    if (rc || (rc = h->cuda(cudaStreamSynchronize(h->stream), "cudaStreamSynchronize"))) return rc;
    double* dst[4] = {u, v, t, p};
    for (int f = 0; f < 4; f++) {
        const double* src = hb.data() + f * nt;
        for (size_t k = 0; k < nc; k++) dst[f][h->cell_of[k]] = src[k];
        for (size_t g = 0; g < ng; g++) dst[f][h->ghost_id[h->ghost_line[g]] - 1] = src[nc + g];
    }
    return TNS_OK;
}

int tns_node_averages(tns_handle* h, double* pn, double* un, double* vn, double* tn) {
    if (!h || !pn || !un || !vn || !tn) return TNS_ERR_ARG;
    if (!h->have_run) return h->fail(TNS_ERR_STATE, "tns_node_averages: no iteration has run");
    int rc;
    const size_t nnode = h->unstructured ? (size_t)h->nods : (size_t)(h->ni + 1) * (h->nj + 1);
    DevBuf<double> dn;
    if ((rc = h->cuda(dn.alloc(4 * nnode), "cudaMalloc"))) return rc;
    if (h->unstructured) {
        if ((rc = tns_rt::umesh_node_averages(h, dn.p))) {
            dn.release();
            return rc;
        }
    } else {
        if ((rc = fill_primitives(h))) {
            dn.release();
            return rc;
        }
        tns::launch_node_average(h->M, h->primout.p, dn.p, h->stream);
    }
    std::vector<double> hb(4 * nnode);
    rc = h->cuda(cudaMemcpyAsync(hb.data(), dn.p, 4 * nnode * 8, cudaMemcpyDeviceToHost, h->stream),
                 "cudaMemcpyAsync");
    if (!rc) rc = h->cuda(cudaStreamSynchronize(h->stream), "cudaStreamSynchronize");
    dn.release();
    if (rc) return rc;
    double* dst[4] = {pn, un, vn, tn};
    for (int f = 0; f < 4; f++)
        for (size_t k = 0; k < nnode; k++) dst[f][h->node_of[k] - 1] = hb[f * nnode + k];
    return TNS_OK;
}

}  // extern "C"

namespace {
// Boundary-face sums (mode 0: out[4]; mode 1: out[2]) of the last stage's state.
int boundary_sums(tns_handle* h, int type, int side, int mode, double* out, int nout) {
    int rc;
    DevBuf<double> acc;
    if ((rc = h->cuda(acc.alloc(4), "cudaMalloc"))) return rc;
    cudaMemsetAsync(acc.p, 0, 4 * sizeof(double), h->stream);
    if (h->unstructured) {
        rc = tns_rt::umesh_boundary_sums(h, type, side, mode, acc.p);
    } else if (!(rc = fill_primitives(h))) {
        tns::launch_boundary_sums(h->P, h->M, h->primout.p, type, side, mode, acc.p, h->stream);
    }
    if (!rc)
        rc = h->cuda(cudaMemcpyAsync(out, acc.p, nout * sizeof(double), cudaMemcpyDeviceToHost, h->stream),
                     "cudaMemcpyAsync");
    if (!rc) rc = h->cuda(cudaStreamSynchronize(h->stream), "cudaStreamSynchronize");
    acc.release();
    return rc;
}
}  // namespace

extern "C" {

int tns_boundary_integrals(tns_handle* h, int type, int side, double out[4]) {
    if (!h || !out || type < 0 || type > 7 || side < 0 || side > 4) return TNS_ERR_ARG;
    if (!h->have_run) return h->fail(TNS_ERR_STATE, "tns_boundary_integrals: no iteration has run");
    return boundary_sums(h, type, side, 0, out, 4);
}

int tns_total_pressure_sums(tns_handle* h, int type, int side, double out[2]) {
    if (!h || !out || type < 0 || type > 7 || side < 0 || side > 4) return TNS_ERR_ARG;
    if (!h->have_run) return h->fail(TNS_ERR_STATE, "tns_total_pressure_sums: no iteration has run");
    return boundary_sums(h, type, side, 1, out, 2);
}

int tns_boundary_face_states(tns_handle* h, double* out) {
    if (!h || !out) return TNS_ERR_ARG;
    if (!h->have_run) return h->fail(TNS_ERR_STATE, "tns_boundary_face_states: no iteration has run");
    const size_t ng = (size_t)h->nghosts;
    if (ng == 0) return TNS_OK;
    int rc;
    DevBuf<double> dv;
    if ((rc = h->cuda(dv.alloc(5 * ng), "cudaMalloc"))) return rc;
    if (h->unstructured) {
        rc = tns_rt::umesh_face_states(h, dv.p);
    } else if (!(rc = fill_primitives(h))) {
        tns::launch_face_states(h->P, h->M, h->primout.p, dv.p, h->stream);
    }
    std::vector<double> hb(5 * ng);
    if (!rc)
        rc = h->cuda(cudaMemcpyAsync(hb.data(), dv.p, 5 * ng * 8, cudaMemcpyDeviceToHost, h->stream), "cudaMemcpyAsync");
    if (!rc) rc = h->cuda(cudaStreamSynchronize(h->stream), "cudaStreamSynchronize");
    dv.release();
    if (rc) return rc;
    // device ghost order -> bc.in line order
    for (int f = 0; f < 5; f++)
        for (size_t g = 0; g < ng; g++) out[f * ng + h->ghost_line[g]] = hb[f * ng + g];
    return TNS_OK;
}

int tns_debug_fetch(tns_handle* h, int which, double* out) {
    if (!h || !out || which < 0 || which > 2) return TNS_ERR_ARG;
    if (!h->have_run) return h->fail(TNS_ERR_STATE, "tns_debug_fetch: no iteration has run");
    const size_t nc = h->ncell();
    const int cnt = which == 0 ? 5 : which == 1 ? 4 : 1;
    const double* src = which == 0 ? h->d.p : which == 1 ? h->vis.p : h->dt.p;
    std::vector<double> hb(cnt * nc);
    if (h->precision == 1 && !(which == 2 && !h->P.local)) {
        const float* fs = which == 0 ? h->df.p : which == 1 ? h->visf.p : h->dtf.p;
        std::vector<float> fb(cnt * nc);
        int rc = h->cuda(cudaMemcpyAsync(fb.data(), fs, cnt * nc * 4, cudaMemcpyDeviceToHost, h->stream),
                         "cudaMemcpyAsync");
        if (rc || (rc = h->cuda(cudaStreamSynchronize(h->stream), "cudaStreamSynchronize"))) return rc;
        for (size_t k = 0; k < hb.size(); k++) hb[k] = fb[k];
    } else if (which == 2 && !h->P.local) {
        double dm = 0;
        int rc = h->cuda(cudaMemcpy(&dm, h->dtmin.p, 8, cudaMemcpyDeviceToHost), "cudaMemcpy");
        if (rc) return rc;
        std::fill(hb.begin(), hb.end(), dm);
    } else {
        int rc = h->cuda(cudaMemcpyAsync(hb.data(), src, cnt * nc * 8, cudaMemcpyDeviceToHost, h->stream),
                         "cudaMemcpyAsync");
        if (rc || (rc = h->cuda(cudaStreamSynchronize(h->stream), "cudaStreamSynchronize"))) return rc;
    }
    for (int f = 0; f < cnt; f++)
        for (size_t k = 0; k < nc; k++) out[f * nc + h->cell_of[k]] = hb[f * nc + k];
    return TNS_OK;
}

int tns_set_stream(tns_handle* h, void* stream) {
    if (!h) return TNS_ERR_ARG;
    cudaStream_t s = stream ? (cudaStream_t)stream : h->own;
    if (s != h->stream) {
        cudaStreamSynchronize(h->stream);
        h->stream = s;
    }
    return TNS_OK;
}

int tns_profile(tns_handle* h, int enable) {
    if (!h) return TNS_ERR_ARG;
    h->profile = enable != 0;
    if (h->profile)
        for (int k = 0; k < K_NKERNEL; k++) { h->kms[k] = 0; h->kcount[k] = 0; }
    return TNS_OK;
}

int tns_kernel_times(tns_handle* h, int kernel, double* ms, long long* launches) {
    if (!h || kernel < 0 || kernel >= K_NKERNEL) return TNS_ERR_ARG;
    if (ms) *ms = h->kms[kernel];
    if (launches) *launches = h->kcount[kernel];
    return TNS_OK;
}

long long tns_launch_count(tns_handle* h) { return h ? h->launches : -1; }

int tns_debug_math(int fn, long long n, const double* a, const double* b, double* out) {
    if (fn < 0 || fn > 2 || n < 0 || (n > 0 && (!a || !out || (fn == 1 && !b)))) return TNS_ERR_ARG;
    if (n == 0) return TNS_OK;
    double* d = nullptr;
    const size_t bytes = (size_t)n * sizeof(double);
    if (cudaMalloc((void**)&d, 3 * bytes) != cudaSuccess) return TNS_ERR_CUDA;
    cudaError_t e = cudaMemcpy(d, a, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && fn == 1) e = cudaMemcpy(d + n, b, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        tns::launch_debug_math(fn, n, d, d + n, d + 2 * n, 0);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * n, bytes, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? TNS_OK : TNS_ERR_CUDA;
}

const char* tns_last_error(tns_handle* h) { return h ? h->err.c_str() : "null handle"; }

}  // extern "C"

// ----------------------------------------------------------- allocation-free time step
//
// Scratch of tns_time_step_noalloc, in device memory that exists as soon as the library
// is loaded: one partial minimum per block, then the blocks' completion counter.
// Every GPU that loads the library keeps this array until the process exits.
static __device__ __align__(256) unsigned char g_step_scratch[TNS_NOALLOC_MAX_BLOCKS * sizeof(double) + 256];

namespace {
std::mutex g_step_mutex;
void* g_step_ptr[256] = {};  // device address of g_step_scratch, per device ordinal
}  // namespace

extern "C" {

int tns_time_step_noalloc(const double* d_q, const double* d_cfldl, long long ncell,
                          const tns_params* params, double* d_dt, double* d_dtmin, void* stream) {
    if (!d_q || !d_cfldl || !params || !d_dt || !d_dtmin || ncell <= 0) return TNS_ERR_ARG;
    const long long per_block = 256LL * TNS_NOALLOC_CELLS_PER_THREAD;
    const long long nblocks = (ncell + per_block - 1) / per_block;
    if (nblocks > TNS_NOALLOC_MAX_BLOCKS) return TNS_ERR_TOO_LARGE;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) return TNS_ERR_CUDA;
    void* base = nullptr;
    {
        // set-up, once per device: the host-side name of the array is not a device
        // address, so ask the runtime for it with this device current
        std::lock_guard<std::mutex> lock(g_step_mutex);
        if (!g_step_ptr[dev]) {
            void* p = nullptr;
            if (cudaGetSymbolAddress(&p, g_step_scratch) != cudaSuccess || !p) {
                cudaGetLastError();
                return TNS_ERR_CUDA;
            }
            g_step_ptr[dev] = p;
        }
        base = g_step_ptr[dev];
    }
    double* partial = static_cast<double*>(base);
    unsigned int* counter =
        reinterpret_cast<unsigned int*>(static_cast<unsigned char*>(base) + TNS_NOALLOC_MAX_BLOCKS * sizeof(double));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const Params P = make_params(*params);
    if (ncell <= tns::STEP_CLUSTER_CELLS) {  // (after the set-up, which a later call may rely on)
        tns::launch_time_step_cluster(P, d_q, d_cfldl, ncell, d_dt, d_dtmin, s);
        return cudaGetLastError() == cudaSuccess ? TNS_OK : TNS_ERR_CUDA;
    }
    // the array keeps whatever the previous call left: the counter must start at zero
    if (cudaMemsetAsync(counter, 0, sizeof(unsigned int), s) != cudaSuccess) return TNS_ERR_CUDA;
    tns::launch_time_step_scratch(P, d_q, d_cfldl, ncell, d_dt, partial, counter, d_dtmin,
                                  (int)nblocks, s);
    return cudaGetLastError() == cudaSuccess ? TNS_OK : TNS_ERR_CUDA;
}

void tns_destroy(tns_handle* h) {
    if (!h) return;
    if (h->stream) cudaStreamSynchronize(h->stream);
    tns_rt::adjoint_release(h);
    tns_rt::umesh_release(h);
    if (h->graph) cudaGraphExecDestroy(h->graph);
    for (auto g : h->graph_mx)
        if (g) cudaGraphExecDestroy(g);
    for (auto g : h->graph_block)
        if (g) cudaGraphExecDestroy(g);
    for (auto g : h->graph_mon_mx)
        if (g) cudaGraphExecDestroy(g);
    if (h->graph_mon) cudaGraphExecDestroy(h->graph_mon);
    h->qa2.release(); h->dqb.release(); h->dqc.release(); h->df.release(); h->visf.release(); h->ef.release();
    h->dtf.release(); h->tref.release(); h->dcell_of.release(); h->renum.release();
    for (auto* b : {&h->x, &h->y, &h->cfldl, &h->gxc, &h->gyc, &h->ginj, &h->gport, &h->qa, &h->qb,
                    &h->qc, &h->d, &h->vis, &h->dt, &h->dtmin, &h->partial, &h->primout, &h->cvol, &h->vcfl, &h->e,
                    &h->wport, &h->wport_i, &h->stile, &h->vtile})
        b->release();
    h->grec.release(); h->bnode.release(); h->gtype.release(); h->grank.release(); h->ports.release();
    h->counter.release(); h->status.release(); h->cdiff.release();
    if (h->pinned) cudaFreeHost(h->pinned);
    if (h->status_host) cudaFreeHost(h->status_host);
    for (auto& e : h->ev)
        if (e) cudaEventDestroy(e);
    if (h->fork) cudaEventDestroy(h->fork);
    if (h->join) cudaEventDestroy(h->join);
    if (h->side) {
        cudaStreamSynchronize(h->side);
        cudaStreamDestroy(h->side);
    }
    if (h->own) cudaStreamDestroy(h->own);
    delete h;
}

}  // extern "C"
