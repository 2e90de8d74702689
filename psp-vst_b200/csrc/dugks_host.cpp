// Host-side preparation of the DUGKS step: OpenFOAM mesh geometry,
// surface-interpolation weights, least-squares gradient vectors, and the
// cell and face order the device passes work in.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>

#include "dugks_internal.h"

namespace {

inline double dot3(const double* a, const double* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
inline double magsqr3(const double* a) { return dot3(a, a); }

// symmetric tensor (xx xy xz yy yz zz) inverse by the adjugate
void sym_inverse(const double* a, double* r) {
    const double xx = a[0], xy = a[1], xz = a[2], yy = a[3], yz = a[4], zz = a[5];
    const double det = xx * yy * zz + xy * yz * xz + xz * xy * yz - xx * yz * yz - xy * xy * zz - xz * yy * xz;
    r[0] = (yy * zz - yz * yz) / det;
    r[1] = (xz * yz - xy * zz) / det;
    r[2] = (xy * yz - xz * yy) / det;
    r[3] = (xx * zz - xz * xz) / det;
    r[4] = (xy * xz - xx * yz) / det;
    r[5] = (xx * yy - xy * xy) / det;
}

void sym_apply(const double* t, const double* d, double* o) {
    o[0] = t[0] * d[0] + t[1] * d[1] + t[2] * d[2];
    o[1] = t[1] * d[0] + t[3] * d[1] + t[4] * d[2];
    o[2] = t[2] * d[0] + t[4] * d[1] + t[5] * d[2];
}

}  // namespace

extern "C" int dugks_mesh_geometry(int32_t n_points, const double* p, int32_t n_faces, const int64_t* fo,
                                   const int64_t* fp, const int64_t* owner, int32_t n_internal,
                                   const int64_t* neighbour, int32_t n_cells, double* Cf, double* Sf, double* C,
                                   double* V) {
    if (!p || !fo || !fp || !owner || (n_internal && !neighbour) || !Cf || !Sf || !C || !V || n_cells <= 0 ||
        n_faces < n_internal || n_points <= 0)
        return DUGKS_ERR_ARG;
    // face centres and area vectors: triangle fan about the point average
    for (int32_t f = 0; f < n_faces; ++f) {
        const int64_t b = fo[f], e = fo[f + 1];
        const int np = static_cast<int>(e - b);
        if (np < 3) return DUGKS_ERR_ARG;
        for (int64_t k = b; k < e; ++k)
            if (fp[k] < 0 || fp[k] >= n_points) return DUGKS_ERR_ARG;
        if (np == 3) {
            const double *a = p + 3 * fp[b], *bb = p + 3 * fp[b + 1], *c = p + 3 * fp[b + 2];
            const double u[3] = {bb[0] - a[0], bb[1] - a[1], bb[2] - a[2]};
            const double v[3] = {c[0] - a[0], c[1] - a[1], c[2] - a[2]};
            for (int k = 0; k < 3; ++k) Cf[3 * f + k] = (1.0 / 3.0) * (a[k] + bb[k] + c[k]);
            Sf[3 * f + 0] = 0.5 * (u[1] * v[2] - u[2] * v[1]);
            Sf[3 * f + 1] = 0.5 * (u[2] * v[0] - u[0] * v[2]);
            Sf[3 * f + 2] = 0.5 * (u[0] * v[1] - u[1] * v[0]);
            continue;
        }
        double fc[3] = {0, 0, 0};
        for (int i = 0; i < np; ++i)
            for (int k = 0; k < 3; ++k) fc[k] += p[3 * fp[b + i] + k];
        for (int k = 0; k < 3; ++k) fc[k] /= np;
        double sn[3] = {0, 0, 0}, sa = 0, sac[3] = {0, 0, 0};
        for (int i = 0; i < np; ++i) {
            const double* pi = p + 3 * fp[b + i];
            const double* pn = p + 3 * fp[b + (i + 1) % np];
            double c[3], u[3], v[3];
            for (int k = 0; k < 3; ++k) {
                c[k] = pi[k] + pn[k] + fc[k];
                u[k] = pn[k] - pi[k];
                v[k] = fc[k] - pi[k];
            }
            const double n[3] = {u[1] * v[2] - u[2] * v[1], u[2] * v[0] - u[0] * v[2], u[0] * v[1] - u[1] * v[0]};
            const double a = std::sqrt(magsqr3(n));
            for (int k = 0; k < 3; ++k) {
                sn[k] += n[k];
                sac[k] += a * c[k];
            }
            sa += a;
        }
        for (int k = 0; k < 3; ++k) {
            Cf[3 * f + k] = sa < 1e-150 ? fc[k] : (1.0 / 3.0) * sac[k] / sa;
            Sf[3 * f + k] = sa < 1e-150 ? 0.0 : 0.5 * sn[k];
        }
    }
    // cell centres and volumes: face pyramids about the face-centre average
    std::vector<double> est(3 * static_cast<size_t>(n_cells), 0.0);
    std::vector<int> nf(n_cells, 0);
    for (int32_t f = 0; f < n_faces; ++f) {
        if (owner[f] < 0 || owner[f] >= n_cells) return DUGKS_ERR_ARG;
        for (int k = 0; k < 3; ++k) est[3 * owner[f] + k] += Cf[3 * f + k];
        nf[owner[f]]++;
    }
    for (int32_t f = 0; f < n_internal; ++f) {
        if (neighbour[f] < 0 || neighbour[f] >= n_cells) return DUGKS_ERR_ARG;
        for (int k = 0; k < 3; ++k) est[3 * neighbour[f] + k] += Cf[3 * f + k];
        nf[neighbour[f]]++;
    }
    for (int32_t c = 0; c < n_cells; ++c) {
        if (nf[c] == 0) return DUGKS_ERR_ARG;
        for (int k = 0; k < 3; ++k) est[3 * c + k] /= nf[c];
    }
    std::fill(C, C + 3 * static_cast<size_t>(n_cells), 0.0);
    std::fill(V, V + n_cells, 0.0);
    auto pyramid = [&](int32_t f, int64_t c, double sgn) {
        const double d[3] = {sgn * (Cf[3 * f] - est[3 * c]), sgn * (Cf[3 * f + 1] - est[3 * c + 1]),
                             sgn * (Cf[3 * f + 2] - est[3 * c + 2])};
        const double pyr3 = dot3(Sf + 3 * f, d);
        for (int k = 0; k < 3; ++k) C[3 * c + k] += pyr3 * ((3.0 / 4.0) * Cf[3 * f + k] + (1.0 / 4.0) * est[3 * c + k]);
        V[c] += pyr3;
    };
    for (int32_t f = 0; f < n_faces; ++f) pyramid(f, owner[f], 1.0);
    for (int32_t f = 0; f < n_internal; ++f) pyramid(f, neighbour[f], -1.0);
    for (int32_t c = 0; c < n_cells; ++c) {
        if (std::fabs(V[c]) > 1e-300) {
            for (int k = 0; k < 3; ++k) C[3 * c + k] /= V[c];
        } else {
            for (int k = 0; k < 3; ++k) C[3 * c + k] = est[3 * c + k];
        }
        V[c] *= (1.0 / 3.0);
    }
    return DUGKS_OK;
}

namespace dugks {

int set_error(dugks_handle* h, int code, const std::string& msg) {
    if (h) h->last_error = msg;
    return code;
}

// surfaceInterpolation::makeWeights / makeDeltaCoeffs and the weighted
// least-squares vectors of zeroBoundaryVectors.C:90-221 with the
// non-coupled boundary terms restored (stock leastSquares).  The boundary
// d-vector is fvPatch::delta() for non-coupled patches, n (n . (Cf - C)).
void compute_weights_and_ls(dugks_handle* h, int weighting) {
    const int nC = h->nC, nIF = h->nIF, nBF = h->nBF;
    const int nF = nIF + nBF;
    std::vector<double> magSf(nF);
    for (int f = 0; f < nF; ++f) magSf[f] = std::sqrt(magsqr3(&h->Sf[3 * f]));
    h->weights.assign(nIF, 0.0);
    h->dc.assign(nIF, 0.0);
    for (int f = 0; f < nIF; ++f) {
        const double* S = &h->Sf[3 * f];
        const double* co = &h->C[3 * h->owner[f]];
        const double* cn = &h->C[3 * h->neighbour[f]];
        const double* cf = &h->Cf[3 * f];
        const double a[3] = {cf[0] - co[0], cf[1] - co[1], cf[2] - co[2]};
        const double b[3] = {cn[0] - cf[0], cn[1] - cf[1], cn[2] - cf[2]};
        const double so = std::fabs(dot3(S, a)), sn = std::fabs(dot3(S, b));
        h->weights[f] = sn / (so + sn);
        const double d[3] = {cn[0] - co[0], cn[1] - co[1], cn[2] - co[2]};
        h->dc[f] = 1.0 / std::sqrt(magsqr3(d));
    }
    auto face_factor = [&](int f, double wgt, const double* d, bool own_side, bool boundary) {
        if (weighting == DUGKS_LS_MAGSF) {
            const double c = magSf[f] / magsqr3(d);
            if (boundary) return c;
            return own_side ? (1 - wgt) * c : wgt * c;
        }
        if (weighting == DUGKS_LS_INVDIST) return 1.0 / magsqr3(d);
        return 1.0;
    };
    std::vector<double> dd(6 * static_cast<size_t>(nC), 0.0);
    for (int f = 0; f < nIF; ++f) {
        const int64_t o = h->owner[f], n = h->neighbour[f];
        const double d[3] = {h->C[3 * n] - h->C[3 * o], h->C[3 * n + 1] - h->C[3 * o + 1],
                             h->C[3 * n + 2] - h->C[3 * o + 2]};
        const double sq[6] = {d[0] * d[0], d[0] * d[1], d[0] * d[2], d[1] * d[1], d[1] * d[2], d[2] * d[2]};
        const double fo = face_factor(f, h->weights[f], d, true, false);
        const double fn = face_factor(f, h->weights[f], d, false, false);
        for (int k = 0; k < 6; ++k) {
            dd[6 * o + k] += fo * sq[k];
            dd[6 * n + k] += fn * sq[k];
        }
    }
    std::vector<double> bdelta(3 * static_cast<size_t>(nBF));
    for (int b = 0; b < nBF; ++b) {
        const int f = nIF + b;
        const int64_t o = h->owner[f];
        const double* S = &h->Sf[3 * f];
        const double nrm[3] = {S[0] / magSf[f], S[1] / magSf[f], S[2] / magSf[f]};
        const double cfc[3] = {h->Cf[3 * f] - h->C[3 * o], h->Cf[3 * f + 1] - h->C[3 * o + 1],
                               h->Cf[3 * f + 2] - h->C[3 * o + 2]};
        const double dn = dot3(nrm, cfc);
        double* d = &bdelta[3 * b];
        for (int k = 0; k < 3; ++k) d[k] = nrm[k] * dn;
        const double sq[6] = {d[0] * d[0], d[0] * d[1], d[0] * d[2], d[1] * d[1], d[1] * d[2], d[2] * d[2]};
        const double fb = face_factor(f, 1.0, d, true, true);
        for (int k = 0; k < 6; ++k) dd[6 * o + k] += fb * sq[k];
    }
    // OpenFOAM's inverse of a symmTensorField drops the directions whose
    // diagonal is negligible in the first tensor (2-D and 1-D meshes)
    bool rm[3] = {false, false, false};
    if (nC > 0) {
        const double* t = dd.data();
        const double scale = t[0] * t[0] + 2 * t[1] * t[1] + 2 * t[2] * t[2] + t[3] * t[3] + 2 * t[4] * t[4] + t[5] * t[5];
        rm[0] = t[0] * t[0] / scale < 1e-15;
        rm[1] = t[3] * t[3] / scale < 1e-15;
        rm[2] = t[5] * t[5] / scale < 1e-15;
    }
    std::vector<double> inv(6 * static_cast<size_t>(nC));
    for (int c = 0; c < nC; ++c) {
        double a[6];
        std::memcpy(a, &dd[6 * c], sizeof a);
        if (rm[0]) a[0] += 1.0;
        if (rm[1]) a[3] += 1.0;
        if (rm[2]) a[5] += 1.0;
        sym_inverse(a, &inv[6 * c]);
        if (rm[0]) inv[6 * c] -= 1.0;
        if (rm[1]) inv[6 * c + 3] -= 1.0;
        if (rm[2]) inv[6 * c + 5] -= 1.0;
    }
    h->lsP.assign(3 * static_cast<size_t>(nIF), 0.0);
    h->lsN.assign(3 * static_cast<size_t>(nIF), 0.0);
    h->lsB.assign(3 * static_cast<size_t>(nBF), 0.0);
    for (int f = 0; f < nIF; ++f) {
        const int64_t o = h->owner[f], n = h->neighbour[f];
        const double d[3] = {h->C[3 * n] - h->C[3 * o], h->C[3 * n + 1] - h->C[3 * o + 1],
                             h->C[3 * n + 2] - h->C[3 * o + 2]};
        const double fo = face_factor(f, h->weights[f], d, true, false);
        const double fn = -face_factor(f, h->weights[f], d, false, false);
        double a[3], b[3];
        sym_apply(&inv[6 * o], d, a);
        sym_apply(&inv[6 * n], d, b);
        for (int k = 0; k < 3; ++k) {
            h->lsP[3 * f + k] = fo * a[k];
            h->lsN[3 * f + k] = fn * b[k];
        }
    }
    for (int b = 0; b < nBF; ++b) {
        const int f = nIF + b;
        const double* d = &bdelta[3 * b];
        const double fb = face_factor(f, 1.0, d, true, true);
        double a[3];
        sym_apply(&inv[6 * h->owner[f]], d, a);
        for (int k = 0; k < 3; ++k) h->lsB[3 * b + k] = fb * a[k];
    }
}

}  // namespace dugks

namespace {

// Recursive coordinate bisection: cut the cell set along the longest axis
// of its bounding box so that the first part holds a whole number of tiles,
// until every part is one tile.  Consecutive tiles are neighbours in space.
// by_index: within a tile the caller's order stays, whose runs along a grid
// line make the neighbours of consecutive cells consecutive.
void rcb_order(const std::vector<double>& C, std::vector<int32_t>& idx, size_t b, size_t e, int tile, bool by_index) {
    const size_t n = e - b;
    if (n <= static_cast<size_t>(tile)) {
        if (by_index) std::sort(idx.begin() + b, idx.begin() + e);
        return;
    }
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (size_t i = b; i < e; ++i)
        for (int k = 0; k < 3; ++k) {
            lo[k] = std::min(lo[k], C[3 * idx[i] + k]);
            hi[k] = std::max(hi[k], C[3 * idx[i] + k]);
        }
    int ax = 0;
    for (int k = 1; k < 3; ++k)
        if (hi[k] - lo[k] > hi[ax] - lo[ax]) ax = k;
    const size_t nt = (n + tile - 1) / tile;
    const size_t nl = (nt / 2) * static_cast<size_t>(tile);
    std::stable_sort(idx.begin() + b, idx.begin() + e, [&](int32_t p, int32_t q) { return C[3 * p + ax] < C[3 * q + ax]; });
    rcb_order(C, idx, b, b + nl, tile, by_index);
    rcb_order(C, idx, b + nl, e, tile, by_index);
}

// Greedy tile boundaries over the RCB cell order: each tile takes the next
// cells in order while it keeps at most kMaxTile L0 cells, kMaxLocal cells
// with its ring and kMaxItems faces.  Tiles end where the ring, not a fixed size, runs
// out.
std::vector<int32_t> greedy_bounds(int nC, int nIF, const std::vector<int64_t>& owner,
                                   const std::vector<int64_t>& neighbour, const std::vector<int32_t>& cfo,
                                   const std::vector<int32_t>& cfl, const std::vector<int32_t>& perm,
                                   const std::vector<int32_t>& iperm) {
    std::vector<int32_t> bounds(1, 0);
    std::vector<unsigned char> in_l0(nC, 0);
    std::vector<int32_t> ring_cnt(nC, 0);  // L0 neighbours of a cell outside L0
    std::vector<int32_t> fresh;
    int b = 0, ring = 0, items = 0;
    // fn(n) for every face of renumbered cell c: n the renumbered cell on
    // the other side, -1 for a boundary face
    auto others = [&](int c, auto&& fn) {
        const int o = perm[c];
        for (int k = cfo[o]; k < cfo[o + 1]; ++k) {
            const int f = cfl[k];
            if (f < nIF) fn(iperm[owner[f] == o ? neighbour[f] : owner[f]]);
            else fn(-1);
        }
    };
    for (int c = 0; c < nC; ++c) {
        int d_items = 0, d_ring = ring_cnt[c] > 0 ? -1 : 0;
        fresh.clear();
        others(c, [&](int n) {
            if (n < 0) {
                ++d_items;
            } else if (!in_l0[n]) {
                ++d_items;
                if (ring_cnt[n] == 0 && std::find(fresh.begin(), fresh.end(), n) == fresh.end()) {
                    fresh.push_back(n);
                    ++d_ring;
                }
            }
        });
        const int n0 = c - b;
        const bool fits = n0 + 1 <= dugks::kMaxTile && n0 + 1 + ring + d_ring <= dugks::kMaxLocal &&
                          items + d_items <= dugks::kMaxItems;
        if (n0 > 0 && !fits) {
            // close the tile [b, c); cell c starts the next one
            for (int x = b; x < c; ++x) {
                in_l0[x] = 0;
                others(x, [&](int n) {
                    if (n >= 0) ring_cnt[n] = 0;
                });
            }
            bounds.push_back(c);
            b = c;
            ring = items = 0;
            --c;
            continue;
        }
        in_l0[c] = 1;
        items += d_items;
        ring += d_ring;
        others(c, [&](int n) {
            if (n >= 0 && !in_l0[n]) ++ring_cnt[n];
        });
    }
    bounds.push_back(nC);
    return bounds;
}

// whether every tile [bounds[i], bounds[i+1]) keeps the limits of greedy_bounds
bool tiles_fit(int nIF, const std::vector<int64_t>& owner, const std::vector<int64_t>& neighbour,
               const std::vector<int32_t>& cfo, const std::vector<int32_t>& cfl, const std::vector<int32_t>& perm,
               const std::vector<int32_t>& iperm, const std::vector<int32_t>& bounds) {
    std::vector<int32_t> seen(perm.size(), -1);
    for (size_t t = 0; t + 1 < bounds.size(); ++t) {
        const int b = bounds[t], e = bounds[t + 1];
        int ring = 0, items = 0;
        for (int c = b; c < e; ++c)
            for (int k = cfo[perm[c]]; k < cfo[perm[c] + 1]; ++k) {
                const int f = cfl[k];
                const int n = f >= nIF ? -1 : iperm[owner[f] == perm[c] ? neighbour[f] : owner[f]];
                const bool inside = n >= b && n < e;
                if (!inside || c < n) ++items;
                if (n >= 0 && !inside && seen[n] != static_cast<int>(t)) {
                    seen[n] = static_cast<int>(t);
                    ++ring;
                }
            }
        if (e - b + ring > dugks::kMaxLocal || items > dugks::kMaxItems) return false;
    }
    return true;
}

// Compact tiles of the mesh, of at most tile_cells cells (0: as large as the
// limits of greedy_bounds allow).  No kernel works tile by tile; dugks_layout
// reports them, and FP32 rows round one product by them (DevMesh::cface).
// Returns the tile of every (caller's) cell.
std::vector<int32_t> tile_cells_of(const dugks_handle* h, int tile_cells, dugks::Tiling& t) {
    const int nC = h->nC, nIF = h->nIF, nF = nIF + h->nBF;
    std::vector<int32_t> cfo(nC + 1, 0);
    for (int f = 0; f < nF; ++f) cfo[h->owner[f] + 1]++;
    for (int f = 0; f < nIF; ++f) cfo[h->neighbour[f] + 1]++;
    for (int c = 0; c < nC; ++c) cfo[c + 1] += cfo[c];
    std::vector<int32_t> cfl(cfo[nC]), fill(cfo.begin(), cfo.end() - 1), perm(nC), iperm(nC), bounds;
    for (int f = 0; f < nF; ++f) {
        cfl[fill[h->owner[f]]++] = f;
        if (f < nIF) cfl[fill[h->neighbour[f]]++] = f;
    }
    for (int tile = std::min(tile_cells, dugks::kMaxTile);; tile = std::max(4, tile * 7 / 8)) {
        std::iota(perm.begin(), perm.end(), 0);
        rcb_order(h->C, perm, 0, nC, tile_cells > 0 ? tile : 4, false);
        for (int c = 0; c < nC; ++c) iperm[perm[c]] = c;
        bounds.clear();
        if (tile_cells <= 0) {
            bounds = greedy_bounds(nC, nIF, h->owner, h->neighbour, cfo, cfl, perm, iperm);
            break;
        }
        for (int b = 0; b < nC; b += tile) bounds.push_back(b);
        bounds.push_back(nC);
        if (tile <= 4 || tiles_fit(nIF, h->owner, h->neighbour, cfo, cfl, perm, iperm, bounds)) break;
    }
    t.fits = tiles_fit(nIF, h->owner, h->neighbour, cfo, cfl, perm, iperm, bounds);
    t.n_tiles = static_cast<int>(bounds.size()) - 1;
    t.tile_cells = 0;
    std::vector<int32_t> tile_of(nC);
    for (int i = 0; i < t.n_tiles; ++i) {
        t.tile_cells = std::max(t.tile_cells, bounds[i + 1] - bounds[i]);
        for (int c = bounds[i]; c < bounds[i + 1]; ++c) tile_of[perm[c]] = i;
    }
    return tile_of;
}

}  // namespace

namespace dugks {

// Cell order, face order and the tables of the step's kernels.  Cells are
// renumbered by recursive coordinate bisection down to 1,024 cells, so that a CTA's cells and their neighbours meet in L1 and L2.
// Smaller parts cost the gathers more sectors than they save: on a 6 x 16^3
// cubed sphere the face values' L1 load is 51 % with parts of 4, 44 % with 256,
// 40 % with 1,024.  Internal faces are numbered by the
// lower of their two cells: in blocks of 32 cells, the first faces of the
// block's cells, then the second ones and so on, so that the k-th faces of
// consecutive cells are nearly consecutive.  Boundary faces follow in the
// caller's order.  Stencils and face lists are slot-major ([slot][cell]).
void build_tiling(dugks_handle* h, int tile_cells) {
    Tiling& t = h->tiling;
    const int nC = h->nC, nIF = h->nIF, nBF = h->nBF, nF = nIF + nBF;
    t.perm.resize(nC);
    std::iota(t.perm.begin(), t.perm.end(), 0);
    const std::vector<int32_t> tile_of = tile_cells_of(h, tile_cells, t);
    rcb_order(h->C, t.perm, 0, nC, 1024, true);
    t.iperm.assign(nC, 0);
    for (int c = 0; c < nC; ++c) t.iperm[t.perm[c]] = c;

    // cell -> faces, those it owns first, each part in the caller's face order
    // (the order the cell's gradient and fluxes are summed in)
    std::vector<int32_t> cfo(nC + 1, 0);
    for (int f = 0; f < nF; ++f) cfo[t.iperm[h->owner[f]] + 1]++;
    for (int f = 0; f < nIF; ++f) cfo[t.iperm[h->neighbour[f]] + 1]++;
    t.nf_max = 0;
    for (int c = 0; c < nC; ++c) {
        t.nf_max = std::max(t.nf_max, cfo[c + 1]);
        cfo[c + 1] += cfo[c];
    }
    std::vector<int32_t> cfl(cfo[nC]), fill(cfo.begin(), cfo.end() - 1);
    for (int f = 0; f < nF; ++f) cfl[fill[t.iperm[h->owner[f]]]++] = f;
    for (int f = 0; f < nIF; ++f) cfl[fill[t.iperm[h->neighbour[f]]]++] = f;

    // face order
    struct Key {
        int block, rank, cell, face;
        bool operator<(const Key& o) const {
            if (block != o.block) return block < o.block;
            if (rank != o.rank) return rank < o.rank;
            return cell < o.cell;
        }
    };
    std::vector<Key> keys;
    keys.reserve(nIF);
    t.nb_max = 0;
    for (int c = 0; c < nC; ++c) {
        int rank = 0, nb = 0;
        for (int k = cfo[c]; k < cfo[c + 1]; ++k) {
            const int f = cfl[k];
            if (f >= nIF) continue;
            ++nb;
            const int o = t.iperm[h->owner[f]], n = t.iperm[h->neighbour[f]];
            if (std::min(o, n) == c) keys.push_back({c / 32, rank++, c, f});
        }
        t.nb_max = std::max(t.nb_max, nb);
    }
    std::sort(keys.begin(), keys.end());
    t.forig.resize(nF);
    t.fnew.resize(nF);
    for (int i = 0; i < nF; ++i) {
        t.forig[i] = i < nIF ? keys[i].face : i;
        t.fnew[t.forig[i]] = i;
    }
    t.fown.resize(nF);
    t.fnei.resize(std::max(nIF, 1));
    t.fgeo.assign(9 * static_cast<size_t>(nF), 0.0);
    for (int i = 0; i < nF; ++i) {
        const int f = t.forig[i];
        const int64_t o = h->owner[f];
        t.fown[i] = t.iperm[o];
        for (int q = 0; q < 3; ++q) {
            t.fgeo[static_cast<size_t>(q) * nF + i] = h->Sf[3 * f + q];
            t.fgeo[static_cast<size_t>(3 + q) * nF + i] = h->Cf[3 * f + q] - h->C[3 * o + q];
        }
        if (f >= nIF) continue;
        const int64_t n = h->neighbour[f];
        t.fnei[i] = t.iperm[n];
        for (int q = 0; q < 3; ++q) t.fgeo[static_cast<size_t>(6 + q) * nF + i] = h->Cf[3 * f + q] - h->C[3 * n + q];
    }

    // gradient stencils and face lists, slots in that order
    t.nbr.resize(static_cast<size_t>(std::max(t.nb_max, 1)) * nC);
    for (size_t i = 0; i < t.nbr.size(); ++i) t.nbr[i] = static_cast<int32_t>(i % nC);
    t.nbr_ls.assign(static_cast<size_t>(std::max(t.nb_max, 1)) * 3 * nC, 0.0);
    t.cface.assign(static_cast<size_t>(t.nf_max) * nC, -1);
    for (int c = 0; c < nC; ++c) {
        int sb = 0, sf = 0;
        for (int k = cfo[c]; k < cfo[c + 1]; ++k) {
            const int f = cfl[k], i = t.fnew[f];
            const bool is_own = t.fown[i] == c;
            if (f < nIF) {
                t.nbr[static_cast<size_t>(sb) * nC + c] = is_own ? t.fnei[i] : t.fown[i];
                const double* ls = is_own ? &h->lsP[3 * f] : &h->lsN[3 * f];
                for (int q = 0; q < 3; ++q) t.nbr_ls[(static_cast<size_t>(sb) * 3 + q) * nC + c] = ls[q];
                ++sb;
            }
            const bool in_tile = f < nIF && tile_of[h->owner[f]] == tile_of[h->neighbour[f]];
            t.cface[static_cast<size_t>(sf) * nC + c] = 4 * i + (in_tile ? 2 : 0) + (is_own ? 0 : 1);
            ++sf;
        }
    }
}

}  // namespace dugks
