// The kernels of one DUGKS step over (DV, cell) and (DV, face) arrays (sm_100a).
//
// Every (entity, DV) array of the step is laid out [block of 32 cells or
// faces][dv][32] (DevMesh): a warp's 32 entities read and write contiguously,
// a thread, which keeps one entity's geometry and coefficients in registers and
// walks DVs, finds the next DV a constant 32 elements on, so that a group of
// DVs shares one address, and a group's rows of a warp are one contiguous
// copy.  DVs are walked in segments (DevMesh::n_seg): up to 32 consecutive DVs
// of one row of the tensor product (the n1d DVs along x at fixed y and z), or
// of the DV list.  Within a row xi = (x_j, Y, Z) varies in x only, so xi.S, the
// Shakhov exponent and the raw moments split into a part computed once per
// segment (Y, Z) and a short per-DV part in x.
//
//   k_half_step     cells  gbar+ = relaxed g~ (updateGHbarPvol, fvDVM.C:648-683)
//   k_face_values   cells  least-squares gradient of gbar+ and, for every face the
//                          cell is the upwind side of, the reconstruction at the
//                          half step (fvDVM.C:456-485, :755-1029)
//   k_face_moments  faces  raw face moments (updateMacroSurf, :1181-1297) and the
//                          wall out-flux; incoming boundary DFs; then face macros
//   k_face_flux     faces  relaxation of the face value (updateGHsurf, :1362-1457),
//                          flux xi.S g_f in place
//   k_update        cells  flux gather and g~ update (updateGHtildeVol, :1462-1519),
//                          raw cell moments (updateMacroVol, :1528-1554), then the
//                          cell macros
//
// Why five streaming kernels: the step moves per (cell, DV) and field 2 reals
// (half step), 1 + D (face values written), D (moments), 2 D (flux) and D + 2
// (update), seven times the state's own traffic, but each kernel is a
// plain stream at high occupancy.  The tiled form (two passes of 512-thread CTAs,
// 16 warps per SM, two or three CTA barriers per 8 to 16 DVs) issued on 30 % of
// the cycles and recomputed gbar+ of each tile's ring.  24,576 cells and 16^3
// DVs in FP64 (100 M updates): 9.4 ms tiled, 3.7 ms now: half step 0.29, face
// values 1.16, tangential pairs 0.12, moments 0.41, flux 0.90, update 0.84.
#include <algorithm>
#include <type_traits>

#include "dugks_device.cuh"

namespace dugks {

namespace {

constexpr int kLanes = 32;      // entities per CTA of the reducing kernels
constexpr int kParts = 4;       // warps per CTA of the reducing kernels: segments interleaved
constexpr int kStream = 128;    // threads per CTA of k_half_step
constexpr int kFaces = 128;     // internal faces per CTA of k_face_moments and k_face_flux
constexpr int kGroupDv = 8;     // DVs per stage of their rings
constexpr int kCells = 256;     // threads per CTA of k_face_values: its L1 holds the block's ring
constexpr int kFast = 6;        // neighbours and faces of a cell kept in registers (a hexahedron)

// FP32 storage holds deviations from the per-DV reference Maxwellian
// (DevMesh::gref, href): g = stored + ref.  DV lists store absolute values.
template <typename Real, bool GEN>
__device__ __forceinline__ double dv_ref(const double* ref, int d) {
    if constexpr (sizeof(Real) == 4 && !GEN) return __ldg(ref + d);
    else return 0.0;
}

// ---------------------------------------------------------------------
// segments
// ---------------------------------------------------------------------
struct Seg {
    int ix0, len, d0, iy, iz;   // first x index, DVs, first local DV, row indices
};

// (d0, len and ix0 by arithmetic on the segment's number, which is uniform
// over the warp: the row addresses they lead to stay in uniform registers)
template <bool GEN>
__device__ __forceinline__ Seg seg_at(const DevMesh& m, int s) {
    Seg q;
    if constexpr (GEN) {
        q.ix0 = q.iy = q.iz = 0;
        q.d0 = s * kSeg;
        q.len = min(kSeg, m.nv_loc - q.d0);
    } else {
        const int two = m.n1d > kSeg, row = s >> two, k = s & two;   // n1d <= 64: one or two segments a row
        q.ix0 = k * kSeg;
        q.d0 = row * m.n1d + q.ix0;   // as seg_dv
        q.len = min(kSeg, m.n1d - q.ix0);
        const int2 t = __ldg(m.row_yz + row);
        q.iy = chk(t.x, 0, m.n1d, m.err);
        q.iz = chk(t.y, 0, m.n1d, m.err);
    }
    return q;
}

// this thread's warp in its CTA, known to be uniform
__device__ __forceinline__ int warp_id() { return __shfl_sync(0xffffffffu, threadIdx.x / kLanes, 0); }

// element of entity e, DV 0, in an (entity, DV) array of nd DVs; DV d is 32 d on
__device__ __forceinline__ size_t slot(int e, int nd) {
    return static_cast<size_t>(e >> 5) * nd * 32 + (e & 31);
}

// the same in gbar+ and hbar+, whose first DV held is a.d_bar
__device__ __forceinline__ ptrdiff_t bar_slot(const StepArgs& a, int c) {
    return static_cast<ptrdiff_t>(slot(c, a.dm.nv_bar)) - 32 * static_cast<ptrdiff_t>(a.d_bar);
}

// calls f(j, U) for groups of U consecutive DVs of a segment, then narrower
// groups for the rest: the loads of a group are issued together
template <int U, class F>
__device__ __forceinline__ void groups(int len, F&& f) {
    int j = 0;
    for (; j + U <= len; j += U) f(j, std::integral_constant<int, U>{});
    if constexpr (U >= 8) {
        if (j + 4 <= len) {
            f(j, std::integral_constant<int, 4>{});
            j += 4;
        }
    }
    if constexpr (U >= 4) {
        if (j + 2 <= len) {
            f(j, std::integral_constant<int, 2>{});
            j += 2;
        }
    }
    if (U > 1 && j < len) f(j, std::integral_constant<int, 1>{});
}

// Walks the segments s, s + step, ... below s1 in groups of U DVs, the loads
// of a group issued one group ahead (into the next segment at a segment's
// end), so that a warp's loads are in flight while it computes.  load(q, j, buf)
// reads DVs j .. j + U - 1 of segment q (past its end what follows: the arrays
// are allocated with kSlack elements to spare); row(q) forms
// what depends on the segment; body(q, j, buf) uses a group, DVs past the
// segment's end excluded; fold(q) closes a segment.
template <int U, bool GEN, typename Buf, class Load, class Row, class Body, class Fold>
__device__ __forceinline__ void walk_dvs(const DevMesh& m, int s, int s1, int step, Load&& load, Row&& row, Body&& body,
                                         Fold&& fold) {
    if (s >= s1) return;
    Seg q = seg_at<GEN>(m, s);
    Buf cur, ahead;
    load(q, 0, cur);
    for (;;) {
        const bool more = s + step < s1;
        const Seg qn = more ? seg_at<GEN>(m, s + step) : q;
        row(q);
        for (int j = 0; j < q.len; j += U) {
            if (j + U < q.len) load(q, j + U, ahead);
            else if (more) load(qn, 0, ahead);
            body(q, j, cur);
            cur = ahead;
        }
        fold(q);
        if (!more) return;
        s += step;
        q = qn;
    }
}

// one-dimensional nodes and weights of the DV set in shared memory
__device__ __forceinline__ void load_nodes(const DevMesh& m, double* x1, double* w1) {
    for (int i = threadIdx.x; i < m.n1d; i += blockDim.x) {
        x1[i] = __ldg(m.X1 + i);
        w1[i] = __ldg(m.W1 + i);
    }
    __syncthreads();
}

// velocity and weight of DV j of a segment
struct Dv {
    double x, y, z, w;
};
template <int D, bool GEN>
__device__ __forceinline__ Dv dv_at(const DevMesh& m, const Seg& q, const double* x1, int j) {
    Dv v;
    if constexpr (GEN) {
        const int d = m.dv_base + q.d0 + j;
        v.x = __ldg(m.xi + 3 * d);
        v.y = __ldg(m.xi + 3 * d + 1);
        v.z = D == 3 ? __ldg(m.xi + 3 * d + 2) : 0.0;
        v.w = __ldg(m.w + d);
    } else {
        v.x = x1[q.ix0 + j];
        v.y = x1[q.iy];
        v.z = D == 3 ? x1[q.iz] : 0.0;
        v.w = 0.0;
    }
    return v;
}

// per-segment DV constants of a row: its y, z velocity and weight and the
// products the moment fold needs.  The DV weight is w1[iz] w1[iy] w1[ix]
// (3-D) or w1[iy] w1[ix] (2-D), as the tensor product is formed.
struct RowConst {
    double Y, Z, R2, wyz, cY, cZ, cYY, cYZ, cZZ;
};

template <int D>
__device__ __forceinline__ RowConst row_const(const double* x1, const double* w1, const Seg& p) {
    RowConst q;
    q.Y = x1[p.iy];
    q.Z = D == 3 ? x1[p.iz] : 0.0;
    q.wyz = D == 3 ? w1[p.iz] * w1[p.iy] : w1[p.iy];
    q.R2 = q.Y * q.Y + q.Z * q.Z;
    q.cY = q.wyz * q.Y;
    q.cZ = q.wyz * q.Z;
    q.cYY = q.cY * q.Y;
    q.cYZ = q.cY * q.Z;
    q.cZZ = q.cZ * q.Z;
    return q;
}

// Raw moments of one segment, summed along x (a = w_x g, b = w_x h):
// S_k = sum a x^k (k = 0..3), B_k = sum b x^k (k = 0, 1), O = sum a xi.S
// over outgoing wall DVs.  row_fold turns them into the moment record
// (layout in dugks_internal.h) with |xi|^2 = x^2 + Y^2 + Z^2.
struct RowSums {
    double S0 = 0, S1 = 0, S2 = 0, S3 = 0, B0 = 0, B1 = 0, O = 0;
};

// HZ: h is identically zero (D = 3, KInner = 0); its sums stay zero
template <bool HZ>
__device__ __forceinline__ double row_add(RowSums& r, double wx, double x, double g, double h) {
    const double a = wx * g;
    r.S0 += a;
    const double ax = a * x;
    r.S1 += ax;
    const double ax2 = ax * x;
    r.S2 += ax2;
    r.S3 = fma(ax2, x, r.S3);
    if constexpr (!HZ) {
        const double b = wx * h;
        r.B0 += b;
        r.B1 = fma(b, x, r.B1);
    }
    return a;
}

// A CTA of the reducing kernels holds 32 faces (or cells) and kParts warps
// that share the segments of its DV chunk.  Their sums meet in shared memory
// in a fixed order, the chunk's sums go to memory, and the CTA that finishes an
// entity block last (a counter per block) adds the chunks in order and forms
// the macros: no launch of its own, no wait.
struct Finish {
    double red[kParts][15][kLanes];
    double tot[15][kLanes];
    double mac[5][kLanes];   // U, 1/RT, A of the entity
    int last;
};

// moment sums of one thread: its column of Finish::red (rows, updated once
// per segment: 30 registers less in the DV loops), or registers (DV lists,
// updated once per DV) that put() copies there
struct SumsShared {
    double* p;
    __device__ __forceinline__ explicit SumsShared(Finish& f) : p(&f.red[threadIdx.x / kLanes][0][threadIdx.x % kLanes]) {
#pragma unroll
        for (int j = 0; j < 15; ++j) p[j * kLanes] = 0.0;
    }
    __device__ __forceinline__ double& operator[](int j) { return p[j * kLanes]; }
    __device__ __forceinline__ void put(Finish&) {}
};
struct SumsRegs {
    double v[15];
    __device__ __forceinline__ explicit SumsRegs(Finish&) : SumsRegs() {}
    __device__ __forceinline__ SumsRegs() {
#pragma unroll
        for (int j = 0; j < 15; ++j) v[j] = 0.0;
    }
    __device__ __forceinline__ double& operator[](int j) { return v[j]; }
    __device__ __forceinline__ void put(Finish& f) {
#pragma unroll
        for (int j = 0; j < 15; ++j) f.red[threadIdx.x / kLanes][j][threadIdx.x % kLanes] = v[j];
    }
};
template <bool GEN>
using Sums = std::conditional_t<GEN, SumsRegs, SumsShared>;

template <int D, typename Acc>
__device__ __forceinline__ void row_fold(Acc& acc, const RowSums& r, const RowConst& q) {
    const double c = q.wyz;
    const double Wb = r.S2 + fma(q.R2, r.S0, r.B0);   // sum a |xi|^2 + b
    const double Vx = r.S3 + fma(q.R2, r.S1, r.B1);   // sum (a |xi|^2 + b) x
    acc[MOM_M0] = fma(c, r.S0, acc[MOM_M0]);
    acc[MOM_M1] = fma(c, r.S1, acc[MOM_M1]);
    acc[MOM_M1 + 1] = fma(q.cY, r.S0, acc[MOM_M1 + 1]);
    acc[MOM_W] = fma(c, Wb, acc[MOM_W]);
    acc[MOM_V3] = fma(c, Vx, acc[MOM_V3]);
    acc[MOM_V3 + 1] = fma(q.cY, Wb, acc[MOM_V3 + 1]);
    acc[MOM_M2] = fma(c, r.S2, acc[MOM_M2]);
    acc[MOM_M2 + 1] = fma(q.cY, r.S1, acc[MOM_M2 + 1]);
    acc[MOM_M2 + 3] = fma(q.cYY, r.S0, acc[MOM_M2 + 3]);
    if (D == 3) {
        acc[MOM_M1 + 2] = fma(q.cZ, r.S0, acc[MOM_M1 + 2]);
        acc[MOM_V3 + 2] = fma(q.cZ, Wb, acc[MOM_V3 + 2]);
        acc[MOM_M2 + 2] = fma(q.cZ, r.S1, acc[MOM_M2 + 2]);
        acc[MOM_M2 + 4] = fma(q.cYZ, r.S0, acc[MOM_M2 + 4]);
        acc[MOM_M2 + 5] = fma(q.cZZ, r.S0, acc[MOM_M2 + 5]);
    }
    acc[MOM_OUT] = fma(c, r.O, acc[MOM_OUT]);
}

// moments of one DV of a segment: along the row, or straight into acc (DV list)
template <int D, bool HZ, bool GEN, typename Acc>
__device__ __forceinline__ double add_dv(Acc& acc, RowSums& rs, const double* w1, const Seg& q, const Dv& v, int j,
                                         double g, double h) {
    if constexpr (GEN) {
        const double xi[3] = {v.x, v.y, v.z};
        accum<D>(acc.v, v.w, xi, v.x * v.x + v.y * v.y + v.z * v.z, g, h);
        return v.w * g;
    } else {
        return row_add<HZ>(rs, w1[q.ix0 + j], v.x, g, h);
    }
}

// xi.S rounded as the reference evaluates it, ((x Sx + y Sy) + z Sz) without
// fused multiply-adds
__device__ __forceinline__ double xs_dv(const Dv& v, const double* S) {
    return __dadd_rn(__dadd_rn(__dmul_rn(v.x, S[0]), __dmul_rn(v.y, S[1])), __dmul_rn(v.z, S[2]));
}

// ---------------------------------------------------------------------
// Shakhov relaxation of one entity over the DVs of a segment
//   gbar = (1-r) g + r gS,  hbar = (1-r) h + r hS   (fvDVM.C:668-679, :1374-1391)
//   gS = E (1 + s (cs - D - 2)),  hS = E RTh (K3D + s ((cs - D) K3D - 2 K))
//   cs = |xi-U|^2 / RT = (x-Ux)^2 / RT + Cyz,  s = (xi-U).qv = (x-Ux) qx + Syz
//   r E = (A e_x(x)) (r e_y(Y) e_z(Z)) from the entity's one-dimensional tables
// ---------------------------------------------------------------------
// What depends on the row only is formed per segment from the record in
// memory (it stays in L1), so that a thread holds five numbers per entity.
template <int D, bool HZ, bool GEN>
struct Relax {
    const double* rec;   // the entity's record and tables: fields and nodes are 32 apart
    const double* tab;
    double Ux, invRT, qx, RTh, r;
    double Cyz, Syz, eyzr;                  // rows
    double Uy, Uz, qy, qz, rA;              // DV lists
    __device__ __forceinline__ Relax(const double* rec_, const double* tab_, int n1d, int e, double r_) {
        rec = rec_ + slot(e, REC_N);
        tab = tab_ + slot(e, D * n1d);
        Ux = field(REC_UX);
        invRT = field(REC_INVRT);
        qx = field(REC_QX);
        RTh = HZ ? 0.0 : field(REC_RTH);
        r = r_;
        if constexpr (GEN) {
            Uy = field(REC_UY);
            Uz = field(REC_UZ);
            qy = field(REC_QY);
            qz = field(REC_QZ);
            rA = r * field(REC_A);
        }
    }
    __device__ __forceinline__ double field(int k) const { return __ldg(rec + 32 * k); }
    __device__ __forceinline__ void row(const DevMesh& m, const Seg& q, double Y, double Z) {
        if constexpr (!GEN) {
            const double cy = Y - field(REC_UY), vy = field(REC_QY);
            const double ey = __ldg(tab + 32 * (m.n1d + q.iy));
            if constexpr (D == 3) {
                const double cz = Z - field(REC_UZ), vz = field(REC_QZ);
                const double ez = __ldg(tab + 32 * (2 * m.n1d + q.iz));
                Cyz = (cy * cy + cz * cz) * invRT;
                Syz = cy * vy + cz * vz;
                eyzr = r * ey * ez;
            } else {
                Cyz = cy * cy * invRT;
                Syz = cy * vy;
                eyzr = r * ey;
            }
        }
    }
    // the Maxwellian factor of DV j of a segment
    __device__ __forceinline__ double factor(const Seg& q, int j) const {
        if constexpr (GEN) return 0.0;
        else return __ldg(tab + 32 * (q.ix0 + j));
    }
    __device__ __forceinline__ void operator()(const Dv& v, double e, double g, double h, double K3D, double c0h,
                                               double& go, double& ho) const {
        const double cx = v.x - Ux;
        double cs, sq, Er;
        if constexpr (GEN) {
            const double cy = v.y - Uy, cz = D == 3 ? v.z - Uz : 0.0;
            cs = (cx * cx + cy * cy + cz * cz) * invRT;
            sq = cx * qx + cy * qy + (D == 3 ? cz * qz : 0.0);
            Er = rA * exp(-0.5 * cs);
        } else {
            cs = fma(cx * cx, invRT, Cyz);
            sq = fma(cx, qx, Syz);
            Er = e * eyzr;
        }
        const double omr = 1.0 - r;
        go = fma(omr, g, Er * fma(sq, cs - double(D + 2), 1.0));
        if constexpr (HZ) ho = 0.0;
        else ho = fma(omr, h, (Er * RTh) * fma(sq, fma(cs, K3D, c0h), K3D));
    }
};

// K + 3 - D and -(D (K + 3 - D) + 2 K) of h^S
template <int D>
__device__ __forceinline__ double k3d(const DevMesh& m) { return m.K + 3.0 - D; }
template <int D>
__device__ __forceinline__ double c0h_of(const DevMesh& m) { return -(D * (m.K + 3.0 - D) + 2.0 * m.K); }

// a cell's relax factor of this step (fvDVM.C:668); its record holds tau
__device__ __forceinline__ double cell_r(const StepArgs& a, int c) {
    const double dt = step_dt(a), tau = __ldg(a.ds.cellrec + slot(c, REC_N) + 32 * REC_R);
    return 1.5 * dt / (2.0 * tau + dt);
}

// ---------------------------------------------------------------------
// k_half_step
// ---------------------------------------------------------------------
// Reads g~ and writes gbar+: 16 B per (cell, DV) and FP64 field, bound by HBM
// (100 M updates in 0.295 ms: 5.4 TB/s).
template <int D, typename Real, bool HZ, bool GEN>
__global__ void __launch_bounds__(kStream) k_half_step(const __grid_constant__ StepArgs a) {
    const DevMesh& m = a.dm;
    __shared__ double x1[kMaxN1d], w1[kMaxN1d];
    load_nodes(m, x1, w1);
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 2 && !a.keep_co) a.ds.co[threadIdx.x] = 0.0;
    const int c = blockIdx.x * kStream + threadIdx.x;
    if (c >= m.nC) return;
    const size_t at = slot(c, m.nv_loc);
    const double K3D = k3d<D>(m), c0h = c0h_of<D>(m);
    Relax<D, HZ, GEN> rx(a.ds.cellrec, a.ds.ctab, m.n1d, c, cell_r(a, c));
    const int ns = a.seg1 - a.seg0;
    const int s0 = a.seg0 + seg_begin(ns, blockIdx.y, gridDim.y), s1 = a.seg0 + seg_begin(ns, blockIdx.y + 1, gridDim.y);
    const Real* __restrict__ g = reinterpret_cast<const Real*>(a.ds.g) + at;
    const Real* __restrict__ h = reinterpret_cast<const Real*>(a.ds.h) + at;
    Real* __restrict__ gb = reinterpret_cast<Real*>(a.ds.gbar) + bar_slot(a, c);
    Real* __restrict__ hb = reinterpret_cast<Real*>(a.ds.hbar) + bar_slot(a, c);
    constexpr int U = 4;
    struct Buf {
        Real g[U], h[U];
        double e[U];
    };
    walk_dvs<U, GEN, Buf>(
        m, s0, s1, 1,
        [&](const Seg& q, int j, Buf& b) {
            const Real *gs = g + 32 * static_cast<size_t>(q.d0 + j), *hs = h + 32 * static_cast<size_t>(q.d0 + j);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                b.g[u] = __ldcs(gs + 32 * u);
                if (!HZ) b.h[u] = __ldcs(hs + 32 * u);
                b.e[u] = rx.factor(q, j + u);
            }
        },
        [&](const Seg& q) { rx.row(m, q, x1[q.iy], x1[q.iz]); },
        [&](const Seg& q, int j, const Buf& b) {
            Real *gd = gb + 32 * static_cast<size_t>(q.d0 + j), *hd = hb + 32 * static_cast<size_t>(q.d0 + j);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (j + u < q.len) {
                    const double gr = dv_ref<Real, GEN>(m.gref, q.d0 + j + u), hr = dv_ref<Real, GEN>(m.href, q.d0 + j + u);
                    double go, ho;
                    rx(dv_at<D, GEN>(m, q, x1, j + u), b.e[u], double(b.g[u]) + gr, HZ ? 0.0 : double(b.h[u]) + hr, K3D,
                       c0h, go, ho);
                    gd[32 * u] = Real(go - gr);
                    if (!HZ) hd[32 * u] = Real(ho - hr);
                }
            }
        },
        [](const Seg&) {});
}

// ---------------------------------------------------------------------
// k_face_values
// ---------------------------------------------------------------------
// Reconstruction at the half step from one side of a face
// (fvDVM.C:832-836): gbar+ + grad . v, v = Cf - C - xi dt/2, x first, one
// fused multiply-add per dimension and one for each component of v.
template <int D, typename Real>
__device__ __forceinline__ Real recon(Real gb, const Real* G, const Real* v) {
    Real r = fma(G[0], v[0], gb);
    r = fma(G[1], v[1], r);
    if (D == 3) r = fma(G[D - 1], v[D - 1], r);
    return r;
}

// One component of v = Cf - C - xi dt/2 in the storage type.  Along a row the x
// product is fused and the y and z products are rounded first; a DV list rounds
// all.  Nothing in the method asks for this: it is how the compiler contracted the
// former kernels' loops, kept so that FP32 runs give what they gave.
template <typename Real>
__device__ __forceinline__ Real fused_dist(Real d, Real hdt, double x) {
    return fma(-hdt, Real(x), d);
}
template <typename Real>
__device__ __forceinline__ Real rounded_dist(Real d, Real hdt, double x) {
    if constexpr (sizeof(Real) == 4) return __fsub_rn(d, __fmul_rn(hdt, Real(x)));
    else return fma(-hdt, x, d);
}
// (likewise, 2-D rows round the x product too at the first and last of every
// eight nodes, on faces inside a tile: the former kernel's batches and tiles)
template <int D, typename Real, bool GEN>
constexpr bool kRoundsRows = D == 2 && sizeof(Real) == 4 && !GEN;
__device__ __forceinline__ bool rounds_node(int ix) { return ((ix + 1) & 6) == 0; }
// rounded: the x product is rounded first
template <int D, typename Real, bool GEN>
__device__ __forceinline__ void half_dist(const Real* d, double hdt, const Dv& v, bool rounded, Real* r) {
    if constexpr (GEN && sizeof(Real) == 4) {
        r[0] = d[0] - Real(hdt * v.x);
        r[1] = d[1] - Real(hdt * v.y);
        if (D == 3) r[D - 1] = d[D - 1] - Real(hdt * v.z);
    } else {
        const Real h = Real(hdt);
        r[0] = rounded ? rounded_dist<Real>(d[0], h, v.x) : fused_dist<Real>(d[0], h, v.x);
        r[1] = rounded_dist<Real>(d[1], h, v.y);
        if (D == 3) r[D - 1] = rounded_dist<Real>(d[D - 1], h, v.z);
    }
}

// gradient of cell c's gbar+ (f: the field's element of cell 0 and one DV) from the tables in
// memory: cells with more than kFast neighbours, and tangential faces
template <int D, typename Real>
__device__ __forceinline__ void grad_mem(const DevMesh& m, const Real* f, int c, Real* G, int k0, int* err) {
    const size_t nC = static_cast<size_t>(m.nC);
    const Real f0 = f[slot(c, m.nv_bar)];
    for (int k = k0; k < m.nb_max; ++k) {
        const int n = chk(__ldg(m.nbr + k * nC + c), 0, m.nC, err);
        const Real df = f[slot(n, m.nv_bar)] - f0;
#pragma unroll
        for (int q = 0; q < D; ++q) G[q] = fma(Real(__ldg(m.nbr_ls + (k * 3 + q) * nC + c)), df, G[q]);
    }
}

// the reconstruction from one side of face f, everything from memory
template <int D, typename Real, bool GEN>
__device__ __forceinline__ Real recon_mem(const DevMesh& m, const Real* row, int f, int side, int c, double hdt,
                                          const Dv& v, bool rounded, int* err) {
    const size_t nF = static_cast<size_t>(m.nF);
    Real G[D];
#pragma unroll
    for (int q = 0; q < D; ++q) G[q] = Real(0);
    grad_mem<D, Real>(m, row, c, G, 0, err);
    Real d[D], r[D];
#pragma unroll
    for (int q = 0; q < D; ++q) d[q] = Real(__ldg(m.fgeo + (3 + 3 * side + q) * nF + f));
    half_dist<D, Real, GEN>(d, hdt, v, rounded, r);
    return recon<D, Real>(row[slot(c, m.nv_bar)], G, r);
}

// *p = v where cond is not 0, as one predicated store
__device__ __forceinline__ void store_if(double* p, double v, unsigned cond) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q st.global.f64 [%0], %1;\n}\n" ::"l"(p), "d"(v), "r"(cond)
                 : "memory");
}
__device__ __forceinline__ void store_if(float* p, float v, unsigned cond) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q st.global.f32 [%0], %1;\n}\n" ::"l"(p), "f"(v), "r"(cond)
                 : "memory");
}

// One thread per cell: the gradient from its neighbours' gbar+ (gathered
// through L1: a CTA's cells are a compact block of the mesh) and the value of
// every face it is upwind of (one bit per face and DV, DevMesh::upw).  The
// gradient never leaves registers.  On an exactly tangential internal face
// no side is upwind; k_tangential averages both there.
// Off: 32-bit element offsets wherever the arrays have fewer than 2^32 elements.
template <int D, typename Real, bool HZ, bool GEN, int NS, typename Off>
__global__ void __launch_bounds__(kCells, 2) k_face_values(const __grid_constant__ StepArgs a) {
    const DevMesh& m = a.dm;
    __shared__ double x1[kMaxN1d], w1[kMaxN1d];
    constexpr bool kRowDist = sizeof(Real) == 4 && !GEN;   // v's y and z components formed once per row
    __shared__ Real dist_s[NS * D * kCells];
    __shared__ Real row_s[kRowDist ? NS * (D - 1) * kCells : 1];
    load_nodes(m, x1, w1);
    const int c = blockIdx.x * kCells + threadIdx.x;
    if (c >= m.nC) return;
    const size_t nC = static_cast<size_t>(m.nC), nF = static_cast<size_t>(m.nF);
    const Real* __restrict__ gbar = reinterpret_cast<const Real*>(a.ds.gbar) - 32 * static_cast<ptrdiff_t>(a.d_bar);
    const Real* __restrict__ hbar = reinterpret_cast<const Real*>(a.ds.hbar) - 32 * static_cast<ptrdiff_t>(a.d_bar);
    Real* __restrict__ fvg = reinterpret_cast<Real*>(a.ds.fvg);
    Real* __restrict__ fvh = reinterpret_cast<Real*>(a.ds.fvh);
    const double hdt = 0.5 * step_dt(a);
    // FP64 folds the DV's part of v once per cell, gbar+ - G.xi dt/2; FP32
    // keeps the reference's order, one v per face
    constexpr bool kFold = sizeof(Real) == 8;
    // DVs whose loads are issued together, as the registers allow
    constexpr int kGroup = sizeof(Real) == 4 ? 4 : HZ || D == 2 ? 2 : 1;
    const Off own = static_cast<Off>(slot(c, m.nv_bar));
    Off nb[NS], fo[NS];   // the neighbours' and faces' elements
    unsigned uo[NS];      // the faces' upwind words in a segment's row
    unsigned has = 0, in_tile = 0;
    Real ls[NS][D];
    Real* dist = dist_s + threadIdx.x;   // Cf - C of slot k, dimension q: dist[(k D + q) kCells]
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        nb[k] = static_cast<Off>(slot(k < m.nb_max ? chk(__ldg(m.nbr + k * nC + c), 0, m.nC, a.ds.err) : c, m.nv_bar));
        const int code = k < m.nf_max ? chk(__ldg(m.cface + k * nC + c), -1, 4 * m.nF, a.ds.err) : -1;
        const int f = code < 0 ? 0 : code >> 2, sd = code < 0 ? 0 : code & 1;
        fo[k] = static_cast<Off>(slot(f, m.nv_loc));
        uo[k] = 2u * f + sd;
        has |= (code >= 0 ? 1u : 0u) << k;
        if (kRoundsRows<D, Real, GEN> && code >= 0) in_tile |= ((code >> 1) & 1u) << k;
#pragma unroll
        for (int q = 0; q < D; ++q) {
            ls[k][q] = k < m.nb_max ? Real(__ldg(m.nbr_ls + (k * 3 + q) * nC + c)) : Real(0);
            dist[(k * D + q) * kCells] = Real(__ldg(m.fgeo + (3 + 3 * sd + q) * nF + f));
        }
    }
    const int ns = a.seg1 - a.seg0;
    const int s0 = a.seg0 + seg_begin(ns, blockIdx.y, gridDim.y), s1 = a.seg0 + seg_begin(ns, blockIdx.y + 1, gridDim.y);
    const bool more = m.nb_max > NS || m.nf_max > NS;
    for (int s = s0; s < s1; ++s) {
        const Seg q = seg_at<GEN>(m, s);
        const double Y = x1[q.iy], Z = x1[q.iz];
        unsigned up[NS];   // the segment's upwind bits
        const uint32_t* us = m.upw + s * nF * 2;
#pragma unroll
        for (int k = 0; k < NS; ++k)
            up[k] = (has >> k) & 1u ? __ldg(us + uo[k]) : 0u;
        Real* rowd = row_s + (kRowDist ? threadIdx.x : 0);
        if constexpr (kRowDist) {
#pragma unroll
            for (int k = 0; k < NS; ++k) {
                rowd[k * (D - 1) * kCells] = rounded_dist<Real>(dist[(k * D + 1) * kCells], Real(hdt), Y);
                if (D == 3) rowd[(k * (D - 1) + 1) * kCells] = rounded_dist<Real>(dist[(k * D + D - 1) * kCells], Real(hdt), Z);
            }
        }
        const Real *gr = gbar + 32 * static_cast<size_t>(q.d0), *hr = hbar + 32 * static_cast<size_t>(q.d0);
        Real *fg = fvg + 32 * static_cast<size_t>(q.d0), *fh = fvh + 32 * static_cast<size_t>(q.d0);
        groups<kGroup>(q.len, [&](int j0, auto uc) {
            constexpr int U = decltype(uc)::value;
            Real g0[U], h0[U], G[U][D], H[U][D];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const Real *gj = gr + 32 * j0, *hj = hr + 32 * j0;
                Real dg[NS], dh[NS];
                g0[u] = __ldg(gj + own + 32 * u);
                if (!HZ) h0[u] = __ldg(hj + own + 32 * u);
#pragma unroll
                for (int k = 0; k < NS; ++k) {
                    dg[k] = __ldg(gj + nb[k] + 32 * u);
                    if (!HZ) dh[k] = __ldg(hj + nb[k] + 32 * u);
                }
#pragma unroll
                for (int p = 0; p < D; ++p) G[u][p] = H[u][p] = Real(0);
#pragma unroll
                for (int k = 0; k < NS; ++k) {
                    const Real x = dg[k] - g0[u];
#pragma unroll
                    for (int p = 0; p < D; ++p) G[u][p] = fma(ls[k][p], x, G[u][p]);
                    if (!HZ) {
                        const Real y = dh[k] - h0[u];
#pragma unroll
                        for (int p = 0; p < D; ++p) H[u][p] = fma(ls[k][p], y, H[u][p]);
                    }
                }
            }
            Dv v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = j0 + u;
                v[u] = dv_at<D, GEN>(m, q, x1, j);
                if constexpr (!GEN) {
                    v[u].y = Y;
                    v[u].z = Z;
                }
                if (more) {
                    grad_mem<D, Real>(m, gr + 32 * j, c, G[u], NS, a.ds.err);
                    if (!HZ) grad_mem<D, Real>(m, hr + 32 * j, c, H[u], NS, a.ds.err);
                    for (int k = NS; k < m.nf_max; ++k) {
                        const int cd = chk(__ldg(m.cface + k * nC + c), -1, 4 * m.nF, a.ds.err);
                        if (cd < 0) break;
                        const int f = cd >> 2, sd = cd & 1;
                        if ((__ldg(us + 2 * f + sd) >> j) & 1u) {
                            Real dk[D], vk[D];
#pragma unroll
                            for (int p = 0; p < D; ++p) dk[p] = Real(__ldg(m.fgeo + (3 + 3 * sd + p) * nF + f));
                            half_dist<D, Real, GEN>(dk, hdt, v[u], kRoundsRows<D, Real, GEN> && (cd & 2) && rounds_node(q.ix0 + j),
                                                     vk);
                            fg[slot(f, m.nv_loc) + 32 * j] = recon<D, Real>(g0[u], G[u], vk);
                            if (!HZ) fh[slot(f, m.nv_loc) + 32 * j] = recon<D, Real>(h0[u], H[u], vk);
                        }
                    }
                }
                if constexpr (kFold) {
                    const Real t[3] = {Real(-hdt * v[u].x), Real(-hdt * v[u].y), Real(-hdt * v[u].z)};
                    g0[u] = recon<D, Real>(g0[u], G[u], t);
                    if (!HZ) h0[u] = recon<D, Real>(h0[u], H[u], t);
                }
            }
            // every face's value, stored where the cell is upwind: without
            // branches, which cost more than the values not needed
#pragma unroll
            for (int k = 0; k < NS; ++k) {
                const unsigned bits = up[k] >> j0;
                Real* pg = fg + 32 * j0 + fo[k];
                Real* ph = fh + 32 * j0 + fo[k];
                Real dk[D];
#pragma unroll
                for (int p = 0; p < D; ++p)
                    dk[p] = kRowDist && p > 0 ? rowd[(k * (D - 1) + p - 1) * kCells] : dist[(k * D + p) * kCells];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    Real vk[D];
                    if constexpr (kFold) {
#pragma unroll
                        for (int p = 0; p < D; ++p) vk[p] = dk[p];
                    } else if constexpr (kRowDist) {
                        vk[0] = ((in_tile >> k) & 1u) && rounds_node(q.ix0 + j0 + u)
                                    ? rounded_dist<Real>(dk[0], Real(hdt), v[u].x)
                                    : fused_dist<Real>(dk[0], Real(hdt), v[u].x);
#pragma unroll
                        for (int p = 1; p < D; ++p) vk[p] = dk[p];
                    } else {
                        half_dist<D, Real, GEN>(dk, hdt, v[u], false, vk);
                    }
                    store_if(pg + 32 * u, recon<D, Real>(g0[u], G[u], vk), bits & (1u << u));
                    if (!HZ) store_if(ph + 32 * u, recon<D, Real>(h0[u], H[u], vk), bits & (1u << u));
                }
            }
        });
    }
}

// whether internal face f of owner o lies inside a tile (cell face code, bit 1)
__device__ __forceinline__ bool in_tile_face(const DevMesh& m, int f, int o) {
    for (int k = 0; k < m.nf_max; ++k) {
        const int code = __ldg(m.cface + static_cast<size_t>(k) * m.nC + o);
        if (code >= 0 && (code >> 2) == f) return code & 2;
    }
    return false;
}

// upwind bits of every face and segment (geometry and DV set only; once at
// creation).  Bit j of word (s, f, side): DV j of segment s leaves through
// face f from that side -- internal faces by the switch of fvDVM.C:829-863
// (neither side on an exactly tangential face), boundary faces the outgoing
// DVs (:916-923), symmetry faces the tangential ones too (:1013-1023);
// zero-gradient faces take the cell's value for every DV instead.  Counts the
// tangential (face, DV) pairs of internal faces into count[0], with `tiles`
// those of faces between tiles into count[1].
template <int D, bool GEN>
__global__ void k_upwind_bits(const DevMesh m, uint32_t* upw, bool tiles, unsigned long long* count) {
    __shared__ double x1[kMaxN1d], w1[kMaxN1d];
    load_nodes(m, x1, w1);
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= m.nF) return;
    const size_t nF = static_cast<size_t>(m.nF);
    const double S[3] = {__ldg(m.fgeo + f), __ldg(m.fgeo + nF + f), __ldg(m.fgeo + 2 * nF + f)};
    const int pt = f < m.nIF ? 0 : __ldg(m.bface_ptype + f - m.nIF);
    const bool sym = pt == DUGKS_PATCH_SYMMETRY || pt == DUGKS_PATCH_DVM_SYMMETRY;
    int tangential = 0;
    for (int s = blockIdx.y; s < m.n_seg; s += gridDim.y) {
        const Seg q = seg_at<GEN>(m, s);
        uint32_t own = 0, nei = 0;
        for (int j = 0; j < q.len; ++j) {
            const double xs = xs_dv(dv_at<D, GEN>(m, q, x1, j), S);
            if (pt == 0) {
                if (xs >= kVSmall) own |= 1u << j;
                else if (xs < -kVSmall) nei |= 1u << j;
            } else if (pt != DUGKS_PATCH_ZERO_GRADIENT) {
                if (sym ? xs > -kVSmall : xs > 0) own |= 1u << j;
            }
        }
        uint32_t* w = upw + (static_cast<size_t>(s) * nF + f) * 2;
        w[0] = own;
        w[1] = nei;
        if (pt == 0) tangential += q.len - __popc(own) - __popc(nei);
    }
    if (!tangential) return;
    atomicAdd(count, static_cast<unsigned long long>(tangential));
    if (tiles && !in_tile_face(m, f, chk(__ldg(m.fown + f), 0, m.nC, m.err)))
        atomicAdd(count + 1, static_cast<unsigned long long>(tangential));
}

// the list of those pairs (DevMesh::tang), pairs of one DV and consecutive
// faces together, and the places of the rests of faces between tiles (cursor:
// pairs listed, rests placed)
template <bool GEN>
__global__ void k_list_tangential(const DevMesh m, int2* list, unsigned long long* cursor, uint2* at, unsigned* seg) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    const size_t nF = static_cast<size_t>(m.nF);
    const bool between = at && f < m.nIF && !in_tile_face(m, f, chk(__ldg(m.fown + f), 0, m.nC, m.err));
    const unsigned tiles = __ballot_sync(0xffffffffu, between), lt = (1u << (threadIdx.x % 32)) - 1u;
    for (int s = blockIdx.y; s < m.n_seg; s += gridDim.y) {
        const Seg q = seg_at<GEN>(m, s);
        unsigned t = 0;
        if (f < m.nIF) {
            const uint2 up = reinterpret_cast<const uint2*>(m.upw)[s * nF + f];
            t = ~(up.x | up.y) & (q.len == 32 ? 0xffffffffu : (1u << q.len) - 1u);
        }
        const unsigned rest = __reduce_or_sync(0xffffffffu, between ? t : 0u);
        const bool first = threadIdx.x % 32 == 0 && f < m.nIF;
        if (seg && first) seg[(f / 32) * static_cast<size_t>(m.n_seg) + s] = rest;
        if (!__any_sync(0xffffffffu, t != 0)) continue;
        for (int j = 0; j < q.len; ++j) {
            const unsigned who = __ballot_sync(0xffffffffu, (t >> j) & 1u);
            if (!who) continue;
            unsigned long long base = 0;
            if (threadIdx.x % 32 == 0) base = atomicAdd(cursor, static_cast<unsigned long long>(__popc(who)));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (at && first) {
                const unsigned inter = who & tiles;
                at[(f / 32) * static_cast<size_t>(m.nv_loc) + q.d0 + j] =
                    make_uint2(inter, static_cast<unsigned>(atomicAdd(cursor + 1, static_cast<unsigned long long>(__popc(inter)))));
            }
            if ((t >> j) & 1u) list[base + __popc(who & lt)] = make_int2(f, s * kSeg + j);
        }
    }
}

// Exactly tangential DVs of internal faces: both sides averaged
// (fvDVM.C:847-863).  One thread per listed pair, each side's gradient formed
// again from gbar+: pairs are few (a node at rest on an axis-aligned mesh: one
// DV in n1d) but sit on few faces, where a face's own thread in
// k_face_moments took 3.2 ms of a 110,592-cell ball's 4.5.
template <int D, typename Real, bool HZ, bool GEN>
__global__ void __launch_bounds__(kStream) k_tangential(const __grid_constant__ StepArgs a) {
    const DevMesh& m = a.dm;
    __shared__ double x1[kMaxN1d], w1[kMaxN1d];
    load_nodes(m, x1, w1);
    const double hdt = 0.5 * step_dt(a);
    for (long long i = blockIdx.x * static_cast<long long>(kStream) + threadIdx.x; i < m.n_tang;
         i += static_cast<long long>(gridDim.x) * kStream) {
        const int2 t = __ldg(m.tang + i);
        const int f = chk(t.x, 0, m.nIF, a.ds.err), s = chk(t.y / kSeg, 0, m.n_seg, a.ds.err);
        if (s < a.seg0 || s >= a.seg1) continue;
        const Seg q = seg_at<GEN>(m, s);
        const int j = chk(t.y % kSeg, 0, q.len, a.ds.err);
        const int o = chk(__ldg(m.fown + f), 0, m.nC, a.ds.err), n = chk(__ldg(m.fnei + f), 0, m.nC, a.ds.err);
        bool rounded = false;
        if constexpr (kRoundsRows<D, Real, GEN>) rounded = rounds_node(q.ix0 + j) && in_tile_face(m, f, o);
        const Dv v = dv_at<D, GEN>(m, q, x1, j);
        const size_t rc = 32 * static_cast<size_t>(q.d0 + j), rf = slot(f, m.nv_loc) + rc;
        // the place of its rest, if the face is between tiles
        size_t place = 0;
        bool between = false;
        if constexpr (sizeof(Real) == 4 && !GEN) {
            if (m.tang_at) {
                const uint2 w = __ldg(m.tang_at + static_cast<size_t>(f / 32) * m.nv_loc + q.d0 + j);
                const unsigned bit = 1u << (f % 32);
                between = w.x & bit;
                place = between ? chk_place(w.y + static_cast<unsigned>(__popc(w.x & (bit - 1))), m.n_rest, a.ds.err) : 0;
            }
        }
        auto average = [&](const void* bar, void* fv, float* res) {
            const Real* b = reinterpret_cast<const Real*>(bar) + (rc - 32 * static_cast<size_t>(a.d_bar));
            const Real vn = recon_mem<D, Real, GEN>(m, b, f, 1, n, hdt, v, rounded, a.ds.err);
            const Real vo = recon_mem<D, Real, GEN>(m, b, f, 0, o, hdt, v, rounded, a.ds.err);
            const Real mean = Real(0.5) * (vn + vo);
            reinterpret_cast<Real*>(fv)[rf] = mean;
            // what the moments of a face between tiles add: its two halves, not their rounded sum
            if constexpr (sizeof(Real) == 4)
                if (between) res[place] = float(0.5 * double(vo) + 0.5 * double(vn) - double(mean));
        };
        average(a.ds.gbar, a.ds.fvg, a.ds.tang_res);
        if (!HZ) average(a.ds.hbar, a.ds.fvh, a.ds.tang_res + m.n_rest);
    }
}

// Zero-gradient faces of a part of pass A: the owner's gbar+, which the face
// moments cannot read once the next part has taken its place.  Launched where
// gbar+ is held in parts; otherwise k_face_moments reads it.
template <typename Real>
__global__ void __launch_bounds__(kStream) k_zero_gradient(const __grid_constant__ StepArgs a) {
    const DevMesh& m = a.dm;
    const int b = blockIdx.x * kLanes + threadIdx.x % kLanes;
    if (b >= m.nBF || __ldg(m.bface_ptype + b) != DUGKS_PATCH_ZERO_GRADIENT) return;
    const ptrdiff_t own = bar_slot(a, chk(__ldg(m.bface_owner + b), 0, m.nC, a.ds.err));
    const size_t f = slot(m.nIF + b, m.nv_loc);
    const int d1 = min(a.d_bar + m.nv_bar, m.nv_loc);
    for (int d = a.d_bar + threadIdx.x / kLanes; d < d1; d += kStream / kLanes) {
        const size_t o = 32 * static_cast<size_t>(d);
        reinterpret_cast<Real*>(a.ds.fvg)[f + o] = reinterpret_cast<const Real*>(a.ds.gbar)[own + static_cast<ptrdiff_t>(o)];
        if (!a.hzero)
            reinterpret_cast<Real*>(a.ds.fvh)[f + o] = reinterpret_cast<const Real*>(a.ds.hbar)[own + static_cast<ptrdiff_t>(o)];
    }
}

// ---------------------------------------------------------------------
// Rings of face rows in shared memory
// ---------------------------------------------------------------------
// The face kernels stream their faces' values: a warp's group of DVs is one
// contiguous run (32 faces x kGroupDv DVs), which one lane copies with a bulk
// asynchronous copy into the warp's own ring, kStages groups ahead.  The loads
// need no registers and no address arithmetic in the other lanes, stay in flight
// while a group is used, and no barrier joins the warps.  Register prefetch at
// 24 warps per SM reached 4.5 TB/s in k_face_flux and 2.5 in k_face_moments.
__device__ __forceinline__ unsigned smem_addr(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint64_t* b) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
// waits for phase `parity` of b; false after about a second (the copy's
// completion is the hardware's to signal: the limit only bounds the wait)
__device__ __forceinline__ bool mbar_wait(uint64_t* b, unsigned parity) {
    const unsigned addr = smem_addr(b);
    for (int k = 0; k < 1 << 20; ++k) {
        unsigned ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(addr), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, uint64_t* b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(b))
                 : "memory");
}

// Walks the groups of kGroupDv DVs of the segments s0 .. s1 - 1 through the
// warp's ring.  issue(q, j, n, stage, barrier) copies n DVs from j on, n * dv_bytes in
// all; use(q, j, n, stage) takes them.  Whole warps call it, the barriers
// initialised and visible.  Returns false when a wait ran out.
template <bool GEN, int STAGES, class Issue, class Use>
__device__ __forceinline__ bool ring_walk(const DevMesh& m, uint64_t* full, int s0, int s1, unsigned dv_bytes, Issue&& issue,
                                          Use&& use) {
    int ps = s0, pj = 0;   // the producer's position
    auto fill = [&](int stage) {
        if (ps >= s1) return;
        const Seg q = seg_at<GEN>(m, ps);
        const int n = min(kGroupDv, q.len - pj);
        if (threadIdx.x % 32 == 0) {
            mbar_expect(full + stage, n * dv_bytes);
            issue(q, pj, n, stage, full + stage);
        }
        pj += kGroupDv;
        if (pj >= q.len) {
            pj = 0;
            ++ps;
        }
    };
    for (int i = 0; i < STAGES; ++i) fill(i);
    int stage = 0;
    unsigned parity = 0;
    for (int s = s0; s < s1; ++s) {
        const Seg q = seg_at<GEN>(m, s);
        for (int j = 0; j < q.len; j += kGroupDv) {
            if (!__all_sync(0xffffffffu, mbar_wait(full + stage, parity))) {
                // give up: let the copies in flight land, within the same limit, before the CTA ends
                for (int i = 0; i < STAGES; ++i) {
                    mbar_wait(full + stage, parity);
                    if (++stage == STAGES) {
                        stage = 0;
                        parity ^= 1;
                    }
                }
                return false;
            }
            use(q, j, min(kGroupDv, q.len - j), stage);
            __syncwarp();   // the stage is free
            fill(stage);
            if (++stage == STAGES) {
                stage = 0;
                parity ^= 1;
            }
        }
    }
    return true;
}

// ---------------------------------------------------------------------
// Reductions of the face and cell kernels
// ---------------------------------------------------------------------
// after this CTA's chunk sums went to memory: true in the CTA that completes
// the entity block
__device__ __forceinline__ bool last_chunk(int* done, int& last) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const int k = gridDim.y > 1 ? atomicAdd(done, 1) : 0;
        last = k == static_cast<int>(gridDim.y) - 1;
        if (last && gridDim.y > 1) *done = 0;   // for the next launch
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    return true;
}

// this CTA's chunk, from its warps' sums in f.red, into part [chunk][kNM][n];
// true in the CTA that completes the entity block
__device__ __forceinline__ bool reduce_chunk(Finish& f, double* part, size_t n, int e0, int count, int* done, bool fused) {
    const int lane = threadIdx.x % kLanes, w = threadIdx.x / kLanes;
    __syncthreads();
    for (int j = w; j < 15; j += kParts) {
        double v = f.red[0][j][lane];
        for (int p = 1; p < kParts; ++p) v += f.red[p][j][lane];
        if (lane < count) part[(static_cast<size_t>(blockIdx.y) * kNM + j) * n + e0 + lane] = v;
    }
    return fused && last_chunk(done, f.last);
}

// chunk sums of the block's entities, added in chunk order, into f.tot
__device__ __forceinline__ void sum_chunks(Finish& f, const double* part, size_t n, int e0, int count, int chunks) {
    const int lane = threadIdx.x % kLanes, w = threadIdx.x / kLanes;
    for (int j = w; j < 15; j += kParts) {
        double v = 0.0;
        if (lane < count) {
#pragma unroll 4
            for (int ch = 0; ch < chunks; ++ch) v += __ldcg(part + (static_cast<size_t>(ch) * kNM + j) * n + e0 + lane);
        }
        f.tot[j][lane] = v;
    }
    __syncthreads();
}

// one-dimensional Maxwellian factors of the block's entities (layout in
// dugks_internal.h): D * n1d exponentials each, shared by the CTA's warps
__device__ __forceinline__ void write_tables(const Finish& f, const DevMesh& m, double* tab, int e0, int count) {
    const int lane = threadIdx.x % kLanes, w = threadIdx.x / kLanes;
    if (lane >= count) return;
    const double inv = f.mac[3][lane];
    for (int k = 0; k < m.D; ++k) {
        const double U = f.mac[k][lane], A = k == 0 ? f.mac[4][lane] : 1.0;
        double* t = tab + slot(e0 + lane, m.D * m.n1d) + 32 * k * m.n1d;
        // (four exponentials in flight: few CTAs run when a block finishes)
#pragma unroll 4
        for (int i = w; i < m.n1d; i += kParts) {
            const double x = __ldg(m.X1 + i) - U;
            t[32 * i] = exp(-0.5 * x * x * inv) * A;
        }
    }
}

// chunk sums of one entity, added in chunk order
__device__ __forceinline__ void sum_chunks_of(double* s, const double* part, size_t n, int e, int chunks) {
#pragma unroll
    for (int j = 0; j < 15; ++j) s[j] = 0.0;
#pragma unroll 2
    for (int ch = 0; ch < chunks; ++ch) {
        const double* p = part + static_cast<size_t>(ch) * kNM * n + e;
#pragma unroll
        for (int j = 0; j < 15; ++j) s[j] += __ldcg(p + j * n);
    }
}

// Face macros, relaxation coefficients and Maxwellian tables of one face from
// its chunk sums (updateMaxwellWallRho fvDVM.C:1032-1052,
// calculatedMaxwellFvPatchField.C:140-164, updateMacroSurf :1248-1300), and
// the warp's Courant numbers.  Whole warps call it; f < 0: no face.  With fin
// the CTA's warps share the chunk sums (fin->tot) before and the tables
// (write_tables) after: a block of 32 boundary faces has one warp here.
__device__ __noinline__ void finish_face(const StepArgs& a, const Consts& kc, int f, int chunks, Finish* fin = nullptr) {
    const DevMesh& m = a.dm;
    const size_t nF = static_cast<size_t>(m.nF);
    double co = 0.0;
    if (f >= 0) {
        const double dt = step_dt(a);
        double s[15];
        if (fin)
            for (int j = 0; j < 15; ++j) s[j] = fin->tot[j][threadIdx.x % kLanes];
        else
            sum_chunks_of(s, a.ds.partF, nF, f, chunks);
        if (f >= m.nIF && __ldg(m.bface_ptype + f - m.nIF) == DUGKS_PATCH_MAXWELL_WALL) {
            // rho_w = outGoing / |inComingByRho|; the incoming wall DFs enter through it
            BRec* br = a.ds.brec + (f - m.nIF);
            const double rho_w = s[MOM_OUT] / fabs(br->inByRho);
            br->rho_in = rho_w;
            const double* mi = a.ds.bmom_in + static_cast<size_t>(f - m.nIF) * kNM;
            for (int j = 0; j < 14; ++j) s[j] += rho_w * mi[j];
        }
        double rho, U[3], T, q[3], tau;
        macros_from_moments(s, kc, rho, U, T, q, tau);
        const double fac = 2.0 * tau / (2.0 * tau + 0.5 * dt * kc.Pr);  // fvDVM.C:1300
        for (int i = 0; i < 3; ++i) q[i] *= fac;
        const int fo = chk(__ldg(m.forig + f), 0, m.nF, a.ds.err);
        double* fm = a.ds.fm + static_cast<size_t>(fo) * 9;
        fm[0] = rho;
        fm[4] = T;
        fm[8] = tau;
        const double RT = kc.R * T, A = rho * inv_norm(RT, kc.D), invRT = 1.0 / RT;
        const double qs = kc.Pr1 / (5.0 * rho * RT * RT);
        double* fr = a.ds.facerec + slot(f, REC_N);
        for (int i = 0; i < 3; ++i) {
            fm[1 + i] = U[i];
            fm[5 + i] = q[i];
            fr[(REC_UX + i) * 32] = U[i];
            fr[(REC_QX + i) * 32] = q[i] * qs;
        }
        fr[REC_INVRT * 32] = invRT;
        fr[REC_A * 32] = A;
        fr[REC_R * 32] = 0.5 * dt / (2.0 * tau + 0.5 * dt);
        fr[REC_RTH * 32] = RT;
        if (f < m.nIF)  // getCoNum, fvDVM.C:2180-2182
            co = __ldg(m.dc + fo) * (sqrt(U[0] * U[0] + U[1] * U[1] + U[2] * U[2]) + m.xi_max_co);
        if (fin) {
            const int lane = threadIdx.x % kLanes;
            for (int i = 0; i < 3; ++i) fin->mac[i][lane] = U[i];
            fin->mac[3][lane] = invRT;
            fin->mac[4][lane] = A;
        } else if (!m.general_dv) {
            // one-dimensional Maxwellian factors (layout in dugks_internal.h)
            for (int k = 0; k < m.D; ++k) {
                const double Uk = k == 0 ? U[0] : k == 1 ? U[1] : U[2], Ak = k == 0 ? A : 1.0;
                double* tab = a.ds.ftab + slot(f, m.D * m.n1d) + 32 * k * m.n1d;
#pragma unroll 4
                for (int i = 0; i < m.n1d; ++i) {
                    const double x = __ldg(m.X1 + i) - Uk;
                    tab[32 * i] = exp(-0.5 * x * x * invRT) * Ak;
                }
            }
        }
    }
    double vmax = co, vsum = co;
    for (int o = 16; o > 0; o >>= 1) {
        vmax = fmax(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
        vsum += __shfl_xor_sync(0xffffffffu, vsum, o);
    }
    if (threadIdx.x % kLanes == 0) {
        // non-negative doubles order like their bit patterns
        atomicMax(reinterpret_cast<unsigned long long*>(a.ds.co), static_cast<unsigned long long>(__double_as_longlong(vmax)));
        atomicAdd(a.ds.co + 1, vsum);
    }
}

// the coefficient record of the next half step
__device__ __noinline__ void write_cellrec(const StepArgs& a, const Consts& k, int c, double rho, const double* U,
                                           double T, const double* q, double tau) {
    const double RT = k.R * T;
    const double qs = k.Pr1 / (5.0 * rho * RT * RT);
    double* cr = a.ds.cellrec + slot(c, REC_N);
    for (int i = 0; i < 3; ++i) {
        cr[(REC_UX + i) * 32] = U[i];
        cr[(REC_QX + i) * 32] = q[i] * qs;
    }
    cr[REC_INVRT * 32] = 1.0 / RT;
    cr[REC_A * 32] = rho * inv_norm(RT, k.D);
    cr[REC_R * 32] = tau;
    cr[REC_RTH * 32] = RT;
}

// macroFlux yes (fvDVM.C:1523-1526, :1613-1679): the cell's old rho, rho U,
// rho E advanced by this step's face macro fluxes, faces in face order.  The
// face stress is zero (its sum is commented out, fvDVM.C:1270, :1305); the
// boundary momentum flux takes Sf of the internal face at the patch-local
// index (fvDVM.C:1668-1669); "X & Sf*dt/V" is X & ((Sf dt)/V).
__device__ __forceinline__ void macro_flux_update(const StepArgs& a, const Consts& k, int c, double& rho, double rU[3],
                                                  double& rE) {
    const DevMesh& m = a.dm;
    const double* cm = a.ds.cm + static_cast<size_t>(c) * 9;
    const double U0[3] = {cm[1], cm[2], cm[3]};
    rho = cm[0];
    for (int i = 0; i < 3; ++i) rU[i] = rho * U0[i];
    rE = rho * (0.5 * (U0[0] * U0[0] + U0[1] * U0[1] + U0[2] * U0[2]) + (k.Kin + 3) / 2.0 * k.R * cm[4]);
    const double V = __ldg(m.mf_V + c), dt = k.dt;
    for (int e = __ldg(m.mf_off + c); e < __ldg(m.mf_off + c + 1); ++e) {
        const int code = __ldg(m.mf_ent + e), f = chk(code >> 1, 0, m.nIF + m.nBF, a.ds.err);
        const bool add = code & 1;
        const double* fm = a.ds.fm + static_cast<size_t>(f) * 9;
        const double rf = fm[0], Uf[3] = {fm[1], fm[2], fm[3]}, qf[3] = {fm[5], fm[6], fm[7]};
        const double* S = m.mf_Sf + 3 * static_cast<size_t>(f);
        const double* Sm = f < m.nIF ? S
                                     : m.mf_Sf + 3 * static_cast<size_t>(chk(__ldg(m.bface_patch_local + f - m.nIF), 0,
                                                                             m.nIF + m.nBF, a.ds.err));
        const double rUf[3] = {__dmul_rn(rf, Uf[0]), __dmul_rn(rf, Uf[1]), __dmul_rn(rf, Uf[2])};
        const double rEf = __dmul_rn(rf, __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(Uf[0], Uf[0]), __dmul_rn(Uf[1], Uf[1])),
                                                             __dmul_rn(Uf[2], Uf[2])),
                                                   __dmul_rn(__dmul_rn((k.Kin + 3) / 2.0, k.R), fm[4])));
        double ev[3], Sd[3], Smd[3];
        for (int i = 0; i < 3; ++i) {
            ev[i] = __dadd_rn(__dmul_rn(rEf, Uf[i]), qf[i]);
            Sd[i] = __ddiv_rn(__dmul_rn(__ldg(S + i), dt), V);
            Smd[i] = __ddiv_rn(__dmul_rn(__ldg(Sm + i), dt), V);
        }
        const double mr = __ddiv_rn(__dmul_rn(xi_dot_s(rUf, S), dt), V);
        const double mE = xi_dot_s(ev, Sd);
        double mU[3];
        for (int i = 0; i < 3; ++i) {
            const double t[3] = {__dmul_rn(rUf[i], Uf[0]), __dmul_rn(rUf[i], Uf[1]), __dmul_rn(rUf[i], Uf[2])};
            mU[i] = xi_dot_s(t, Smd);
        }
        if (add) {
            rho += mr;
            for (int i = 0; i < 3; ++i) rU[i] += mU[i];
            rE += mE;
        } else {
            rho -= mr;
            for (int i = 0; i < 3; ++i) rU[i] -= mU[i];
            rE -= mE;
        }
    }
}

// cell macros and record from the moment sums s
__device__ __noinline__ void cell_macros(const StepArgs& a, const Consts& k, int c, const double* s, int chunks) {
    const DevMesh& m = a.dm;
    double rho, U[3], T, q[3], tau;
    if (!m.macro_flux) {
        macros_from_moments(s, k, rho, U, T, q, tau);
    } else {
        // rho, U, T from the fluxes; q from the DF moments about that U:
        // q = 1/2 [V3 - 2 M2.U + |U|^2 M1 - U W + 2 U (M1.U) - U |U|^2 M0]
        double rU[3], rE;
        if (!m.general_dv) {
            macro_flux_update(a, k, c, rho, rU, rE);
        } else {
            // the velocity-mesh branch (fvDVM.C:1562-1611): the old rho, rho U,
            // rho E plus the moments of the update's flux term (pass B)
            const double* cm = a.ds.cm + static_cast<size_t>(c) * 9;
            double f[5] = {0, 0, 0, 0, 0};
            for (int ch = 0; ch < chunks; ++ch)
                for (int j = 0; j < 5; ++j)
                    f[j] += __ldcg(a.ds.partX + (static_cast<size_t>(ch) * kFX + j) * m.nC + c);
            const double U0[3] = {cm[1], cm[2], cm[3]};
            rho = cm[0] + f[0];
            for (int i = 0; i < 3; ++i) rU[i] = cm[0] * U0[i] + f[1 + i];
            rE = cm[0] * (0.5 * (U0[0] * U0[0] + U0[1] * U0[1] + U0[2] * U0[2]) + (k.Kin + 3) / 2.0 * k.R * cm[4]) +
                 f[4];
        }
        for (int i = 0; i < 3; ++i) U[i] = rU[i] / rho;
        const double u2 = U[0] * U[0] + U[1] * U[1] + U[2] * U[2];
        T = (rE - 0.5 * rho * u2) / ((k.Kin + 3.0) / 2.0 * k.R * rho);
        tau = k.muRef * exp(k.omega * log(T / k.Tref)) / rho / T / k.R;
        const double* M2 = s + MOM_M2;
        const double M2U[3] = {M2[0] * U[0] + M2[1] * U[1] + M2[2] * U[2], M2[1] * U[0] + M2[3] * U[1] + M2[4] * U[2],
                               M2[2] * U[0] + M2[4] * U[1] + M2[5] * U[2]};
        const double M1U = s[MOM_M1] * U[0] + s[MOM_M1 + 1] * U[1] + s[MOM_M1 + 2] * U[2];
        for (int i = 0; i < 3; ++i)
            q[i] = 0.5 * (s[MOM_V3 + i] - 2.0 * M2U[i] + u2 * s[MOM_M1 + i] - U[i] * s[MOM_W] + 2.0 * U[i] * M1U -
                          U[i] * u2 * s[MOM_M0]);
    }
    const double fac = 2.0 * tau / (2.0 * tau + k.dt * k.Pr);  // fvDVM.C:1742
    for (int i = 0; i < 3; ++i) q[i] *= fac;
    if (!(rho > 0.0) || !(T > 0.0) || !isfinite(rho + T + U[0] + U[1] + U[2])) atomicOr(a.ds.err, 1);
    double* cm = a.ds.cm + static_cast<size_t>(c) * 9;
    cm[0] = rho;
    cm[1] = U[0];
    cm[2] = U[1];
    cm[3] = U[2];
    cm[4] = T;
    cm[5] = q[0];
    cm[6] = q[1];
    cm[7] = q[2];
    cm[8] = tau;
    write_cellrec(a, k, c, rho, U, T, q, tau);
}

// record factors of the block's cells for their tables
__device__ __forceinline__ void tables_of_records(Finish& sm, const StepArgs& a, int c0, int count) {
    const int lane = threadIdx.x % kLanes;
    if (threadIdx.x < kLanes && lane < count) {
        const double* cr = a.ds.cellrec + slot(c0 + lane, REC_N);
        for (int i = 0; i < 3; ++i) sm.mac[i][lane] = cr[(REC_UX + i) * 32];
        sm.mac[3][lane] = cr[REC_INVRT * 32];
        sm.mac[4][lane] = cr[REC_A * 32];
    }
    __syncthreads();
    if (!a.dm.general_dv) write_tables(sm, a.dm, a.ds.ctab, c0, count);
}

// Cell macros (updateMacroVol, fvDVM.C:1682-1742) and the coefficient
// records of the next half step, of the block's cells from the chunk sums.
__device__ __noinline__ void finish_cells(Finish& sm, const StepArgs& a, const Consts& kc, int c0, int count, int chunks) {
    sum_chunks(sm, a.ds.partC, static_cast<size_t>(a.dm.nC), c0, count, chunks);
    const int lane = threadIdx.x % kLanes;
    if (threadIdx.x < kLanes && lane < count) {
        Consts k = kc;
        k.dt = step_dt(a);
        double s[15];
        for (int j = 0; j < 15; ++j) s[j] = sm.tot[j][lane];
        cell_macros(a, k, c0 + lane, s, chunks);
    }
    tables_of_records(sm, a, c0, count);
}

// cell records and tables from the cell macros in cm
__global__ void __launch_bounds__(kLanes* kParts) k_cell_records(const __grid_constant__ StepArgs a,
                                                                 const __grid_constant__ Consts k) {
    __shared__ Finish sm;
    const int c0 = blockIdx.x * kLanes, count = min(kLanes, a.dm.nC - c0), lane = threadIdx.x % kLanes;
    if (threadIdx.x < kLanes && lane < count) {
        const double* cm = a.ds.cm + static_cast<size_t>(c0 + lane) * 9;
        const double U[3] = {cm[1], cm[2], cm[3]}, q[3] = {cm[5], cm[6], cm[7]};
        write_cellrec(a, k, c0 + lane, cm[0], U, cm[4], q, cm[8]);
    }
    tables_of_records(sm, a, c0, count);
}

// ---------------------------------------------------------------------
// k_face_moments
// ---------------------------------------------------------------------
// the Maxwellian a boundary face's incoming DFs take (fvDVM.C:926-938,
// :1079-1092; mixed patches discreteVelocity.C:226-258)
struct Incoming {
    double rK, inv, hf, U[3];
    template <int D>
    __device__ __forceinline__ void at(const Dv& v, double& g, double& h) const {
        const double cx = v.x - U[0], cy = v.y - U[1], cz = v.z - U[2];
        g = rK * exp(-0.5 * (cx * cx + cy * cy + cz * cz) * inv);
        h = g * hf;
    }
};

__device__ __forceinline__ Incoming load_incoming(const StepArgs& a, int b, int pt) {
    const BRec* br = a.ds.brec + b;
    Incoming t;
    t.rK = br->rho_in * br->K_in;
    t.inv = br->invRT_in;
    t.hf = br->hfac;
    if (pt == DUGKS_PATCH_MAXWELL_WALL || pt == DUGKS_PATCH_MIXED) {
        for (int i = 0; i < 3; ++i) t.U[i] = br->U[i];
    } else {
        const int own = chk(__ldg(a.dm.bface_owner + b), 0, a.dm.nC, a.ds.err);
        for (int i = 0; i < 3; ++i) t.U[i] = a.ds.cellrec[slot(own, REC_N) + 32 * (REC_UX + i)];
    }
    return t;
}

// boundary faces of one chunk: by patch type (fvDVM.C:866-1027).  CUT: gbar+
// is held in parts, and k_zero_gradient has stored the zero-gradient faces (as
// a test at run time it cost a 3,721-cell step 1.5 of 216 us)
template <int D, typename Real, bool HZ, bool GEN, bool CUT>
__device__ __noinline__ void boundary_moments(const StepArgs& a, const double* x1, const double* w1, int f, int s0,
                                              int s1, int w, Finish& sm) {
    const DevMesh& m = a.dm;
    Sums<GEN> acc(sm);
    const size_t nF = static_cast<size_t>(m.nF);
    Real* fg = reinterpret_cast<Real*>(a.ds.fvg) + slot(f, m.nv_loc);
    Real* fh = reinterpret_cast<Real*>(a.ds.fvh) + slot(f, m.nv_loc);
    const int b = f - m.nIF, pt = __ldg(m.bface_ptype + b);
    const bool wall = pt == DUGKS_PATCH_MAXWELL_WALL, zero_grad = pt == DUGKS_PATCH_ZERO_GRADIENT;
    const bool sym = pt == DUGKS_PATCH_SYMMETRY || pt == DUGKS_PATCH_DVM_SYMMETRY;
    const double S[3] = {__ldg(m.fgeo + f), __ldg(m.fgeo + nF + f), __ldg(m.fgeo + 2 * nF + f)};
    const int own = chk(__ldg(m.bface_owner + b), 0, m.nC, a.ds.err);
    const int axis = sym ? __ldg(m.bface_mirror + b) : -1;
    double S0[3] = {0, 0, 0};
    if (axis >= 0) {
        const int b0 = chk(b - __ldg(m.bface_patch_local + b), 0, m.nBF, a.ds.err);
        for (int i = 0; i < 3; ++i) S0[i] = __ldg(m.bS + 3 * b0 + i);
    }
    Incoming in{};
    if (!wall && !zero_grad && !sym) in = load_incoming(a, b, pt);
    for (int s = s0 + w; s < s1; s += kParts) {
        const Seg q = seg_at<GEN>(m, s);
        RowSums rs;
        Real g4[4] = {0, 0, 0, 0}, h4[4] = {0, 0, 0, 0};
        for (int j = 0; j < q.len; ++j) {
            const int d = q.d0 + j;
            const size_t o = 32 * static_cast<size_t>(d);
            if ((j & 3) == 0) {
                // the stored values of four DVs at a time (those of incoming DVs are not used)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const size_t ou = o + 32 * u;
                    g4[u] = fg[ou];
                    if (!HZ) h4[u] = fh[ou];
                }
            }
            const Real gv = g4[0], hv = h4[0];
            g4[0] = g4[1], g4[1] = g4[2], g4[2] = g4[3];
            h4[0] = h4[1], h4[1] = h4[2], h4[2] = h4[3];
            const Dv v = dv_at<D, GEN>(m, q, x1, j);
            const double xs = xs_dv(v, S);
            const double gr = dv_ref<Real, GEN>(m.gref, d), hr = dv_ref<Real, GEN>(m.href, d);
            double g, h = 0.0;
            if (zero_grad) {
                // every DV: the owner cell's gbar+ (fvDVM.C:887-891)
                const size_t oc = slot(own, m.nv_loc) + o;
                const Real gc = CUT ? gv : reinterpret_cast<const Real*>(a.ds.gbar)[oc];
                if (!CUT) fg[o] = gc;
                g = double(gc) + gr;
                if (!HZ) {
                    const Real hc = CUT ? hv : reinterpret_cast<const Real*>(a.ds.hbar)[oc];
                    if (!CUT) fh[o] = hc;
                    h = double(hc) + hr;
                }
            } else if (sym) {
                // incoming through the patch's first face (updateGHbarSurfSymmetryIn,
                // fvDVM.C:1100-1179, discreteVelocity.C:691-773): the face value of the
                // mirror DV along the patch's axis; a DV that is its own mirror stays.
                // Values reconstructed this step are those outgoing or tangential here;
                // on a face tilted against the first others stay without one: zero, not
                // the last step's flux that their slot holds
                const bool here = xs > -kVSmall;
                bool counted = here, mirrored = false;
                Real gn = here ? gv : Real(0), hn = here && !HZ ? hv : Real(0);
                if constexpr (!GEN) {
                    if (!(xs_dv(v, S0) > 0)) {
                        const int n = m.n1d, st = axis == 0 ? 1 : axis == 1 ? n : n * n;
                        const int i = axis == 0 ? q.ix0 + j : axis == 1 ? q.iy : q.iz;
                        const int t = d + (n - 1 - 2 * i) * st;
                        if (t != d) {
                            counted = true;
                            // of two mirrors that are both incoming the later one keeps its value
                            Dv vt = v;
                            (axis == 0 ? vt.x : axis == 1 ? vt.y : vt.z) = x1[n - 1 - i];
                            mirrored = xs_dv(vt, S0) > 0 || t > d;
                            if (mirrored) {
                                const bool there = xs_dv(vt, S) > -kVSmall;
                                const size_t ot = 32 * static_cast<size_t>(t);
                                const double grt = dv_ref<Real, GEN>(m.gref, t), hrt = dv_ref<Real, GEN>(m.href, t);
                                gn = Real((double(there ? fg[ot] : Real(0)) + grt) - gr);
                                if (!HZ) hn = Real((double(there ? fh[ot] : Real(0)) + hrt) - hr);
                            }
                        }
                    }
                }
                if (mirrored || !here) {
                    fg[o] = gn;
                    if (!HZ) fh[o] = hn;
                }
                if (!counted) continue;
                g = double(gn) + gr;
                if (!HZ) h = double(hn) + hr;
            } else if (xs > 0) {
                // outgoing: upwind from the owner (fvDVM.C:916-923, :950-961)
                g = double(gv) + gr;
                if (!HZ) h = double(hv) + hr;
            } else if (wall) {
                continue;   // incoming wall DFs enter through rho_w
            } else {
                in.at<D>(v, g, h);
                // rounded as k_face_flux rounds the same incoming DF
                g = double(Real(g - gr)) + gr;
                h = double(Real(h - hr)) + hr;
            }
            const double aw = add_dv<D, HZ, GEN>(acc, rs, w1, q, v, j, g, h);
            if (wall) {
                if constexpr (GEN) acc[MOM_OUT] = fma(aw, xs, acc[MOM_OUT]);
                else rs.O = fma(aw, xs, rs.O);
            }
        }
        if constexpr (!GEN) row_fold<D>(acc, rs, row_const<D>(x1, w1, q));
    }
    acc.put(sm);
}

constexpr int kStagesM = 4;   // ring stages of k_face_moments
constexpr int kStagesF = 3;   // and of k_face_flux, whose stages hold e_x too

template <typename Real, bool HZ>
constexpr size_t ring_moments() {
    const size_t ring = static_cast<size_t>(kStagesM) * (HZ ? 1 : 2) * kGroupDv * kFaces * sizeof(Real);
    return ring > sizeof(Finish) ? ring : sizeof(Finish);   // boundary blocks hold their sums there
}

// Internal faces: reads each face value once (8 B per face, DV and FP64
// field) and adds seven FP64 operations.  Boundary faces: 32 per CTA, the
// segments split over its warps, as incoming DFs cost an exponential each.
template <int D, typename Real, bool HZ, bool GEN, bool CUT>
__global__ void __launch_bounds__(kFaces, 5) k_face_moments(const __grid_constant__ StepArgs a,
                                                            const __grid_constant__ Consts kc) {
    static_assert(kFaces == kLanes * kParts, "one CTA size for internal and boundary blocks");
    const DevMesh& m = a.dm;
    extern __shared__ __align__(128) unsigned char ring_raw[];
    __shared__ double x1[kMaxN1d], w1[kMaxN1d];
    __shared__ __align__(8) uint64_t full[kParts * kStagesM];
    __shared__ int last;
    if (threadIdx.x < kParts * kStagesM) mbar_init(full + threadIdx.x);
    load_nodes(m, x1, w1);
    const size_t nF = static_cast<size_t>(m.nF);
    const int s0 = seg_begin(m.n_seg, blockIdx.y, gridDim.y), s1 = seg_begin(m.n_seg, blockIdx.y + 1, gridDim.y);
    // boundary face blocks first: they take longest
    const int nbB = (m.nBF + kLanes - 1) / kLanes, bx = blockIdx.x;
    if (bx < nbB) {
        const int f0 = m.nIF + bx * kLanes, count = min(kLanes, m.nF - f0), lane = threadIdx.x % kLanes;
        const int w = warp_id();
        Finish& sm = *reinterpret_cast<Finish*>(ring_raw);
        if (lane < count) boundary_moments<D, Real, HZ, GEN, CUT>(a, x1, w1, f0 + lane, s0, s1, w, sm);
        if (reduce_chunk(sm, a.ds.partF, nF, f0, count, a.ds.done + bx, a.fused != 0)) {
            sum_chunks(sm, a.ds.partF, nF, f0, count, gridDim.y);
            if (w == 0) finish_face(a, kc, lane < count ? f0 + lane : -1, gridDim.y, &sm);
            __syncthreads();
            if (!m.general_dv) write_tables(sm, m, a.ds.ftab, f0, count);
        }
        return;
    }
    const int f0 = (bx - nbB) * kFaces, f = f0 + threadIdx.x;
    const bool active = f < m.nIF;
    Real* fg = reinterpret_cast<Real*>(a.ds.fvg);
    Real* fh = reinterpret_cast<Real*>(a.ds.fvh);
    // the copies see the barriers' set-up
    asm volatile("fence.proxy.async;" ::: "memory");
    __syncthreads();
    SumsRegs acc;
    RowSums rs;
    // the warp's 32 faces and ring
    constexpr int NH = HZ ? 1 : 2;
    const int w = warp_id(), wf0 = f0 + w * kLanes;
    Real* ring = reinterpret_cast<Real*>(ring_raw) + w * kStagesM * NH * kGroupDv * kLanes;
    const Real* wg = fg + slot(wf0, m.nv_loc);
    const Real* wh = fh + slot(wf0, m.nv_loc);
    // FP32 storage: what rounding took from the mean of tangential pairs on
    // faces between tiles, added after a group (a test in the group's loop cost
    // every case 2 % of its step)
    unsigned tang = 0;   // the segment's DVs with such pairs among the warp's faces
    auto tang_rest = [&](int d, double& g, double& h) {
        const uint2 t = __ldg(m.tang_at + static_cast<size_t>(wf0 / kLanes) * m.nv_loc + d);
        const unsigned bit = 1u << (threadIdx.x % kLanes);
        if (!(t.x & bit)) return;
        const size_t i = chk_place(t.y + static_cast<unsigned>(__popc(t.x & (bit - 1))), m.n_rest, a.ds.err);
        g += double(a.ds.tang_res[i]);
        if (!HZ) h += double(a.ds.tang_res[m.n_rest + i]);
    };
    const bool ok = ring_walk<GEN, kStagesM>(
        m, full + w * kStagesM, s0, wf0 < m.nIF ? s1 : s0, NH * kLanes * sizeof(Real),
        [&](const Seg& q, int j, int n, int stage, uint64_t* bar) {
            Real* dst = ring + stage * NH * kGroupDv * kLanes;
            const size_t o = kLanes * static_cast<size_t>(q.d0 + j);
            bulk_load(dst, wg + o, n * kLanes * sizeof(Real), bar);
            if (!HZ) bulk_load(dst + kGroupDv * kLanes, wh + o, n * kLanes * sizeof(Real), bar);
        },
        [&](const Seg& q, int j, int n, int stage) {
            const Real* st = ring + stage * NH * kGroupDv * kLanes + threadIdx.x % kLanes;
            if constexpr (sizeof(Real) == 4 && !GEN) {
                if (m.tang_at && j == 0)
                    tang = __ldg(m.tang_seg + static_cast<size_t>(wf0 / kLanes) * m.n_seg +
                                 ((q.d0 - q.ix0) / m.n1d << (m.n1d > kSeg)) + q.ix0 / kSeg);
            }
            // FP32 storage: the deviations only; the reference part is added once below
            groups<kGroupDv>(n, [&](int i, auto uc) {
                constexpr int U = decltype(uc)::value;
                const Real* su = st + i * kLanes;
#pragma unroll
                for (int u = 0; u < U; ++u)
                    add_dv<D, HZ, GEN>(acc, rs, w1, q, dv_at<D, GEN>(m, q, x1, j + i + u), j + i + u,
                                       double(su[u * kLanes]), HZ ? 0.0 : double(su[(kGroupDv + u) * kLanes]));
            });
            if constexpr (sizeof(Real) == 4 && !GEN) {
                for (unsigned b = tang & (0xffu << j); b; b &= b - 1) {
                    const int i = __ffs(b) - 1;
                    double g = 0.0, h = 0.0;
                    tang_rest(q.d0 + i, g, h);
                    add_dv<D, HZ, GEN>(acc, rs, w1, q, dv_at<D, GEN>(m, q, x1, i), i, g, h);
                }
            }
            if constexpr (!GEN) {
                if (j + kGroupDv >= q.len) {
                    row_fold<D>(acc, rs, row_const<D>(x1, w1, q));
                    rs = RowSums();
                }
            }
        });
    if (!ok) atomicOr(a.ds.err, 2);
    if constexpr (sizeof(Real) == 4 && !GEN) {
        // an internal face counts every DV in full: the reference's moments once
        if (blockIdx.y == 0)
            for (int j = 0; j < 14; ++j) acc[j] += __ldg(a.ds.refmom + j);
    }
    if (active) {
#pragma unroll
        for (int j = 0; j < 15; ++j) a.ds.partF[(static_cast<size_t>(blockIdx.y) * kNM + j) * nF + f] = acc[j];
    }
    if (a.fused && last_chunk(a.ds.done + bx, last)) finish_face(a, kc, active ? f : -1, gridDim.y);
}

// the finishing part alone, for sharded handles: the chunk sums of all
// shards have been added into chunk 0
__global__ void __launch_bounds__(kFaces) k_finish_faces(const __grid_constant__ StepArgs a,
                                                         const __grid_constant__ Consts kc) {
    const int f = blockIdx.x * kFaces + threadIdx.x;
    finish_face(a, kc, f < a.dm.nF ? f : -1, 1);
}
__global__ void __launch_bounds__(kLanes* kParts) k_finish_cells(const __grid_constant__ StepArgs a,
                                                                 const __grid_constant__ Consts kc) {
    __shared__ Finish sm;
    const int c0 = blockIdx.x * kLanes;
    finish_cells(sm, a, kc, c0, min(kLanes, a.dm.nC - c0), 1);
}

// ---------------------------------------------------------------------
// k_face_flux
// ---------------------------------------------------------------------
// Reads a face value, relaxes it and writes the flux xi.S g_f in its place:
// 16 B per (face, DV) and FP64 field.  The ring's stages carry the faces' e_x
// rows too (from L2).  FP32 storage keeps the flux of the deviation: the
// reference's cancels over a closed cell (sum of +-Sf = 0).
//
// Boundary faces, by patch type.  Outgoing DFs are relaxed, h with the
// internal-face T at the patch-local index (fvDVM.C:1367, :1413, :1429-1444).
// Incoming ones are not: wall rho_w M(U_w, T_w) (fvDVM.C:1079-1092), far field
// and pressure rho_b M(U_owner, T_b) (fvDVM.C:926-938) and mixed
// rho_b M(U_b, T_b); zero-gradient and symmetry ones are stored.
// DVMsymmetry relaxes every DV once more (fvDVM.C:1445-1453).
template <int D, typename Real, bool HZ, bool GEN>
__device__ __noinline__ void boundary_flux(const StepArgs& a, const double* x1, int f, int s0, int s1, int step) {
    const DevMesh& m = a.dm;
    const size_t nF = static_cast<size_t>(m.nF);
    const double S[3] = {__ldg(m.fgeo + f), __ldg(m.fgeo + nF + f), __ldg(m.fgeo + 2 * nF + f)};
    const double K3D = k3d<D>(m), c0h = c0h_of<D>(m);
    Relax<D, HZ, GEN> rx(a.ds.facerec, a.ds.ftab, m.n1d, f, __ldg(a.ds.facerec + slot(f, REC_N) + 32 * REC_R));
    const int b = f - m.nIF, pt = __ldg(m.bface_ptype + b);
    const int li = chk(__ldg(m.bface_patch_local + b), 0, m.nIF, a.ds.err);
    rx.RTh = m.R * a.ds.fm[static_cast<size_t>(li) * 9 + 4];
    const bool stored = pt == DUGKS_PATCH_ZERO_GRADIENT || pt == DUGKS_PATCH_SYMMETRY || pt == DUGKS_PATCH_DVM_SYMMETRY;
    const bool again = pt == DUGKS_PATCH_DVM_SYMMETRY;
    Incoming in{};
    if (!stored) in = load_incoming(a, b, pt);
    for (int s = s0; s < s1; s += step) {
        const Seg q = seg_at<GEN>(m, s);
        rx.row(m, q, x1[q.iy], x1[q.iz]);
        Real g4[4] = {0, 0, 0, 0}, h4[4] = {0, 0, 0, 0};
        for (int j = 0; j < q.len; ++j) {
            const Dv v = dv_at<D, GEN>(m, q, x1, j);
            const size_t o = slot(f, m.nv_loc) + 32 * static_cast<size_t>(q.d0 + j);
            Real* pg = reinterpret_cast<Real*>(a.ds.fvg) + o;
            Real* ph = reinterpret_cast<Real*>(a.ds.fvh) + o;
            if ((j & 3) == 0) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    g4[u] = pg[32 * u];
                    if (!HZ) h4[u] = ph[32 * u];
                }
            }
            const Real gv = g4[0], hv = h4[0];
            g4[0] = g4[1], g4[1] = g4[2], g4[2] = g4[3];
            h4[0] = h4[1], h4[1] = h4[2], h4[2] = h4[3];
            const double xs = xs_dv(v, S), e = rx.factor(q, j);
            const double gr = dv_ref<Real, GEN>(m.gref, q.d0 + j), hr = dv_ref<Real, GEN>(m.href, q.d0 + j);
            double gf = double(gv) + gr, hf = HZ ? 0.0 : double(hv) + hr;
            if (xs > 0) {
                rx(v, e, gf, hf, K3D, c0h, gf, hf);
            } else if (!stored) {
                in.at<D>(v, gf, hf);
                gf = double(Real(gf - gr)) + gr;
                hf = double(Real(hf - hr)) + hr;
            }
            if (again) rx(v, e, gf, hf, K3D, c0h, gf, hf);
            *pg = Real(xs * (gf - gr));
            if (!HZ) *ph = Real(xs * (hf - hr));
        }
    }
}

template <typename Real, bool HZ, bool GEN>
constexpr size_t ring_flux() {
    return static_cast<size_t>(kStagesF) * kGroupDv * kFaces * ((HZ ? 1 : 2) * sizeof(Real) + (GEN ? 0 : sizeof(double)));
}

template <int D, typename Real, bool HZ, bool GEN>
__global__ void __launch_bounds__(kFaces, 4) k_face_flux(const __grid_constant__ StepArgs a) {
    const DevMesh& m = a.dm;
    extern __shared__ __align__(128) unsigned char ring_raw[];
    __shared__ double x1[kMaxN1d], w1[kMaxN1d];
    __shared__ __align__(8) uint64_t full[kParts * kStagesF];
    if (threadIdx.x < kParts * kStagesF) mbar_init(full + threadIdx.x);
    load_nodes(m, x1, w1);
    asm volatile("fence.proxy.async;" ::: "memory");
    __syncthreads();
    const int s0 = seg_begin(m.n_seg, blockIdx.y, gridDim.y), s1 = seg_begin(m.n_seg, blockIdx.y + 1, gridDim.y);
    // boundary face blocks first, as in k_face_moments
    const int nbB = (m.nBF + kLanes - 1) / kLanes, bx = blockIdx.x;
    if (bx < nbB) {
        const int f = m.nIF + bx * kLanes + threadIdx.x % kLanes;
        if (f < m.nF) boundary_flux<D, Real, HZ, GEN>(a, x1, f, s0 + threadIdx.x / kLanes, s1, kParts);
        return;
    }
    const int f0 = (bx - nbB) * kFaces;
    const bool active = f0 + threadIdx.x < m.nIF;
    const int f = active ? f0 + threadIdx.x : f0;
    const size_t nF = static_cast<size_t>(m.nF);
    Real* fg = reinterpret_cast<Real*>(a.ds.fvg) + slot(f, m.nv_loc);
    Real* fh = reinterpret_cast<Real*>(a.ds.fvh) + slot(f, m.nv_loc);
    const double S[3] = {__ldg(m.fgeo + f), __ldg(m.fgeo + nF + f), __ldg(m.fgeo + 2 * nF + f)};
    const double K3D = k3d<D>(m), c0h = c0h_of<D>(m);
    Relax<D, HZ, GEN> rx(a.ds.facerec, a.ds.ftab, m.n1d, f, __ldg(a.ds.facerec + slot(f, REC_N) + 32 * REC_R));
    double p2 = 0, p3 = 0;
    // the warp's 32 faces and ring
    constexpr int NH = HZ ? 1 : 2;
    const int w = warp_id(), wf0 = f0 + w * kLanes;
    Real* ring = reinterpret_cast<Real*>(ring_raw) + w * kStagesF * NH * kGroupDv * kLanes;
    double* ring_e = reinterpret_cast<double*>(reinterpret_cast<Real*>(ring_raw) + kStagesF * NH * kGroupDv * kFaces) +
                     w * kStagesF * kGroupDv * kLanes;
    const Real* wg = reinterpret_cast<const Real*>(a.ds.fvg) + slot(wf0, m.nv_loc);
    const Real* wh = reinterpret_cast<const Real*>(a.ds.fvh) + slot(wf0, m.nv_loc);
    const double* we = a.ds.ftab + slot(wf0, D * m.n1d);
    const bool ok = ring_walk<GEN, kStagesF>(
        m, full + w * kStagesF, s0, wf0 < m.nIF ? s1 : s0, kLanes * (NH * sizeof(Real) + (GEN ? 0 : sizeof(double))),
        [&](const Seg& q, int j, int n, int stage, uint64_t* bar) {
            Real* dst = ring + stage * NH * kGroupDv * kLanes;
            const size_t o = kLanes * static_cast<size_t>(q.d0 + j);
            bulk_load(dst, wg + o, n * kLanes * sizeof(Real), bar);
            if (!HZ) bulk_load(dst + kGroupDv * kLanes, wh + o, n * kLanes * sizeof(Real), bar);
            if (!GEN)
                bulk_load(ring_e + stage * kGroupDv * kLanes, we + kLanes * (q.ix0 + j), n * kLanes * sizeof(double), bar);
        },
        [&](const Seg& q, int j, int n, int stage) {
            if constexpr (!GEN) {
                if (j == 0) {
                    const double Y = x1[q.iy], Z = x1[q.iz];
                    rx.row(m, q, Y, Z);
                    p2 = __dmul_rn(Y, S[1]);
                    p3 = D == 3 ? __dmul_rn(Z, S[2]) : 0.0;
                }
            }
            const Real* st = ring + stage * NH * kGroupDv * kLanes + threadIdx.x % kLanes;
            const double* se = ring_e + stage * kGroupDv * kLanes + threadIdx.x % kLanes;
            Real *gs = fg + 32 * static_cast<size_t>(q.d0 + j), *hs = fh + 32 * static_cast<size_t>(q.d0 + j);
            groups<HZ ? kGroupDv : 4>(n, [&](int i, auto uc) {
                constexpr int U = decltype(uc)::value;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const Dv v = dv_at<D, GEN>(m, q, x1, j + i + u);
                    double xs;
                    if constexpr (GEN) xs = xs_dv(v, S);
                    else xs = __dadd_rn(__dadd_rn(__dmul_rn(v.x, S[0]), p2), p3);
                    const int d = q.d0 + j + i + u;
                    const double gr = dv_ref<Real, GEN>(m.gref, d), hr = dv_ref<Real, GEN>(m.href, d);
                    double gf, hf;
                    const Real* su = st + i * kLanes;
                    rx(v, GEN ? 0.0 : (se + i * kLanes)[u * kLanes], double(su[u * kLanes]) + gr,
                       HZ ? 0.0 : double(su[(kGroupDv + u) * kLanes]) + hr, K3D, c0h, gf, hf);
                    if (active) {
                        (gs + 32 * i)[32 * u] = Real(xs * (gf - gr));
                        if (!HZ) (hs + 32 * i)[32 * u] = Real(xs * (hf - hr));
                    }
                }
            });
        });
    if (!ok) atomicOr(a.ds.err, 2);
}

// ---------------------------------------------------------------------
// k_update
// ---------------------------------------------------------------------
// One thread per cell and DV segment: gathers the fluxes of the cell's faces
// (owner side: outflow, negated), updates g~ in place and sums the cell's
// moments.  A flux is read by the two cells of its face; the second read hits L2.
template <int D, typename Real, bool HZ, bool GEN, int NS, typename Off>
__global__ void __launch_bounds__(kLanes* kParts, 4) k_update(const __grid_constant__ StepArgs a,
                                                           const __grid_constant__ Consts kc) {
    const DevMesh& m = a.dm;
    __shared__ double x1[kMaxN1d], w1[kMaxN1d];
    __shared__ Finish sm;
    load_nodes(m, x1, w1);
    const int c0 = blockIdx.x * kLanes, count = min(kLanes, m.nC - c0);
    const int lane = threadIdx.x % kLanes, c = c0 + lane;
    const size_t nC = static_cast<size_t>(m.nC);
    const int s0 = seg_begin(m.n_seg, blockIdx.y, gridDim.y), s1 = seg_begin(m.n_seg, blockIdx.y + 1, gridDim.y);
    const int w = warp_id();
    Sums<GEN> acc(sm);
    // macroFlux yes with a DV list (fvDVM.C:1562-1611): the cell's rho, rho U,
    // rho E gain sum_DV w (1, xi, |xi|^2/2 & h/2) times the flux term
    // dt/V sum_f (+-)(xi.S) g_f of the update
    double accx[5] = {0, 0, 0, 0, 0};
    const bool fx = GEN && m.macro_flux;
    if (lane < count) {
        Real* g = reinterpret_cast<Real*>(a.ds.g) + slot(c, m.nv_loc);
        Real* h = reinterpret_cast<Real*>(a.ds.h) + slot(c, m.nv_loc);
        const Real* __restrict__ fvg = reinterpret_cast<const Real*>(a.ds.fvg);
        const Real* __restrict__ fvh = reinterpret_cast<const Real*>(a.ds.fvh);
        const double dtV = step_dt(a) * __ldg(m.invV + c);
        const double K3D = k3d<D>(m), c0h = c0h_of<D>(m);
        Relax<D, HZ, GEN> rx(a.ds.cellrec, a.ds.ctab, m.n1d, c, cell_r(a, c));
        // faces with their sign (owner side: outflow, -1); an absent slot
        // repeats the first face with sign 0
        Off fc[NS];
        Real sign[NS];
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            const int code = k < m.nf_max ? chk(__ldg(m.cface + k * nC + c), -1, 4 * m.nF, a.ds.err) : -1;
            fc[k] = code < 0 ? fc[0] : static_cast<Off>(slot(code >> 2, m.nv_loc));
            sign[k] = code < 0 ? Real(0) : (code & 1) ? Real(1) : Real(-1);
        }
        RowSums rs;
        for (int s = s0 + w; s < s1; s += kParts) {
            const Seg q = seg_at<GEN>(m, s);
            rx.row(m, q, x1[q.iy], x1[q.iz]);
            rs = RowSums();
            groups<HZ || sizeof(Real) == 4 ? 4 : 2>(q.len, [&](int j, auto uc) {
                constexpr int U = decltype(uc)::value;
                struct {
                    Real g[U], h[U], fg[U][NS], fh[U][NS];
                    double e[U];
                } b;
                const size_t dj = 32 * static_cast<size_t>(q.d0 + j);
                Real *gs = g + dj, *hs = h + dj;
                const Real *fgs = fvg + dj, *fhs = fvh + dj;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    b.g[u] = gs[32 * u];
                    if (!HZ) b.h[u] = hs[32 * u];
                    b.e[u] = rx.factor(q, j + u);
#pragma unroll
                    for (int k = 0; k < NS; ++k) {
                        b.fg[u][k] = __ldg(fgs + fc[k] + 32 * u);
                        if (!HZ) b.fh[u][k] = __ldg(fhs + fc[k] + 32 * u);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    {
                        const Dv v = dv_at<D, GEN>(m, q, x1, j + u);
                        const double gr = dv_ref<Real, GEN>(m.gref, q.d0 + j + u),
                                     hr = dv_ref<Real, GEN>(m.href, q.d0 + j + u);
                        double gb, hb;
                        rx(v, b.e[u], double(b.g[u]) + gr, HZ ? 0.0 : double(b.h[u]) + hr, K3D, c0h, gb, hb);
                        // (a product with +-1 is exact: the sum in slot order)
                        Real sg = 0, sh = 0;
    #pragma unroll
                        for (int k = 0; k < NS; ++k) {
                            sg = fma(sign[k], b.fg[u][k], sg);
                            if (!HZ) sh = fma(sign[k], b.fh[u][k], sh);
                        }
                        if (m.nf_max > NS) {
                            for (int k = NS; k < m.nf_max; ++k) {
                                const int code = chk(__ldg(m.cface + k * nC + c), -1, 4 * m.nF, a.ds.err);
                                if (code < 0) break;
                                const size_t of = slot(code >> 2, m.nv_loc) + 32 * u;
                                const Real sk = (code & 1) ? Real(1) : Real(-1);
                                sg = fma(sk, __ldg(fgs + of), sg);
                                if (!HZ) sh = fma(sk, __ldg(fhs + of), sh);
                            }
                        }
                        // the update in FP64, one rounding to the storage type; with a
                        // reference, -g/3 + 4/3 gbar+ - ref = -(g - ref)/3 + 4/3 (gbar+ - ref)
                        const Real gn = Real(fma(-1.0 / 3, double(b.g[u]), fma(4.0 / 3, gb - gr, double(sg) * dtV)));
                        gs[32 * u] = gn;
                        Real hn = 0;
                        if (!HZ) {
                            hn = Real(fma(-1.0 / 3, double(b.h[u]), fma(4.0 / 3, hb - hr, double(sh) * dtV)));
                            hs[32 * u] = hn;
                        }
                        add_dv<D, HZ, GEN>(acc, rs, w1, q, v, j + u, double(gn), double(hn));
                        if constexpr (GEN) {
                            if (fx) {
                                const double fgd = double(sg) * dtV, fhd = double(sh) * dtV, aw = v.w * fgd;
                                accx[0] += aw;
                                accx[1] += aw * v.x;
                                accx[2] += aw * v.y;
                                accx[3] += aw * v.z;
                                accx[4] += 0.5 * v.w * (fgd * (v.x * v.x + v.y * v.y + v.z * v.z) + fhd);
                            }
                        }
                    }
                }
            });
            if constexpr (!GEN) row_fold<D>(acc, rs, row_const<D>(x1, w1, q));
        }
        if constexpr (sizeof(Real) == 4 && !GEN) {
            // FP32 storage: the reference's moments once
            if (blockIdx.y == 0 && threadIdx.x < kLanes)
                for (int j = 0; j < 14; ++j) acc[j] += __ldg(a.ds.refmom + j);
        }
    }
    if constexpr (GEN) {
        if (fx) {
            // the flux term's moments of the chunk, in warp order
            for (int j = 0; j < 5; ++j) sm.red[w][j][lane] = accx[j];
            __syncthreads();
            for (int j = w; j < 5; j += kParts) {
                double v = sm.red[0][j][lane];
                for (int p = 1; p < kParts; ++p) v += sm.red[p][j][lane];
                if (lane < count) a.ds.partX[(static_cast<size_t>(blockIdx.y) * kFX + j) * nC + c] = v;
            }
            __syncthreads();
        }
    }
    acc.put(sm);
    if (reduce_chunk(sm, a.ds.partC, nC, c0, count, a.ds.done + m.done_cells + blockIdx.x, a.fused != 0))
        finish_cells(sm, a, kc, c0, count, gridDim.y);
}

// raw cell moments of the current state (set_state), as k_update sums them
template <int D, typename Real, bool GEN>
__global__ void __launch_bounds__(kLanes* kParts) k_state_moments(const __grid_constant__ StepArgs a,
                                                                  const __grid_constant__ Consts kc) {
    const DevMesh& m = a.dm;
    __shared__ double x1[kMaxN1d], w1[kMaxN1d];
    __shared__ Finish sm;
    load_nodes(m, x1, w1);
    const int c0 = blockIdx.x * kLanes, count = min(kLanes, m.nC - c0);
    const int lane = threadIdx.x % kLanes, c = c0 + lane;
    const size_t nC = static_cast<size_t>(m.nC);
    const int s0 = seg_begin(m.n_seg, blockIdx.y, gridDim.y), s1 = seg_begin(m.n_seg, blockIdx.y + 1, gridDim.y);
    const int w = warp_id();
    Sums<GEN> acc(sm);
    if (lane < count) {
        const Real* __restrict__ g = reinterpret_cast<const Real*>(a.ds.g) + slot(c, m.nv_loc);
        const Real* __restrict__ h = reinterpret_cast<const Real*>(a.ds.h) + slot(c, m.nv_loc);
        for (int s = s0 + w; s < s1; s += kParts) {
            const Seg q = seg_at<GEN>(m, s);
            RowSums rs;
#pragma unroll 4
            for (int j = 0; j < q.len; ++j) {
                const size_t o = 32 * static_cast<size_t>(q.d0 + j);
                const double gr = dv_ref<Real, GEN>(m.gref, q.d0 + j), hr = dv_ref<Real, GEN>(m.href, q.d0 + j);
                add_dv<D, false, GEN>(acc, rs, w1, q, dv_at<D, GEN>(m, q, x1, j), j, double(__ldg(g + o)) + gr,
                                      double(__ldg(h + o)) + hr);
            }
            if constexpr (!GEN) row_fold<D>(acc, rs, row_const<D>(x1, w1, q));
        }
    }
    acc.put(sm);
    if (reduce_chunk(sm, a.ds.partC, nC, c0, count, a.ds.done + m.done_cells + blockIdx.x, a.fused != 0))
        finish_cells(sm, a, kc, c0, count, gridDim.y);
}

int blocks(int n, int per) { return (n + per - 1) / per; }

// CTAs along the DV segments for the kernels without a reduction: about
// eight CTAs of 128 threads on each SM, `waves` times over, so that the
// last wave is short.  (Two for k_face_flux, whose rings and boundary records
// each CTA sets up: 1,728 cells and 10^3 DVs 147 us a step, four 159; the
// others are level from two to eight.)
int stream_chunks(const DevMesh& m, int n_seg, int nb, int waves = 4) {
    const int target = m.sms * 8 * waves;
    return std::max(1, std::min({n_seg, (target + nb - 1) / std::max(nb, 1), 65535}));
}

template <int D, typename Real, bool HZ, bool GEN>
cudaError_t launch_kernel(const StepArgs& a, int which, cudaStream_t s) {
    const DevMesh& m = a.dm;
    const Consts k = make_consts(m, a.dt);
    const int nbF = blocks(m.nIF, kFaces) + blocks(m.nBF, kLanes);
    const bool quad = m.nb_max <= 4 && m.nf_max <= 4;   // quadrilaterals, tetrahedra: shorter face lists
    // (with room for the constant offsets of a group)
    const bool wide = static_cast<unsigned long long>(m.nv_loc) * m.pF + kSlack >= 1ull << 32;
    switch (which) {
        case KERNEL_HALF_STEP: {
            const int nb = blocks(m.nC, kStream);
            k_half_step<D, Real, HZ, GEN><<<dim3(nb, stream_chunks(m, a.seg1 - a.seg0, nb)), kStream, 0, s>>>(a);
            break;
        }
        case KERNEL_FACE_VALUES: {
            const int nb = blocks(m.nC, kCells);
            const dim3 grid(nb, stream_chunks(m, a.seg1 - a.seg0, nb));
            if (wide) k_face_values<D, Real, HZ, GEN, kFast, size_t><<<grid, kCells, 0, s>>>(a);
            else if (quad) k_face_values<D, Real, HZ, GEN, 4, unsigned><<<grid, kCells, 0, s>>>(a);
            else k_face_values<D, Real, HZ, GEN, kFast, unsigned><<<grid, kCells, 0, s>>>(a);
            break;
        }
        case KERNEL_TANGENTIAL: {
            const long long nb = (m.n_tang + kStream - 1) / kStream;
            k_tangential<D, Real, HZ, GEN><<<static_cast<int>(std::min<long long>(nb, m.sms * 64)), kStream, 0, s>>>(a);
            break;
        }
        case KERNEL_ZERO_GRADIENT:
            if (m.nBF > 0) k_zero_gradient<Real><<<blocks(m.nBF, kLanes), kStream, 0, s>>>(a);
            break;
        case KERNEL_FACE_MOMENTS:
            if (m.nv_bar < m.nv_loc)
                k_face_moments<D, Real, HZ, GEN, true><<<dim3(nbF, a.chunks_f), kFaces, ring_moments<Real, HZ>(), s>>>(a, k);
            else
                k_face_moments<D, Real, HZ, GEN, false><<<dim3(nbF, a.chunks_f), kFaces, ring_moments<Real, HZ>(), s>>>(a, k);
            break;
        case KERNEL_FACE_FLUX: {
            k_face_flux<D, Real, HZ, GEN>
                <<<dim3(nbF, stream_chunks(m, m.n_seg, nbF, 2)), kFaces, ring_flux<Real, HZ, GEN>(), s>>>(a);
            break;
        }
        case KERNEL_UPDATE: {
            const dim3 grid(blocks(m.nC, kLanes), a.chunks);
            if (wide) k_update<D, Real, HZ, GEN, kFast, size_t><<<grid, kLanes * kParts, 0, s>>>(a, k);
            else if (quad) k_update<D, Real, HZ, GEN, 4, unsigned><<<grid, kLanes * kParts, 0, s>>>(a, k);
            else k_update<D, Real, HZ, GEN, kFast, unsigned><<<grid, kLanes * kParts, 0, s>>>(a, k);
            break;
        }
        case KERNEL_STATE_MOMENTS:
            k_state_moments<D, Real, GEN><<<dim3(blocks(m.nC, kLanes), a.chunks), kLanes * kParts, 0, s>>>(a, k);
            break;
        default:
            return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// dynamic shared memory of the rings (above the default limit)
template <int D, typename Real, bool HZ, bool GEN>
cudaError_t allow_rings() {
    auto allow = [](auto* kernel, size_t bytes) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    };
    cudaError_t e = allow(k_face_moments<D, Real, HZ, GEN, false>, ring_moments<Real, HZ>());
    if (e == cudaSuccess) e = allow(k_face_moments<D, Real, HZ, GEN, true>, ring_moments<Real, HZ>());
    return e != cudaSuccess ? e : allow(k_face_flux<D, Real, HZ, GEN>, ring_flux<Real, HZ, GEN>());
}

template <int D, typename Real>
cudaError_t launch_d(const StepArgs& a, int which, cudaStream_t s) {
    if (a.dm.general_dv) return launch_kernel<D, Real, false, true>(a, which, s);
    if constexpr (D == 3) {
        if (a.hzero) return launch_kernel<D, Real, true, false>(a, which, s);
    }
    return launch_kernel<D, Real, false, false>(a, which, s);
}

}  // namespace

cudaError_t launch_pass(const StepArgs& a, int precision, int which, cudaStream_t s) {
    if (precision == DUGKS_FP64) return a.dm.D == 3 ? launch_d<3, double>(a, which, s) : launch_d<2, double>(a, which, s);
    return a.dm.D == 3 ? launch_d<3, float>(a, which, s) : launch_d<2, float>(a, which, s);
}

template <int D, typename Real>
static cudaError_t configure_d() {
    cudaError_t e = allow_rings<D, Real, false, false>();
    if (e == cudaSuccess) e = allow_rings<D, Real, false, true>();
    if constexpr (D == 3) {
        if (e == cudaSuccess) e = allow_rings<D, Real, true, false>();
    }
    return e;
}

cudaError_t configure_kernels(int D, int precision) {
    if (precision == DUGKS_FP64) return D == 3 ? configure_d<3, double>() : configure_d<2, double>();
    return D == 3 ? configure_d<3, float>() : configure_d<2, float>();
}

cudaError_t launch_finish(const StepArgs& a, bool faces, cudaStream_t s) {
    const Consts k = make_consts(a.dm, a.dt);
    if (faces) k_finish_faces<<<blocks(a.dm.nF, kFaces), kFaces, 0, s>>>(a, k);
    else k_finish_cells<<<blocks(a.dm.nC, kLanes), kLanes * kParts, 0, s>>>(a, k);
    return cudaGetLastError();
}

cudaError_t launch_cell_records(const StepArgs& a, cudaStream_t s) {
    k_cell_records<<<blocks(a.dm.nC, kLanes), kLanes * kParts, 0, s>>>(a, make_consts(a.dm, a.dt));
    return cudaGetLastError();
}

cudaError_t launch_upwind_bits(const DevMesh& m, uint32_t* upw, unsigned long long* n, cudaStream_t s) {
    // (FP32 storage of a tensor DV set: DevMesh::tang_at)
    const bool tiles = m.prec == DUGKS_FP32C && !m.general_dv;
    const int nb = blocks(m.nF, 128);
    const dim3 grid(nb, std::min(m.n_seg, std::max(1, m.sms * 32 / std::max(nb, 1))));
    if (m.general_dv) {
        if (m.D == 3) k_upwind_bits<3, true><<<grid, 128, 0, s>>>(m, upw, tiles, n);
        else k_upwind_bits<2, true><<<grid, 128, 0, s>>>(m, upw, tiles, n);
    } else {
        if (m.D == 3) k_upwind_bits<3, false><<<grid, 128, 0, s>>>(m, upw, tiles, n);
        else k_upwind_bits<2, false><<<grid, 128, 0, s>>>(m, upw, tiles, n);
    }
    return cudaGetLastError();
}

cudaError_t launch_list_tangential(const DevMesh& m, int2* list, unsigned long long* cursor, uint2* at, unsigned* seg,
                                   cudaStream_t s) {
    const int nb = blocks(m.nIF, 128);
    const dim3 grid(nb, std::min(m.n_seg, std::max(1, m.sms * 32 / std::max(nb, 1))));
    if (m.general_dv) k_list_tangential<true><<<grid, 128, 0, s>>>(m, list, cursor, at, seg);
    else k_list_tangential<false><<<grid, 128, 0, s>>>(m, list, cursor, at, seg);
    return cudaGetLastError();
}

}  // namespace dugks
