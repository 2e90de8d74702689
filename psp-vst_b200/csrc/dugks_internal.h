// Internal declarations of the B200 DUGKS step library: device layout,
// cell and face tables and the handle.  Not part of the public ABI.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "dugks.h"

namespace dugks {

// tiles: what FP32 rounds by (Tiling) and dugks_layout reports; a mesh that does
// not fit them is refused
constexpr int kMaxTile = 128;      // cells per tile at most
constexpr int kMaxLocal = 256;     // cells of a tile with its ring of neighbours at most
constexpr int kMaxItems = 511;     // faces of a tile's cells at most
constexpr int kSeg = 32;           // DVs per segment at most (one bit each in DevMesh::upw)
constexpr int kSlack = 1024;       // elements to spare behind the (entity, DV) arrays (group loads read past a segment)
constexpr int kMaxN1d = 64;        // DV nodes per dimension at most
constexpr int kNM = 16;            // stride of a partial-moment record (doubles)
constexpr int kFX = 8;             // stride of a flux-moment record: M0, M1[3], W/2
constexpr double kVSmall = 1.0e-300;  // OpenFOAM VSMALL (upwind switch, fvDVM.C:829-847)

// Moment record layout (raw velocity moments of one face or cell, summed
// over DVs; a = w g, b = w h, u = a|xi|^2 + b):
//   0 M0 = sum a            1..3  M1 = sum a xi
//   4 W  = sum u            5..7  V3 = sum u xi
//   8..13 M2 = sum a xi xi (xx xy xz yy yz zz)
//   14 outgoing wall flux  sum_{xi.S>0} w (xi.S) gbar   (faces only)
enum {
    MOM_M0 = 0, MOM_M1 = 1, MOM_W = 4, MOM_V3 = 5, MOM_M2 = 8, MOM_OUT = 14
};

// Fields of the coefficient records.  Cell records (gbar+ half step,
// fvDVM.C:668-679) and face records (face relaxation, fvDVM.C:1374-1444)
// share them.
enum {
    REC_UX = 0, REC_UY = 1, REC_UZ = 2,
    REC_INVRT = 3,   // 1/(R T)
    REC_A = 4,       // rho (2 pi R T)^(-D/2)
    REC_R = 5,       // faces: relax factor 0.5 dt/(2 tau + 0.5 dt); cells: tau (the factor follows the step's dt)
    REC_QX = 6, REC_QY = 7, REC_QZ = 8,   // (1-Pr) q / (5 rho (R T)^2)
    REC_RTH = 9,     // R T used by h^S (boundary faces: the internal-face T at the patch-local index)
    REC_N = 10
};

// Incoming-DF parameters of a mesh-boundary face: g_in = rho_in K_in exp(-|U_in - xi|^2 invRT_in / 2),
// h_in = g_in * hfac (fvDVM.C:926-938, :1079-1092).
struct __align__(16) BRec {
    double U[3];       // wall and mixed: patch velocity (farField: the owner-cell U is taken)
    double K_in;       // (2 pi R T_in)^(-D/2)
    double invRT_in;
    double hfac;       // R T_in (K+3-D)
    double rho_in;     // farField, mixed: fixed patch rho; wall: rho_w of the current step;
                       // pressureIn/Out: updated after each step
    double inByRho;    // wall: inComingByRho
    double T;          // T_in
    double p;          // pressureIn / pressureOut value
};

// Device-side view of everything the kernels read.
struct DevMesh {
    int D, K;
    double R, Pr, omega, Tref, muRef;
    int nC, nIF, nBF, nF, nv;
    // (entity, DV) arrays hold blocks of 32 cells or faces, [block][dv][32]:
    // entity e, DV d is element ((e / 32) nv_loc + d) 32 + e % 32.  Records
    // and Maxwellian tables alike: [block][field][32].  pC, pF: nC, nF padded
    int pC, pF;
    int sms;               // multiprocessors of the device
    int* err;              // DevState::err, for the bounds-checked build
    // DVs this device holds: global DVs dv_base .. dv_base + nv_loc - 1, the
    // DV rows row_base ..
    int nv_loc, dv_base, row_base;
    int prec;              // dugks_precision of the state and tables
    // DV set
    const double* xi;      // [nv*3]
    const double* w;       // [nv]
    int n1d;               // nodes per dimension; DV d = (iz n + iy) n + ix
    int general_dv;        // 1: a DV list that is no tensor product (n1d is 1, a "row" is one DV)
    const double* X1;      // [n1d] one-dimensional nodes
    const double* W1;      // [n1d] one-dimensional weights
    // DV segments: up to kSeg consecutive DVs of one row (of the list); the
    // kernels walk DVs by segments and DV chunks are runs of segments
    int n_seg;
    // gbar+ and hbar+ hold nv_bar DVs at a time, those of seg_bar segments: all
    // of them, or as many as memory allowed; pass A then walks the DVs in parts
    int seg_bar, nv_bar;
    const int2* row_yz;            // y and z index of every row of this device
    // Cells in the renumbered order.  Faces in the order of the step's arrays:
    // internal faces grouped by blocks of 32 cells, first faces of a block's
    // cells first, so that neighbouring cells reach neighbouring faces; then
    // the boundary faces in the caller's order.
    int nb_max, nf_max;
    const int32_t* nbr;            // [nb_max][nC] neighbour cells (absent: the cell itself)
    const double* nbr_ls;          // [nb_max][3][nC] least-squares vectors (absent: 0)
    const int32_t* cface;          // [nf_max][nC] faces of a cell: 2 face + (1 if the cell is the neighbour), -1 none
    const double* invV;            // [nC]
    const double* fgeo;            // [9][nF]: S, Cf - C_own, Cf - C_nei
    const int32_t* fown;           // [nF] owner cell
    const int32_t* fnei;           // [nIF] neighbour cell
    const int32_t* forig;          // [nF] the caller's face
    const uint32_t* upw;           // [n_seg][nF][2] upwind bits of a segment's DVs: owner side, neighbour side
    const int2* tang;              // [n_tang] exactly tangential pairs: internal face, segment * kSeg + DV in it
    long long n_tang, n_rest;      // n_rest: FP32 storage of a tensor DV set, those of faces between tiles
    // where the rests of those are, by face block (null without any): the faces
    // that have one at a DV (a bit each) and the first one's place; and the DVs
    // of a segment with any
    const uint2* tang_at;          // [pF/32][nv_loc]
    const unsigned* tang_seg;      // [pF/32][n_seg]
    int done_cells;                // first cell-block counter in DevState::done (face blocks before it)
    const int32_t* bface_patch_local;  // [nBF] index within its patch
    const int32_t* bface_ptype;    // [nBF]
    const int32_t* bface_owner;    // [nBF] renumbered owner cell
    const int32_t* bface_mirror;   // [nBF] symmetry faces: mirrored DV axis 0..2; -1 otherwise
    int n_sym_faces, n_pressure_faces;
    // macroFlux yes: faces of each (renumbered) cell in face order, entry
    // f * 2 + (1 if the cell is the neighbour); face area vectors and volumes
    int macro_flux;
    const int32_t* mf_off;         // [nC+1]
    const int32_t* mf_ent;         // [2 nIF + nBF]
    const double* mf_Sf;           // [nF*3]
    const double* mf_V;            // [nC] renumbered
    const double* dc;              // [nIF] deltaCoeffs
    const double* bS;              // [nBF*3] boundary face area vectors
    double xi_max_co;              // sqrt(D) * xiMax
    // FP32 storage of a tensor DV set: g~, gbar+, the face values and the
    // fluxes are stored as deviations from a per-DV reference Maxwellian,
    // g = stored + gref[d] (h likewise), so that FP32 rounding acts on the
    // deviation only; null for FP64 and for DV lists (absolute storage)
    const double* gref;            // [nv_loc] local DVs
    const double* href;
};

// Mutable device state
struct DevState {
    void* g;           // state g~ (cells, Real), updated in place
    void* h;
    void* gbar;        // gbar+ of the step (cells, Real, nv_bar DVs)
    void* hbar;        // (null while h is identically zero)
    // face values (faces, Real): the upwind reconstruction at the half step,
    // then, relaxed and multiplied by xi.S, the flux
    void* fvg;
    void* fvh;         // (null while h is identically zero)
    float* tang_res;   // [2][n_rest] g and h: what rounding took from those pairs' means
    double* partF;     // [chunks_f][kNM][nF]
    double* partC;     // [chunks][kNM][nC]
    double* partX;     // [chunks][kFX][nC] DV-list macroFlux: moments of the flux term (else null)
    double* redC;      // sharded DV-list macroFlux: [kNM][nC] cell moments then [kFX][nC] flux moments, reduced together
    int* done;         // chunks finished per face block, then per cell block; zero between launches
    double* cellrec;   // cells, REC_N fields
    double* facerec;   // faces, REC_N fields
    // one-dimensional Maxwellian factors, FP64 for both precisions (the
    // equilibrium and the relaxation are evaluated in FP64, so that the FP32
    // path injects no rounding bias into the conserved moments): table k of
    // entity e at node i is field k * n1d + i of D n1d: exp(-(X_i - U_k)^2 /
    // (2 R T)), the x table multiplied by A = rho (2 pi R T)^(-D/2)
    double* ctab;
    double* ftab;
    BRec* brec;        // [nBF]
    double* bmom_in;   // [nBF][kNM] incoming wall moments per unit rho_w
    double* cm;        // cell macros [nC][9]: rho U(3) T q(3) tau (renumbered)
    // FP32 storage of a tensor DV set: the raw moments of the reference
    // Maxwellian over this device's DVs, [kNM] (null otherwise); a face or
    // cell whose DVs all count in full adds them once instead of per DV
    double* refmom;
    double* fm;        // face macros [nF][9], the caller's face order
    double* co;        // [2] Courant max (as ordered bits) and sum
    int* err;          // [4] device error flags
};

// Cell and face order of the device arrays and the tables built on them
struct Tiling {
    int n_tiles = 0;
    int tile_cells = 0;             // cells of the largest tile
    bool fits = true;               // every tile keeps the limits above
    int nb_max = 0, nf_max = 0;
    std::vector<int32_t> perm;      // new -> old cell
    std::vector<int32_t> iperm;     // old -> new
    std::vector<int32_t> forig;     // new -> caller's face
    std::vector<int32_t> fnew;      // caller's -> new face
    std::vector<int32_t> fown, fnei;
    std::vector<double> fgeo;       // [9][nF]
    std::vector<int32_t> nbr;       // [nb_max][nC]
    std::vector<double> nbr_ls;     // [nb_max][3][nC]
    std::vector<int32_t> cface;     // [nf_max][nC]
};

}  // namespace dugks

struct dugks_handle {
    int device = 0;
    int precision = DUGKS_FP64;
    int D = 3;
    int nC = 0, nIF = 0, nBF = 0, nP = 0, nv = 0, n1d = 0;
    dugks_gas gas{};
    double xi_max = 0;
    std::vector<int32_t> patch_type, patch_start;
    std::vector<int32_t> bface_ptype, bface_patch_local;
    std::vector<double> bc_rho, bc_U, bc_T, bc_p;
    std::vector<int32_t> bface_mirror;   // symmetry faces: mirrored DV axis; -1 otherwise
    std::vector<double> xi, w;      // tensor-product DV set
    std::vector<double> X1, W1;     // one-dimensional nodes and weights
    std::vector<double> gref, href; // host copy of the FP32-storage reference (empty: none)
    // geometry (original numbering)
    std::vector<int64_t> owner, neighbour;
    std::vector<double> C, V, Cf, Sf, weights, dc, lsP, lsN, lsB;
    dugks::Tiling tiling;
    int chunks = 1, chunks_f = 1;       // DV chunks of the cell and of the face reductions
    // velocity-space shard (world 1: the whole DV set)
    int shard_rank = 0, shard_world = 1;
    bool shard_nccl = false;
    void* nccl_comm = nullptr;          // ncclComm_t
    int shard_phase_next = 0;           // dugks_shard_phase: the phase expected next
    double shard_dt = 0;                // dugks_shard_phase: dt of the step in progress
    // device
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    dugks::DevMesh dm{};
    dugks::DevState ds{};
    std::vector<void*> allocations;
    bool counted = false;           // among its device's handles (dugks_arena.h)
    int32_t* d_iperm = nullptr;     // Tiling::iperm
    double* d_dt = nullptr;         // [2] device time steps of adaptive stepping (ping-pong)
    double* d_hist = nullptr;       // time steps of the last adaptive call
    int32_t hist_cap = 0;
    bool initialised = false;
    // h~ is identically zero: D = 3 and KInner = 0 make K + 3 - D = 0 in
    // every formula that feeds h (initial state, equilibria, boundary
    // DFs), so h stays zero unless dugks_set_state loads a nonzero h~
    bool h_zero = false;
    long steps_done = 0;
    int64_t launches = 0;           // kernels launched by this handle
    double last_step_ms = 0;
    double* host_cm = nullptr;      // pinned staging of the cell macros (dugks_get_macros)
    std::string last_error;
};

namespace dugks {
// host preparation (dugks_host.cpp)
void compute_weights_and_ls(dugks_handle* h, int weighting);
void build_tiling(dugks_handle* h, int tile_cells);
int set_error(dugks_handle* h, int code, const std::string& msg);
// ABI helpers (dugks_abi.cpp): cell records and tables from ds.cm
int rebuild_cell_records(dugks_handle* h);
// the step's face values at the half step (DevState::fvg, fvh) and their raw
// moments (partF, chunks_f chunks) for a step of size dt from the current
// state, which stays as it is
int record_face_values(dugks_handle* h, double dt);
}  // namespace dugks
