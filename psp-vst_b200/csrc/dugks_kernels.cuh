// Launch interface of the DUGKS step kernels (dugks_kernels.cu).
#pragma once

#include "dugks_internal.h"

namespace dugks {

struct StepArgs {
    DevMesh dm;
    DevState ds;
    double dt;
    int chunks, chunks_f;        // DV chunks of the cell and of the face reductions
    // device-resident time step (adaptive stepping): when set, the kernels
    // read this step's dt from *dtp
    const double* dtp;
    // 1: h is identically zero (3-D, KInner = 0, h~ = 0 in the state): the
    // tensor-DV kernels carry g alone
    int hzero;
    // 1: the reducing kernels form the macros when an entity's last chunk is
    // done; 0: they leave the chunk sums (sharded handles reduce them first)
    int fused;
    int keep_co;                 // 1: leave the Courant sums of the last step
    // the part of pass A whose gbar+ is held: segments seg0 .. seg1 - 1, the
    // first at local DV d_bar (all segments but where DevMesh::seg_bar is less)
    int seg0, seg1, d_bar;
};

enum { STAGE_PASS_A = 0, STAGE_FACE_COMBINE = 1, STAGE_PASS_B = 2, STAGE_CELL_COMBINE = 3 };

// kernels of dugks_passes.cu
enum {
    KERNEL_HALF_STEP = 0, KERNEL_FACE_VALUES = 1, KERNEL_FACE_MOMENTS = 2, KERNEL_FACE_FLUX = 3, KERNEL_UPDATE = 4,
    KERNEL_STATE_MOMENTS = 5, KERNEL_TANGENTIAL = 6, KERNEL_ZERO_GRADIENT = 7
};

// first segment of DV chunk k of n
__host__ __device__ __forceinline__ int seg_begin(int n_seg, int k, int n) {
    return static_cast<int>(static_cast<long long>(n_seg) * k / n);
}

// first local DV of segment s
__host__ __device__ __forceinline__ int seg_dv(const DevMesh& m, int s) {
    if (m.general_dv) return s * kSeg;
    const int two = m.n1d > kSeg;   // n1d <= 64: one or two segments a row
    return (s >> two) * m.n1d + (s & two) * kSeg;
}

// Bounds-checked build (-DDUGKS_CHECK, libdugks_b200_check.so): every index
// the kernels read from a device table is tested against its range before
// use.  One outside [lo, hi) sets bit 2 (value 4) of the handle's error
// flags and is replaced by lo, so the access stays in bounds; the host then
// returns DUGKS_ERR_ARG.  In the normal build the check is the index itself.
#ifdef DUGKS_CHECK
__device__ __forceinline__ int chk(int i, int lo, int hi, int* err) {
    if (i < lo || i >= hi) {
        atomicOr(err, 4);
        return lo;
    }
    return i;
}
// place i of a list of n
__device__ __forceinline__ size_t chk_place(size_t i, size_t n, int* err) {
    if (i >= n) {
        atomicOr(err, 4);
        return 0;
    }
    return i;
}
#else
__device__ __forceinline__ int chk(int i, int, int, int*) { return i; }
__device__ __forceinline__ size_t chk_place(size_t i, size_t, int*) { return i; }
#endif

// one stage of a DUGKS step (fvDVM::evolution) on stream s; `launches` (may be
// null) is incremented by the kernels launched.  Pass A: half step, face
// values, face moments; pass B: face fluxes, update.  The combine stages
// launch kernels only where the reducing kernels leave them the work (fused 0)
// and for the pressure patches.
cudaError_t launch_stage(const StepArgs& a, int precision, int stage, cudaStream_t s, int* launches);
// g~, h~ = Maxwellian; wall inComingByRho and incoming-moment vectors
cudaError_t launch_init(const StepArgs& a, int precision, cudaStream_t s);
// one kernel of dugks_passes.cu
cudaError_t launch_pass(const StepArgs& a, int precision, int which, cudaStream_t s);
// face (or cell) macros and records from the sums in chunk 0
cudaError_t launch_finish(const StepArgs& a, bool faces, cudaStream_t s);
// kernel attributes on the current device
cudaError_t configure_kernels(int D, int precision);
// DevMesh::upw from the geometry and the DV set, with the numbers n_tang and
// n_rest of tangential (internal face, DV) pairs in n[2], and their list
// DevMesh::tang with the places of the rests (n and cursor[2] start at 0)
cudaError_t launch_upwind_bits(const DevMesh& m, uint32_t* upw, unsigned long long* n, cudaStream_t s);
cudaError_t launch_list_tangential(const DevMesh& m, int2* list, unsigned long long* cursor, uint2* at, unsigned* seg,
                                   cudaStream_t s);
// partial moments of all chunks summed into chunk 0 (n doubles per chunk)
cudaError_t launch_sum_chunks(double* part, int chunks, size_t n, cudaStream_t s);
// cell records and Maxwellian tables rebuilt from the cell macros
cudaError_t launch_cell_records(const StepArgs& a, cudaStream_t s);
// entries first .. first + n - 1 of the caller's [dv][cell] array of g~ (or
// h~) at buf, from the state (get) or into it
cudaError_t launch_state_order(const StepArgs& a, int precision, bool second, bool get, const int32_t* iperm, double* buf,
                               size_t first, size_t n, cudaStream_t s);
// the next time step of an adaptive run from the Courant maximum (in ds.co)
// and dt_in, as src/setDeltaTvar.H:34-48 adjusts it; also stored to *hist
// when hist is not null
cudaError_t launch_adapt(const StepArgs& a, const double* dt_in, double* dt_out, double* hist, double max_co,
                         double max_dt, cudaStream_t s);

}  // namespace dugks
