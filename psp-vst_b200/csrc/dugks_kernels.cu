// DUGKS step for sm_100a: initialisation and bookkeeping kernels, and the
// stage sequence of one step.
//
// One fvDVM::evolution() (src/fvDVM/fvDVM/fvDVM.C:2128-2174) is
//   pass A  half step, face values, face moments and macros (dugks_passes.cu)
//   pass B  face fluxes, update, cell moments and macros
// The state g~, h~ is laid out [block of 32 cells][dv][32], the cells
// renumbered by recursive coordinate bisection.
#include <algorithm>

#include "dugks_device.cuh"

namespace dugks {

namespace {

// initial Maxwellian state (fvDVM.C:414-426)
template <typename Real>
__global__ void k_init_state(const StepArgs a) {
    const DevMesh& m = a.dm;
    const size_t n = static_cast<size_t>(m.nv_loc) * m.pC;
    const double K3D = m.K + 3.0 - m.D;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const unsigned row = static_cast<unsigned>(i / 32), blk = row / m.nv_loc;   // [block][dv][32]
        const int dl = static_cast<int>(row - blk * m.nv_loc), d = m.dv_base + dl;
        const int c = static_cast<int>(blk * 32 + i % 32);
        if (c >= m.nC) continue;
        const double* cm = a.ds.cm + static_cast<size_t>(c) * 9;
        const double RT = m.R * cm[4];
        const double cx = cm[1] - m.xi[3 * d], cy = cm[2] - m.xi[3 * d + 1], cz = cm[3] - m.xi[3 * d + 2];
        const double ge = cm[0] * inv_norm(RT, m.D) * exp(-0.5 * (cx * cx + cy * cy + cz * cz) / RT);
        const double he = K3D * ge * RT;
        if (sizeof(Real) == 4 && m.gref) {
            // FP32 storage of a tensor DV set: the deviation from the reference
            reinterpret_cast<Real*>(a.ds.g)[i] = Real(ge - m.gref[dl]);
            reinterpret_cast<Real*>(a.ds.h)[i] = Real(he - m.href[dl]);
        } else {
            reinterpret_cast<Real*>(a.ds.g)[i] = Real(ge);
            reinterpret_cast<Real*>(a.ds.h)[i] = Real(he);
        }
    }
}

// The caller's [dv][cell] order of doubles and the state's blocks of 32 cells,
// an FP32 state with its reference taken off or added.  The caller's side is
// contiguous, the state's in runs of a mesh row inside a bisection block.  The
// host did this entry by entry before (46 of the 54 ms of a 3,721-cell,
// 784-DV state set, stepped twice and read back).
template <typename Real, bool GET>
__global__ void k_state_order(const int nC, const int nv, const int32_t* __restrict__ iperm, Real* __restrict__ state,
                              const double* __restrict__ ref, double* __restrict__ buf, const size_t first, const size_t n,
                              int* err) {
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t d = (first + i) / nC;
        const int c = chk(iperm[first + i - d * nC], 0, nC, err);
        Real* s = state + (static_cast<size_t>(c / 32) * nv + d) * 32 + c % 32;
        const double r = sizeof(Real) == 4 && ref ? ref[d] : 0.0;
        if (GET) buf[i] = sizeof(Real) == 4 && ref ? double(*s) + r : double(*s);
        else *s = sizeof(Real) == 4 && ref ? Real(buf[i] - r) : Real(buf[i]);
    }
}

// wall: inComingByRho_f = sum_{xi.S<0} -w (xi.S) M/rho (fvDVM.C:598-617) and
// the raw moments of the incoming wall DFs per unit rho_w
// (xi.S <= 0, fvDVM.C:1079-1092)
__global__ void k_init_wall(const StepArgs a) {
    const DevMesh& m = a.dm;
    const int b = blockIdx.x;
    if (b >= m.nBF || m.bface_ptype[b] != DUGKS_PATCH_MAXWELL_WALL) return;
    BRec* br = a.ds.brec + b;
    const double S[3] = {m.bS[3 * b], m.bS[3 * b + 1], m.bS[3 * b + 2]};
    double acc[15];
    for (int j = 0; j < 15; ++j) acc[j] = 0.0;
    double inby = 0.0;
    const double K3D = m.K + 3.0 - m.D;
    const double RTw = 1.0 / br->invRT_in;
    for (int d = threadIdx.x; d < m.nv; d += blockDim.x) {
        const double xi[3] = {m.xi[3 * d], m.xi[3 * d + 1], m.xi[3 * d + 2]};
        const double xs = xi_dot_s(xi, S);
        if (xs > 0) continue;
        const double cx = br->U[0] - xi[0], cy = br->U[1] - xi[1], cz = br->U[2] - xi[2];
        const double mm = br->K_in * exp(-(cx * cx + cy * cy + cz * cz) / (2.0 * RTw));
        const double w = m.w[d];
        if (xs < 0) inby += -w * xs * mm;
        const double xi2 = xi[0] * xi[0] + xi[1] * xi[1] + xi[2] * xi[2];
        if (m.D == 3) accum<3>(acc, w, xi, xi2, mm, mm * RTw * K3D);
        else accum<2>(acc, w, xi, xi2, mm, mm * RTw * K3D);
    }
    // block reduction in a fixed order
    __shared__ double red[256][15];
    __shared__ double redi[256];
    for (int j = 0; j < 15; ++j) red[threadIdx.x][j] = acc[j];
    redi[threadIdx.x] = inby;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s[15] = {0};
        double si = 0;
        for (int t = 0; t < static_cast<int>(blockDim.x); ++t) {
            for (int j = 0; j < 15; ++j) s[j] += red[t][j];
            si += redi[t];
        }
        double* mi = a.ds.bmom_in + static_cast<size_t>(b) * kNM;
        for (int j = 0; j < 15; ++j) mi[j] = s[j];
        br->inByRho = si;
    }
}

// adjustable time step of src/setDeltaTvar.H:34-48 from the Courant number
// CoNum = max_f dc_f (|U_f| + sqrt(D) xiMax) dt (fvDVM::getCoNum) of the
// faces in co[0] (the maximum per unit dt, as double bits): F = maxCo /
// (CoNum + SMALL), f = min(min(F, 1 + 0.1 F), 1.2), dt_out = min(f dt, maxDeltaT);
// SMALL = 1e-15 (OpenFOAM's double SMALL).  Unfused operations, so that
// the host evaluation of the same formula gives the same bits.
__global__ void k_adapt(const double* co, const double* dt_in, double* dt_out, double* hist, double max_co,
                        double max_dt) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double per_dt = __longlong_as_double(*reinterpret_cast<const long long*>(co));
    const double dt = *dt_in;
    const double co_num = __dmul_rn(per_dt, dt);
    const double F = max_co / __dadd_rn(co_num, 1.0e-15);
    const double f = fmin(fmin(F, __dadd_rn(1.0, __dmul_rn(0.1, F))), 1.2);
    const double dtn = fmin(__dmul_rn(f, dt), max_dt);
    *dt_out = dtn;
    if (hist) *hist = dtn;
}

// pressureIn / pressureOut faces after the cell macros (updatePressureInOutBC,
// fvDVM.C:1745-1821): the next step's incoming far-field DFs take
//   pressureIn:  rho_b = p / R / T_b
//   pressureOut: rho_b = rho_i + (p - rho_i R T_i) / a_i / a_i, T_b = p / (R rho_i)
// from the owner cell i, a_i = sqrt(R T_i (K+5)/(K+3)); the patch velocity
// follows the characteristics (kept for output).
__global__ void k_pressure_bc(const StepArgs a) {
    const DevMesh& m = a.dm;
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= m.nBF) return;
    const int pt = __ldg(m.bface_ptype + b);
    if (pt != DUGKS_PATCH_PRESSURE_IN && pt != DUGKS_PATCH_PRESSURE_OUT) return;
    BRec* br = a.ds.brec + b;
    const double* cm = a.ds.cm + static_cast<size_t>(chk(__ldg(m.bface_owner + b), 0, m.nC, a.ds.err)) * 9;
    const double rhoi = cm[0], Ui[3] = {cm[1], cm[2], cm[3]}, Ti = cm[4];
    const double R = m.R, p = br->p;
    const double ai = sqrt(R * Ti * (m.K + 5) / (m.K + 3));
    const double S[3] = {__ldg(m.bS + 3 * b), __ldg(m.bS + 3 * b + 1), __ldg(m.bS + 3 * b + 2)};
    const double magS = sqrt(S[0] * S[0] + S[1] * S[1] + S[2] * S[2]);
    const double nv[3] = {S[0] / magS, S[1] / magS, S[2] / magS};
    const double Un = Ui[0] * nv[0] + Ui[1] * nv[1] + Ui[2] * nv[2];
    double UnIn;
    if (pt == DUGKS_PATCH_PRESSURE_IN) {
        br->rho_in = p / R / br->T;
        UnIn = Un + (p - rhoi * R * Ti) / rhoi / ai;
    } else {
        br->rho_in = rhoi + (p - rhoi * R * Ti) / ai / ai;
        br->T = p / (R * rhoi);
        const double RT = R * br->T;
        br->K_in = inv_norm(RT, m.D);
        br->invRT_in = 1.0 / RT;
        br->hfac = RT * (m.K + 3.0 - m.D);
        UnIn = Un + (rhoi * R * Ti - p) / rhoi / ai;
    }
    for (int k = 0; k < 3; ++k) br->U[k] = UnIn * nv[k] + (Ui[k] - Un * nv[k]);
}

// part[0][i] = sum over chunks of part[ch][i], in chunk order (the order the
// combine kernels sum them in), for the cross-shard reduction
__global__ void k_sum_chunks(double* part, int chunks, size_t n) {
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        double v = part[i];
        for (int ch = 1; ch < chunks; ++ch) v += part[static_cast<size_t>(ch) * n + i];
        part[i] = v;
    }
}

}  // namespace

cudaError_t launch_stage(const StepArgs& a, int precision, int stage, cudaStream_t s, int* launches) {
    int n = 0;
    cudaError_t e = cudaSuccess;
    auto pass = [&](int which, const StepArgs& b) {
        if (e == cudaSuccess) e = launch_pass(b, precision, which, s);
        ++n;
    };
    switch (stage) {
        case STAGE_PASS_A:
            for (int seg = 0; seg < a.dm.n_seg; seg += a.dm.seg_bar) {
                StepArgs b = a;
                b.seg0 = seg;
                b.seg1 = std::min(seg + a.dm.seg_bar, a.dm.n_seg);
                b.d_bar = seg_dv(a.dm, seg);
                pass(KERNEL_HALF_STEP, b);
                pass(KERNEL_FACE_VALUES, b);
                if (a.dm.n_tang > 0) pass(KERNEL_TANGENTIAL, b);
                if (a.dm.seg_bar < a.dm.n_seg) pass(KERNEL_ZERO_GRADIENT, b);
            }
            pass(KERNEL_FACE_MOMENTS, a);
            break;
        case STAGE_FACE_COMBINE:
            if (!a.fused) {
                e = launch_finish(a, true, s);
                ++n;
            }
            break;
        case STAGE_PASS_B:
            pass(KERNEL_FACE_FLUX, a);
            pass(KERNEL_UPDATE, a);
            break;
        case STAGE_CELL_COMBINE:
            if (!a.fused) {
                e = launch_finish(a, false, s);
                ++n;
            }
            if (e == cudaSuccess && a.dm.n_pressure_faces > 0) {
                k_pressure_bc<<<(a.dm.nBF + 255) / 256, 256, 0, s>>>(a);
                e = cudaGetLastError();
                ++n;
            }
            break;
        default:
            return cudaErrorInvalidValue;
    }
    if (launches) *launches += n;
    return e;
}

cudaError_t launch_sum_chunks(double* part, int chunks, size_t n, cudaStream_t s) {
    if (chunks <= 1 || n == 0) return cudaSuccess;
    const int tb = 256;
    const int nb = static_cast<int>(std::min<size_t>((n + tb - 1) / tb, 148 * 16));
    k_sum_chunks<<<nb, tb, 0, s>>>(part, chunks, n);
    return cudaGetLastError();
}

cudaError_t launch_adapt(const StepArgs& a, const double* dt_in, double* dt_out, double* hist, double max_co,
                         double max_dt, cudaStream_t s) {
    k_adapt<<<1, 32, 0, s>>>(a.ds.co, dt_in, dt_out, hist, max_co, max_dt);
    return cudaGetLastError();
}

cudaError_t launch_init(const StepArgs& a, int precision, cudaStream_t s) {
    if (precision == DUGKS_FP64) k_init_state<double><<<1184, 256, 0, s>>>(a);
    else k_init_state<float><<<1184, 256, 0, s>>>(a);
    if (cudaError_t e = launch_cell_records(a, s)) return e;
    if (a.dm.nBF > 0) k_init_wall<<<a.dm.nBF, 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_state_order(const StepArgs& a, int precision, bool second, bool get, const int32_t* iperm, double* buf,
                               size_t first, size_t n, cudaStream_t s) {
    const DevMesh& m = a.dm;
    void* st = second ? a.ds.h : a.ds.g;
    const double* ref = second ? m.href : m.gref;
    const unsigned nb = static_cast<unsigned>(std::min<size_t>((n + 255) / 256, 1u << 16));
    if (precision == DUGKS_FP64) {
        double* p = static_cast<double*>(st);
        if (get) k_state_order<double, true><<<nb, 256, 0, s>>>(m.nC, m.nv_loc, iperm, p, ref, buf, first, n, m.err);
        else k_state_order<double, false><<<nb, 256, 0, s>>>(m.nC, m.nv_loc, iperm, p, ref, buf, first, n, m.err);
    } else {
        float* p = static_cast<float*>(st);
        if (get) k_state_order<float, true><<<nb, 256, 0, s>>>(m.nC, m.nv_loc, iperm, p, ref, buf, first, n, m.err);
        else k_state_order<float, false><<<nb, 256, 0, s>>>(m.nC, m.nv_loc, iperm, p, ref, buf, first, n, m.err);
    }
    return cudaGetLastError();
}

}  // namespace dugks
