// k_stepwise.cuh -- the three substep kernels on the reference's own data
// layout, one launch each, FP64 throughout.
//
// These back the member-function API of GPU_Implementation5 (cuda_p2g,
// cuda_update_nodes, cuda_g2p; gpu_implementation5.cu:568-593) so that a
// caller that drives the substep kernel by kernel sees the reference's
// buffers: particle SoA of 16 pitched double rows, grid of 3 pitched double
// rows (mass, momentum x|velocity x, momentum y|velocity y), 100 angular
// force bins. SimParams is passed by value (it sits in the kernel-parameter
// constant bank, which is what __constant__ gprms was for).
//
// Kernel correspondence:
//   k_p2g_ref64     v2_kernel_p2g           gpu_implementation5.cu:148-213
//   k_update_ref64  v2_kernel_update_nodes  gpu_implementation5.cu:215-290
//   k_g2p_ref64     v2_kernel_g2p           gpu_implementation5.cu:294-379
// Out-of-grid stencil nodes raise the error word and are skipped (the
// reference raises gpu_error_indicator but still adds at the bad index).
#pragma once
#include "mpm_math64.cuh"

namespace icm {

__device__ __forceinline__ double *pts_row(const icy_SimParams &P, int r) { return P.pts_array + (size_t)r * P.nPtsPitch; }

// A launch may be a programmatic dependent of the kernel before it: what
// that kernel writes is read only after this, and the next kernel may start.
__device__ __forceinline__ void after_previous_kernel()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Bound by the FP64 atomics at L2 when every particle adds to its nine nodes
// itself (27 M atomics for 999,424 particles: 64 us). The SoA is sorted by
// cell when it is loaded and keeps its order, so neighbouring lanes mostly
// share a cell and so all nine nodes: runs of lanes with one cell are added
// up with shuffles, four lanes at a time, and the first lane of each four
// issues the atomics: 41 us, issue-bound (73 % of cycles). Leaving the terms
// in shared memory and dealing the run's nodes out to its lanes took 51 us.
__global__ void k_p2g_ref64(const __grid_constant__ icy_SimParams P, int *err)
{
    after_previous_kernel();
    const int pt = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, lanes = min(32, (int)(blockDim.x - (threadIdx.x & ~31u)));
    const unsigned mask = lanes == 32 ? 0xffffffffu : (1u << lanes) - 1u;
    const bool on = pt < P.nPts;
    if (!__any_sync(mask, on)) return;
    const int q = on ? pt : P.nPts - 1;  // the lanes past the end compute the last particle and add nothing
    const double h = P.cellsize, m = P.ParticleMass;
    double x = pts_row(P, ICM_IDX_POSX)[q], y = pts_row(P, ICM_IDX_POSX + 1)[q];
    double v0 = pts_row(P, ICM_IDX_VELX)[q], v1 = pts_row(P, ICM_IDX_VELX + 1)[q];
    M2d F = {pts_row(P, ICM_IDX_FE00)[q], pts_row(P, ICM_IDX_FE00 + 1)[q], pts_row(P, ICM_IDX_FE00 + 2)[q],
             pts_row(P, ICM_IDX_FE00 + 3)[q]};
    M2d B = {pts_row(P, ICM_IDX_BP00)[q], pts_row(P, ICM_IDX_BP00 + 1)[q], pts_row(P, ICM_IDX_BP00 + 2)[q],
             pts_row(P, ICM_IDX_BP00 + 3)[q]};
    M2d tau = kirchhoff64(F, P.mu, P.kappa);
    const double c = (P.InitialTimeStep * P.ParticleVolume) * P.Dp_inv;
    const double s00 = h * (m * B.a00 - c * tau.a00), s01 = h * (m * B.a01 - c * tau.a01);
    const double s10 = h * (m * B.a10 - c * tau.a10), s11 = h * (m * B.a11 - c * tau.a11);
    const Stencil64 st = stencil64(x, y, P.cellsize_inv);
    // the lane's place in its run of lanes with one cell
    const int pbx = __shfl_up_sync(mask, st.bx, 1), pby = __shfl_up_sync(mask, st.by, 1);
    const unsigned heads = __ballot_sync(mask, lane == 0 || !on || st.bx != pbx || st.by != pby);
    const int pos = lane - (31 - __clz((int)(heads & (0xffffffffu >> (31 - lane)))));
    const unsigned later = lane == 31 ? 0u : heads >> (lane + 1) << (lane + 1);
    const int end = later ? __ffs((int)later) - 1 : lanes;
    const bool add1 = (pos & 1) == 0 && lane + 1 < end, add2 = (pos & 3) == 0 && lane + 2 < end;
    const bool first = on && (pos & 3) == 0;
    // (volatile: without it the compiler makes an addition and two selects of
    // each; a predicate per addition was slower, 85.5 against 83.9 us a substep)
    auto run_sum = [&](double v) {
        const double a = __shfl_down_sync(mask, v, 1);
        if (add1) asm volatile("add.f64 %0, %0, %1;" : "+d"(v) : "d"(a));
        const double b = __shfl_down_sync(mask, v, 2);
        if (add2) asm volatile("add.f64 %0, %0, %1;" : "+d"(v) : "d"(b));
        return v;
    };
    const bool inside = st.bx >= 0 && st.by >= 0 && st.bx + 2 < P.GridX && st.by + 2 < P.GridY;
    const size_t gp = P.nGridPitch;
    double *g = P.grid_array + ((ptrdiff_t)st.by * P.GridX + st.bx);  // (used inside the grid only)
    // node (i, j) gets W_ij (m, m v + S dpos_ij) = W_ij (m, c + S_h (i, j)^T)
    double u0 = v0 * m - (s00 * st.fx + s01 * st.fy), u1 = v1 * m - (s10 * st.fx + s11 * st.fy);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        double a0 = u0, a1 = u1;
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const double W = st.wx[i] * st.wy[j];
            const double sm = run_sum(W * m), s0 = run_sum(W * a0), s1 = run_sum(W * a1);
            const bool in = inside || (i + st.bx >= 0 && j + st.by >= 0 && i + st.bx < P.GridX && j + st.by < P.GridY);
            if (first && in) {
                double *n = g + (ptrdiff_t)j * P.GridX + i;
                atomicAdd(n, sm);
                atomicAdd(n + gp, s0);
                atomicAdd(n + 2 * gp, s1);
            }
            a0 += s01;
            a1 += s11;
        }
        u0 += s00;
        u1 += s10;
    }
    if (on && !inside) *err = 1;
}

// update_node64 out of line, for the nodes inside the indenter's circle and
// those fast enough to be clamped.
static __device__ __noinline__ NodeOut update_node64_call(const icy_SimParams &P, int ix, int iy, double mass, double p0,
                                                          double p1, double ind_x, double ind_y)
{
    return update_node64(P, ix, iy, mass, p0, p1, ind_x, ind_y);
}

// force_total (may be null): 2 doubles receiving this launch's summed
// reaction. next (may be null): the grid that the next P2G adds to, whose
// nodes are zeroed where the substep before left mass (a quarter of the
// nodes, instead of a clear of the whole grid per substep); nothing else
// uses it meanwhile. Latency-bound: the common node (outside the indenter,
// below the speed limit) is done in line, the others by a call.
__global__ void k_update_ref64(const __grid_constant__ icy_SimParams P, double ind_x, double ind_y,
                               double *force_total, double *next)
{
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    const size_t gp = P.nGridPitch;
    const bool on = idx < P.GridTotal;
    if (next && on && next[idx] != 0.0) {
        next[idx] = 0.0;
        next[gp + idx] = 0.0;
        next[2 * gp + idx] = 0.0;
    }
    after_previous_kernel();
    const double mass = on ? P.grid_array[idx] : 0.0;
    if (mass == 0) return;
    const double p0 = P.grid_array[gp + idx], p1 = P.grid_array[2 * gp + idx];
    const int ix = idx % P.GridX, iy = idx / P.GridX;
    const double dt = P.InitialTimeStep, vmax = 0.5 * P.cellsize / dt;
    double v0 = p0 / mass, v1 = p1 / mass;
    v1 -= dt * P.Gravity;
    const double n0 = ix * P.cellsize - ind_x, n1 = iy * P.cellsize - ind_y;
    if (n0 * n0 + n1 * n1 < P.IndRSq || !(v0 * v0 + v1 * v1 < 0.999 * vmax * vmax)) {
        const NodeOut o = update_node64_call(P, ix, iy, mass, p0, p1, ind_x, ind_y);
        if (o.bin >= 0) {
            atomicAdd(&P.indenter_force_accumulator[2 * o.bin], o.f0);
            atomicAdd(&P.indenter_force_accumulator[2 * o.bin + 1], o.f1);
            if (force_total) {
                atomicAdd(&force_total[0], o.f0);
                atomicAdd(&force_total[1], o.f1);
            }
        }
        v0 = o.v0;
        v1 = o.v1;
    } else {  // update_node64 without contact and clamp
        if (iy <= 2) {
            v0 = 0;
            v1 = 0;
        } else if (iy >= P.GridY - 3 && v1 > 0) {
            v1 = 0;
        }
        if (ix <= 2 && v0 < 0)
            v0 = 0;
        else if (ix >= P.GridX - 3 && v0 > 0)
            v0 = 0;
    }
    P.grid_array[gp + idx] = v0;
    P.grid_array[2 * gp + idx] = v1;
}

__global__ void k_g2p_ref64(const __grid_constant__ icy_SimParams P, int recordPQ)
{
    int pt = blockIdx.x * blockDim.x + threadIdx.x;
    if (pt >= P.nPts) return;  // (a CTA's exit counts as its permission for the next kernel to start)
    const size_t gp = P.nGridPitch;
    const double h_inv = P.cellsize_inv, dt = P.InitialTimeStep;
    double x = pts_row(P, ICM_IDX_POSX)[pt], y = pts_row(P, ICM_IDX_POSX + 1)[pt];
    M2d F = {pts_row(P, ICM_IDX_FE00)[pt], pts_row(P, ICM_IDX_FE00 + 1)[pt], pts_row(P, ICM_IDX_FE00 + 2)[pt],
             pts_row(P, ICM_IDX_FE00 + 3)[pt]};
    uint8_t *crushed_row = (uint8_t *)P.pts_array;
    const short *grain_row = (const short *)((const char *)P.pts_array + P.nPtsPitch);
    uint8_t crushed = crushed_row[pt];
    int grain = grain_row[pt];
    double Jp = pts_row(P, ICM_IDX_JP_INV)[pt];

    Stencil64 st = stencil64(x, y, h_inv);
    // the particle's own state was complete before the grid update could
    // start; the grid is read after it
    after_previous_kernel();
    double v0 = 0, v1 = 0, B00 = 0, B01 = 0, B10 = 0, B11 = 0;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            double d0 = i - st.fx, d1 = j - st.fy;
            double W = st.wx[i] * st.wy[j];
            int i2 = i + st.bx, j2 = j + st.by;
            double n0 = 0, n1 = 0;
            if (i2 >= 0 && j2 >= 0 && i2 < P.GridX && j2 < P.GridY) {
                size_t idx = (size_t)i2 + (size_t)j2 * P.GridX;
                n0 = P.grid_array[gp + idx];
                n1 = P.grid_array[2 * gp + idx];
            }
            v0 += W * n0;
            v1 += W * n1;
            double c = (4. * h_inv) * W;
            B00 += c * (n0 * d0);
            B01 += c * (n0 * d1);
            B10 += c * (n1 * d0);
            B11 += c * (n1 * d1);
        }
    x += v0 * dt;
    y += v1 * dt;
    double M00 = 1 + dt * B00, M01 = dt * B01, M10 = dt * B10, M11 = 1 + dt * B11;
    M2d Fn = {M00 * F.a00 + M01 * F.a10, M00 * F.a01 + M01 * F.a11, M10 * F.a00 + M11 * F.a10,
              M10 * F.a01 + M11 * F.a11};
    double p_tr, q_tr;
    // (an intact particle inside its failure surface needs no SVD: 50 us with
    // it, 38 without, 999,424 particles)
    constitutive64_intact_first(P, Fn, Jp, crushed, grain_res(grain), p_tr, q_tr);

    pts_row(P, ICM_IDX_JP_INV)[pt] = Jp;
    pts_row(P, ICM_IDX_POSX)[pt] = x;
    pts_row(P, ICM_IDX_POSX + 1)[pt] = y;
    pts_row(P, ICM_IDX_VELX)[pt] = v0;
    pts_row(P, ICM_IDX_VELX + 1)[pt] = v1;
    pts_row(P, ICM_IDX_FE00)[pt] = Fn.a00;
    pts_row(P, ICM_IDX_FE00 + 1)[pt] = Fn.a01;
    pts_row(P, ICM_IDX_FE00 + 2)[pt] = Fn.a10;
    pts_row(P, ICM_IDX_FE00 + 3)[pt] = Fn.a11;
    pts_row(P, ICM_IDX_BP00)[pt] = B00;
    pts_row(P, ICM_IDX_BP00 + 1)[pt] = B01;
    pts_row(P, ICM_IDX_BP00 + 2)[pt] = B10;
    pts_row(P, ICM_IDX_BP00 + 3)[pt] = B11;
    crushed_row[pt] = crushed;
    if (recordPQ) {
        pts_row(P, ICM_IDX_P)[pt] = p_tr;
        pts_row(P, ICM_IDX_Q)[pt] = q_tr;
    }
}

}  // namespace icm
