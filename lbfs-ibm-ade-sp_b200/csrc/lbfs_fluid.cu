// Fluid kernels of one LBFS time step; see lbfs_fluid.cuh for the mapping to
// the reference kernels they replace.
#include <cuda_runtime.h>

#include <algorithm>

#include "lbfs_face.cuh"
#include "lbfs_fluid.cuh"
#include "lbfs_internal.h"
#include "lbfs_kernels.h"

namespace lbfs {


// ------------------------------------------------------------------ K1 ----

// REST: the cells beside those of the fused step (kSeparateCell); they also keep their state in prev.
template <typename R, int TB, bool REST>
__global__ void __launch_bounds__(TB, TB == 128 ? 5 : 1) k_cell_gradients(FluidArgs<R> a, int begin, int end, Vec4<R> *prev) {
    pdl_trigger();  // the interior-face kernel may be scheduled behind the last wave
    const int i = begin + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end || (REST && !(a.grid_sides[i] & kSeparateCell))) return;
    const Vec4<R> own = a.state[i];
    if constexpr (REST) prev[i] = own;
    GradRec<R> gr;
    cell_gradient(a, i, own, gr.g);
    reinterpret_cast<GradRec<R> *>(a.grad)[i] = gr;
}

// ------------------------------------------------------------------ K2 ----


// Interior faces of an axis-aligned mesh: faces [0, nfx) x, [nfx, nfx+nfy) y,
// the rest z; warps never mix axes except at the two range boundaries.
// TB threads per block, 640 / TB blocks per SM (at most 102 registers a thread).
// REST: the faces of the cells beside those of the fused step.
template <typename R, int TB, bool REST>
__global__ void __launch_bounds__(TB, 640 / TB) k_face_flux(FluidArgs<R> a, FaceRanges r) {
    int t = blockIdx.x * blockDim.x + threadIdx.x, f;
    if (t < r.count[0]) f = r.start[0] + t;
    else if ((t -= r.count[0]) < r.count[1]) f = r.start[1] + t;
    else if ((t -= r.count[1]) < r.count[2]) f = r.start[2] + t;
    else return;
    if (REST && !(a.grid_sides[__ldg(a.face_cells + f).x] & kSeparateCell)) return;
    Vec4<R> out;
    if (f < a.nfx) out = axis_face_flux<R, 0>(a, f);
    else if (f < a.nfx + a.nfy) out = axis_face_flux<R, 1>(a, f);
    else out = axis_face_flux<R, 2>(a, f);
    a.flux[f] = out;
}

// Interior faces of an axis-aligned mesh, tile by tile: block b takes the
// faces owned by the TB cells of tile tile0 + b -- the x, y and z faces whose
// owner lies in the tile, three contiguous ranges of the face list
// (tiles[3 t + axis] = first face of that axis owned by tile t) -- so the
// tile's cell states and gradients come from DRAM once for all three axes
// instead of once per axis sweep.  Warps take the x faces, then the y, then
// the z faces: one axis per warp at a time.  Load-latency bound: FP64 fits 96
// registers (20 warps per SM; at 80 it spills), FP32 64 (32 warps per SM).
template <typename R, int TB>
__global__ void __launch_bounds__(TB, (sizeof(R) == 4 ? 1024 : 640) / TB) k_face_flux_tiles(FluidArgs<R> a, int tile0) {
    pdl_trigger();
    const int *tp = a.flux_tiles + 3 * (tile0 + (int)blockIdx.x);
    const int f0x = __ldg(tp), f0y = __ldg(tp + 1), f0z = __ldg(tp + 2);
    const int f1x = __ldg(tp + 3), f1y = __ldg(tp + 4), f1z = __ldg(tp + 5);
    pdl_wait();  // the gradients
    for (int f = f0x + (int)threadIdx.x; f < f1x; f += TB) a.flux[f] = axis_face_flux<R, 0>(a, f);
    for (int f = f0y + (int)threadIdx.x; f < f1y; f += TB) a.flux[f] = axis_face_flux<R, 1>(a, f);
    for (int f = f0z + (int)threadIdx.x; f < f1z; f += TB) a.flux[f] = axis_face_flux<R, 2>(a, f);
}

// Interior faces of a mesh that is not axis aligned (every face takes the
// general-normal reconstruction), tile by tile as k_face_flux_tiles: block b
// takes the faces owned by the TB cells of tile tile0 + b, in up to three
// face ranges ordered by owner (the generator's x, y, z faces; an imported
// mesh's internal faces, which OpenFOAM orders by owner, form one range).
// FP64 at 128 registers (16 warps per SM), FP32 at 64 (32 warps per SM).  CONE: the
// faces of the three ranges lie within the cones of x, y and z (FluidArgs::cone), a
// property of the whole mesh: which form a face takes depends on no other face of its
// warp, so results do not depend on the block size.  An imported mesh's one range
// mixes the axes (its faces taken axis by axis through an index list: 48.5 us a step on
// 64,000 cells, 44.4 without).
template <typename R, int TB, bool CONE>
__global__ void __launch_bounds__(TB, (sizeof(R) == 4 ? 1024 : 512) / TB) k_face_flux_general_tiles(FluidArgs<R> a, int tile0) {
    pdl_trigger();
    pdl_wait();  // the gradients
    const int *tp = a.flux_tiles + 3 * (tile0 + (int)blockIdx.x);
    if constexpr (CONE) {
        const int t = (int)threadIdx.x;
        for (int f = __ldg(tp) + t, f1 = __ldg(tp + 3); f < f1; f += TB) a.flux[f] = general_face_flux<R, 0>(a, f, false);
        for (int f = __ldg(tp + 1) + t, f1 = __ldg(tp + 4); f < f1; f += TB) a.flux[f] = general_face_flux<R, 1>(a, f, false);
        for (int f = __ldg(tp + 2) + t, f1 = __ldg(tp + 5); f < f1; f += TB) a.flux[f] = general_face_flux<R, 2>(a, f, false);
    } else {
#pragma unroll 1
        for (int r = 0; r < 3; r++) {
            const int f0 = __ldg(tp + r), f1 = __ldg(tp + 3 + r);
            for (int f = f0 + (int)threadIdx.x; f < f1; f += TB) a.flux[f] = general_face_flux<R, -1>(a, f, false);
        }
    }
}

// Boundary faces (always) and the interior faces of meshes that are not axis
// aligned: the general-normal reconstruction.  `first` is ni (axis-aligned
// meshes) or 0.  REST: those of the cells beside the fused step's.
template <typename R, int TB, bool REST>
__global__ void __launch_bounds__(TB) k_face_flux_general(FluidArgs<R> a, int first) {
    const int f = first + blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= a.nf || (REST && !(a.grid_sides[__ldg(a.face_cells + f).x] & kSeparateCell))) return;
    a.flux[f] = general_face_flux<R, -1>(a, f, f >= a.ni);
}

// ----------------------------------------------------------------- CFL ----
// get_cfl_device (LBFS.cu:2868-2932) per cell, then the minimum over the cells
// (min<128> + min_block, common_kernels.hpp:147-170, Solver_gpu.cu:57-66):
// block minima, the last block takes the minimum of the block minima.  A
// minimum is exact, so the result does not depend on the grid.  The effective
// speed of sound (a constant of the step) is formed on the host.  Products and
// sums use explicitly rounded intrinsics so no multiply-add is contracted,
// as in the reference's evaluation.
template <typename R>
__global__ void __launch_bounds__(256) k_cfl(FluidArgs<R> a) {
    __shared__ double sh[8];
    __shared__ bool last_block;
    double mn = 100000000.0;  // min<128> pads its blocks with 1e8
    const double ce = __dadd_rn(a.cfl_max_velocity, a.cfl_esos);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.nc; i += gridDim.x * blockDim.x) {
        const double4 c = a.cfl[i];  // area x, y, z, volume
        const double rho = (double)a.state[i].rho + (double)a.rho0;
        double eig = __dadd_rn(__dadd_rn(__dmul_rn(ce, c.x), __dmul_rn(ce, c.y)), __dmul_rn(ce, c.z));
        eig = eig / a.cfl_gamma;
        double ve = 2.0 * a.cfl_visc / a.cfl_gamma / rho / c.w;
        ve = __dmul_rn(ve, __dadd_rn(__dadd_rn(__dmul_rn(c.x, c.x), __dmul_rn(c.y, c.y)), __dmul_rn(c.z, c.z)));
        eig = __dadd_rn(eig, __dmul_rn(4.0, ve));
        const double dt = __dmul_rn(a.cfl_factor, c.w) / eig;
        a.dt_local[i] = dt;
        mn = fmin(mn, dt);
    }
    for (int o = 16; o > 0; o >>= 1) mn = fmin(mn, __shfl_down_sync(0xffffffffu, mn, o));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh[warp] = mn;
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = sh[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) b = fmin(b, sh[w]);
        a.dt_partials[blockIdx.x] = b;
        __threadfence();
        last_block = atomicAdd(a.dt_ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last_block && threadIdx.x == 0) {
        __threadfence();
        double b = 100000000.0;
        for (int k = 0; k < (int)gridDim.x; k++) b = fmin(b, __ldcg(a.dt_partials + k));
        *a.dt_min = b;
        *a.dt_ticket = 0u;
    }
}

// ------------------------------------------------------------------ K3 ----

// The convergence test of the reference's loop (Solver_gpu.cu:1206-1208:
// convergence_residual.max_error() < tolerance) on the step's residual norms,
// formed as lbfs_get_residuals forms them, and the drop-in's divergence test
// (non-finite state or density out of range); sets the while node's condition.
// Lanes 0 to 3 of one warp bring the sums.  In the update's last block: a kernel of
// its own behind it cost 0.8 to 1.2 us a step of the loop (32^3 18.6 / 17.8 us,
// 45x37x29 with a membrane 31.5 / 30.3).
template <typename R> __device__ __forceinline__ void until_check(const FluidArgs<R> &a, double sum, int lane) {
    UntilState *u = a.until.u;
    const double r = sqrt(sum / (double)a.nc) / (lane == 0 ? a.until.ref_rho : a.until.ref_mom);
    if (lane < 4) u->res[lane] = r;
    const double r0 = __shfl_sync(0xffffffffu, r, 0), r1 = __shfl_sync(0xffffffffu, r, 1);
    const double r2 = __shfl_sync(0xffffffffu, r, 2), r3 = __shfl_sync(0xffffffffu, r, 3);
    if (lane != 0) return;
    const double m01 = r0 < r1 ? r1 : r0, m23 = r2 < r3 ? r3 : r2;  // std::max
    const double mx = m01 < m23 ? m23 : m01;
    const bool converged = mx < u->tol;
    const bool diverged = (__ldcg(a.flags) & (LBFS_FLAG_NONFINITE | LBFS_FLAG_RHO_RANGE)) != 0u;
    const int c = u->count + 1;
    u->count = c;
    u->stop = converged ? 1 : (diverged ? 2 : 0);
    cudaGraphSetConditional(a.until.handle, (!converged && !diverged && c < u->limit) ? 1u : 0u);
}

// FUSED: behind the fused step, whose cell sums over the interior faces it
// reads (32 B instead of six fluxes of 32 / 16 B).  It subtracts the upper faces
// that other tiles formed, z, x, y, scales the sum and adds the boundary faces.
// MIXED: grids of several spacings, or cells that keep the separate kernels.
enum Sums { GATHER, FUSED, MIXED };
template <typename R, int TB, int SUMS>
__global__ void __launch_bounds__(TB) k_cell_update(FluidArgs<R> a) {
    __shared__ double sh[4][TB / 32];
    __shared__ bool last_block;
    // one instance with few membranes: its grid and the membranes' patches cached per block,
    // with each patch's first and last linear cell (cells outside skip the i, j, k split)
    __shared__ int s_grid[6];                 // cell0, nx, ny, nz, mem0, mem1
    __shared__ int s_patch[kK3PatchCache][10];  // lo[3], dim[3], cells, off, first, last linear cell
    pdl_wait();  // the face fluxes
    const bool cached = a.n_membranes > 0 && a.n_membranes <= kK3PatchCache && !a.cell_instance;
    if (cached) {
        const InstanceGrid g0 = reinterpret_cast<const InstanceGrid *>(a.instances)[0];
        if (threadIdx.x == 0) {
            s_grid[0] = g0.cell0; s_grid[1] = g0.nx; s_grid[2] = g0.ny; s_grid[3] = g0.nz;
            s_grid[4] = g0.mem0; s_grid[5] = g0.mem1;
        }
        const MembraneScalars *ms = (const MembraneScalars *)a.membrane_scalars;
        if ((int)threadIdx.x < a.n_membranes) {
            const MembraneScalars &q = ms[threadIdx.x];
            int *e = s_patch[threadIdx.x];
            for (int c = 0; c < 3; c++) { e[c] = q.patch_lo[c]; e[3 + c] = q.patch_dim[c]; }
            e[6] = q.patch_cells;
            e[7] = q.patch_off;
            e[8] = q.patch_lo[0] + g0.nx * (q.patch_lo[1] + g0.ny * q.patch_lo[2]);
            e[9] = (q.patch_lo[0] + q.patch_dim[0] - 1) +
                   g0.nx * ((q.patch_lo[1] + q.patch_dim[1] - 1) + g0.ny * (q.patch_lo[2] + q.patch_dim[2] - 1));
        }
        __syncthreads();
    }
    double sq[4] = {0, 0, 0, 0};
    unsigned int flag = 0;
    // the step: constant, or the minimum per-cell step, or each cell's own (LBFS_DT_LOCAL)
    const bool local_dt = a.time_stepping == LBFS_DT_LOCAL;
    const double dt_all = (a.time_stepping == LBFS_DT_MIN || a.time_stepping == LBFS_DT_TALTS) ? __ldcg(a.dt_min)
                                                                                                 : a.delta_t;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.nc; i += gridDim.x * blockDim.x) {
        // 1 / volume: products instead of 24 divisions
        const double iv = a.inv_volume_uniform ? a.inv_volume_all : __ldg(a.cell_inv_volume + i);
        double4 t = a.t1[i];  // in flight beside the sums (1 to 2 % of the step when loaded where it is used)
        double r[4] = {0, 0, 0, 0};  // rho, u, v, w
        const unsigned sides = SUMS != GATHER ? a.grid_sides[i] : (unsigned)kSeparateCell;
        if (SUMS == FUSED || (SUMS == MIXED && !(sides & kSeparateCell))) {
            const double4 q = a.grid_res[i];
            r[0] = q.x; r[1] = q.y; r[2] = q.z; r[3] = q.w;
            int sy = a.grid_stride[0], sz = a.grid_stride[1];
            double area = a.grid_area;
            if (SUMS == MIXED || ((sides & 14u) && sy == 0)) {
                const GridCells g = a.grid_cells[__ldg(a.grid_instance + i)];
                sy = g.sy;
                sz = g.sz;
                area = g.area;
            }
            if (sides & 14u) {  // upper faces that another tile formed: z first, as a walk subtracts it
#pragma unroll
                for (int e = 0; e < 3; e++) {
                    const int d = (e + 2) % 3;
                    if (!(sides >> (d + 1) & 1u)) continue;
                    const Vec4<R> fx = a.grid_edge[(size_t)d * a.nc + i + (d == 0 ? 1 : (d == 1 ? sy : sz))];
                    const double fv[4] = {(double)fx.rho, (double)fx.u, (double)fx.v, (double)fx.w};
#pragma unroll
                    for (int m = 0; m < 4; m++) r[m] = r[m] - fv[m];
                }
            }
            const double ia = iv * (SUMS == MIXED ? area : a.grid_area);
#pragma unroll
            for (int m = 0; m < 4; m++) r[m] = __dmul_rn(r[m], ia);  // not contracted with what follows, whatever that is
            if (sides & 1u) {
                for (int e = 0; e < 6; e++) {
                    const int f = __ldg(a.cell_faces + 6 * (size_t)i + e) - 1;
                    if (f < a.ni) continue;
                    const Vec4<R> fx = a.flux[f];
                    const double fv[4] = {(double)fx.rho, (double)fx.u, (double)fx.v, (double)fx.w};
#pragma unroll
                    for (int m = 0; m < 4; m++) r[m] = r[m] + (-fv[m] * iv);
                }
            }
        } else {
            int cfl[6];
            if (a.grid_faces) {  // the structured mesh's faces, formed (no dependent load before the fluxes)
                grid_cell_faces(i, a.grid_n[0], a.grid_n[1], a.grid_n[2], cfl);
            } else {
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    const int2 p = __ldg(reinterpret_cast<const int2 *>(a.cell_faces) + 3 * i + q);
                    cfl[2 * q] = p.x;
                    cfl[2 * q + 1] = p.y;
                }
            }
#pragma unroll
            for (int q = 0; q < 6; q++) {
                const int e = cfl[q];
                const int f = (e > 0 ? e : -e) - 1;
                const Vec4<R> fx = a.flux[f];
                const double fv[4] = {(double)fx.rho, (double)fx.u, (double)fx.v, (double)fx.w};
#pragma unroll
                for (int m = 0; m < 4; m++) r[m] = (e > 0) ? r[m] + (-fv[m] * iv) : r[m] + fv[m] * iv;
            }
        }
        if (a.closure) {
#pragma unroll
            for (int m = 0; m < 3; m++) r[1 + m] = r[1 + m] + __ldg(a.closure + 3 * (size_t)i + m);
        }
        double fx = a.force[0], fy = a.force[1], fz = a.force[2];
        if (cached) {
            const int li = i - s_grid[0];
            for (int m = s_grid[4]; m < s_grid[5]; m++) {
                const int *e = s_patch[m];
                if (e[6] <= 0 || li < e[8] || li > e[9]) continue;
                const int nx = s_grid[1], ny = s_grid[2];
                const int ci = li % nx, cj = (li / nx) % ny, ck = li / (nx * ny);
                const int px = ci - e[0], py = cj - e[1], pz = ck - e[2];
                if (px >= 0 && py >= 0 && pz >= 0 && px < e[3] && py < e[4] && pz < e[5]) {
                    const double *pf = a.patch_force + ((size_t)e[7] + (px + e[3] * (py + e[4] * pz))) * 3;
                    fx = fx + pf[0];
                    fy = fy + pf[1];
                    fz = fz + pf[2];
                }
            }
        } else if (a.n_membranes > 0) {
            const int inst = a.cell_instance ? __ldg(a.cell_instance + i) : 0;
            const InstanceGrid g = reinterpret_cast<const InstanceGrid *>(a.instances)[inst];
            const int li = i - g.cell0;
            const int ci = li % g.nx, cj = (li / g.nx) % g.ny, ck = li / (g.nx * g.ny);
            const MembraneScalars *ms = (const MembraneScalars *)a.membrane_scalars;
            for (int m = g.mem0; m < g.mem1; m++) {
                const int px = ci - ms[m].patch_lo[0], py = cj - ms[m].patch_lo[1], pz = ck - ms[m].patch_lo[2];
                if (ms[m].patch_cells > 0 && px >= 0 && py >= 0 && pz >= 0 && px < ms[m].patch_dim[0] &&
                    py < ms[m].patch_dim[1] && pz < ms[m].patch_dim[2]) {
                    const double *pf = a.patch_force + ((size_t)ms[m].patch_off +
                                                        (px + ms[m].patch_dim[0] * (py + ms[m].patch_dim[1] * pz))) * 3;
                    fx = fx + pf[0];
                    fy = fy + pf[1];
                    fz = fz + pf[2];
                }
            }
        }
        r[1] = r[1] + fx;
        r[2] = r[2] + fy;
        r[3] = r[3] + fz;
        const double dt = local_dt ? a.dt_local[i] : dt_all;
        t.w = t.w + dt * r[0];
        t.x = t.x + dt * r[1];
        t.y = t.y + dt * r[2];
        t.z = t.z + dt * r[3];
        a.t1[i] = t;
        Vec4<R> s;
        s.rho = (R)(t.w - (double)a.rho0);
        s.u = (R)(t.x / t.w);
        s.v = (R)(t.y / t.w);
        s.w = (R)(t.z / t.w);
        a.state[i] = s;
        if (a.res_out) {
            a.res_out[4 * i] = r[0]; a.res_out[4 * i + 1] = r[1];
            a.res_out[4 * i + 2] = r[2]; a.res_out[4 * i + 3] = r[3];
        }
#pragma unroll
        for (int m = 0; m < 4; m++) sq[m] = sq[m] + r[m] * r[m];
        if (!(isfinite(t.w) && isfinite(t.x) && isfinite(t.y) && isfinite(t.z))) flag |= LBFS_FLAG_NONFINITE;
        else if (!(t.w > 0.0) || t.w > 1000.0) flag |= LBFS_FLAG_RHO_RANGE;
    }
    if (flag) atomicOr(a.flags, flag);
    // Block partial sums of the squared residuals (fixed order: warp tree, then warps in order).
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int m = 0; m < 4; m++) {
        double v = sq[m];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) sh[m][warp] = v;
    }
    __syncthreads();
    if (warp == 0) {
        if (lane < 4) {
            double v = 0;
#pragma unroll
            for (int w = 0; w < TB / 32; w++) v += sh[lane][w];
            a.partials[4 * blockIdx.x + lane] = v;
        }
        __syncwarp();
        if (lane == 0) {  // the fence behind the barrier: it orders all four lanes' sums (and the flags) before the ticket
            __threadfence();
            last_block = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
        }
    }
    __syncthreads();
    if (last_block) {
        // Final sum of the block partials by the whole last block: thread t
        // adds partials t, t + blockDim, ... (fixed assignment), then the same
        // warp/block tree as above.  Deterministic for a fixed grid.
        __threadfence();
        double acc[4] = {0, 0, 0, 0};
        for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x)
#pragma unroll
            for (int m = 0; m < 4; m++) acc[m] += __ldcg(a.partials + 4 * b + m);
#pragma unroll
        for (int m = 0; m < 4; m++) {
            double v = acc[m];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) sh[m][warp] = v;
        }
        __syncthreads();
        if (warp == 0) {
            double v = 0;
            if (lane < 4) {
                for (int w = 0; w < (int)(blockDim.x >> 5); w++) v += sh[lane][w];
                a.residual_sums[lane] = v;
            }
            if (lane == 0) *a.ticket = 0u;
            if (a.until.u) until_check(a, v, lane);
        }
    }
}

// ------------------------------------------------------- state transfer ----

template <typename R>
__global__ void k_pack_state(FluidArgs<R> a, const double *__restrict__ stage) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.nc) return;
    const size_t n = (size_t)a.nc;
    const double rho = stage[i], u = stage[n + i], v = stage[2 * n + i], w = stage[3 * n + i];
    Vec4<R> s;
    s.u = (R)u; s.v = (R)v; s.w = (R)w; s.rho = (R)(rho - (double)a.rho0);
    a.state[i] = s;
    a.t1[i] = make_double4(u, v, w, rho);
}

template <typename R>
__global__ void k_unpack_state(FluidArgs<R> a, double *__restrict__ stage) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.nc) return;
    const size_t n = (size_t)a.nc;
    const Vec4<R> s = a.state[i];
    stage[i] = (double)s.rho + (double)a.rho0;
    stage[n + i] = (double)s.u;
    stage[2 * n + i] = (double)s.v;
    stage[3 * n + i] = (double)s.w;
}

// ------------------------------------------------------------ launchers ----

template <typename R> int k3_grid(const FluidArgs<R> &a) {
    const int g = (a.nc + a.tb_update - 1) / a.tb_update;
    return g < a.update_blocks ? g : a.update_blocks;
}

template <typename R> void launch_fluid_gradients_range(const FluidArgs<R> &a, int begin, int end, cudaStream_t s) {
    if (end <= begin) return;
    const int tb = a.tb_grad, g = (end - begin + tb - 1) / tb;
    if (tb == 128) k_cell_gradients<R, 128, false><<<g, 128, 0, s>>>(a, begin, end, nullptr);
    else if (tb == 512) k_cell_gradients<R, 512, false><<<g, 512, 0, s>>>(a, begin, end, nullptr);
    else k_cell_gradients<R, 256, false><<<g, 256, 0, s>>>(a, begin, end, nullptr);
}
// Gradients and fluxes of the cells beside those of the fused step: cells [begin, end) and faces r hold them
// all, with those of the grids between them, whose threads leave at once.
void launch_fluid_rest(const FluidArgs<double> &a, int begin, int end, const FaceRanges &r, Vec4<double> *prev, cudaStream_t s) {
    const int n = r.count[0] + r.count[1] + r.count[2];
    k_cell_gradients<double, 128, true><<<(end - begin + 127) / 128, 128, 0, s>>>(a, begin, end, prev);
    if (n > 0) k_face_flux<double, 128, true><<<(n + 127) / 128, 128, 0, s>>>(a, r);
    if (a.nb > 0) k_face_flux_general<double, 128, true><<<(a.nb + 127) / 128, 128, 0, s>>>(a, a.ni);
}
template <typename R> void launch_fluid_gradients(const FluidArgs<R> &a, cudaStream_t s) {
    launch_fluid_gradients_range<R>(a, 0, a.nc, s);
}
template <typename R> void launch_fluid_flux_axis_ranges(const FluidArgs<R> &a, const FaceRanges &r, cudaStream_t s) {
    const int n = r.count[0] + r.count[1] + r.count[2];
    if (!a.axis_aligned || n == 0) return;
    const int tb = a.tb_flux, g = (n + tb - 1) / tb;
    if (tb == 64) k_face_flux<R, 64, false><<<g, 64, 0, s>>>(a, r);
    else if (tb == 256) k_face_flux<R, 256, false><<<g, 256, 0, s>>>(a, r);
    else k_face_flux<R, 128, false><<<g, 128, 0, s>>>(a, r);
}
// A launch with the programmatic-serialization attribute when `pdl` (the
// kernel directly behind the kernel whose output it reads, on the same stream).
template <typename... KArgs, typename... Args>
void launch_maybe_pdl(void (*kernel)(KArgs...), int g, int tb, cudaStream_t s, bool pdl, Args... args) {
    if (!pdl) {
        kernel<<<g, tb, 0, s>>>(args...);
        return;
    }
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g);
    cfg.blockDim = dim3(tb);
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <typename R, bool CONE>
void launch_general_tiles(const FluidArgs<R> &a, int g, int tile0, cudaStream_t s, bool pdl) {
    if (a.tb_gen == 64) launch_maybe_pdl(k_face_flux_general_tiles<R, 64, CONE>, g, 64, s, pdl, a, tile0);
    else if (a.tb_gen == 256) launch_maybe_pdl(k_face_flux_general_tiles<R, 256, CONE>, g, 256, s, pdl, a, tile0);
    else launch_maybe_pdl(k_face_flux_general_tiles<R, 128, CONE>, g, 128, s, pdl, a, tile0);
}

template <typename R>
void launch_fluid_flux_tiles(const FluidArgs<R> &a, int tile0, int tile1, cudaStream_t s, bool pdl) {
    const int g = tile1 - tile0;
    if (g <= 0) return;
    if (!a.axis_aligned) {
        if (a.cone) launch_general_tiles<R, true>(a, g, tile0, s, pdl);
        else launch_general_tiles<R, false>(a, g, tile0, s, pdl);
        return;
    }
    if (a.tb_flux == 64) launch_maybe_pdl(k_face_flux_tiles<R, 64>, g, 64, s, pdl, a, tile0);
    else if (a.tb_flux == 256) launch_maybe_pdl(k_face_flux_tiles<R, 256>, g, 256, s, pdl, a, tile0);
    else launch_maybe_pdl(k_face_flux_tiles<R, 128>, g, 128, s, pdl, a, tile0);
}
template <typename R> void launch_fluid_flux_axis(const FluidArgs<R> &a, cudaStream_t s, bool pdl) {
    if (a.flux_tiles) {  // interior faces by tiles (axis-aligned or general-normal kernel)
        launch_fluid_flux_tiles<R>(a, 0, a.n_tiles, s, pdl);
        return;
    }
    const FaceRanges r = {{0, a.nfx, a.nfx + a.nfy}, {a.nfx, a.nfy, a.ni - a.nfx - a.nfy}};
    launch_fluid_flux_axis_ranges<R>(a, r, s);
}
// Boundary faces of an axis-aligned mesh: a short launch of long threads (a
// one-wave grid that forms ghost records and general-normal fluxes) that runs
// beside the interior-face tiles on another stream.  Launched with the
// device's greatest scheduling priority so that its blocks are placed first
// and finish under the interior faces instead of after them (the step graph is
// instantiated with per-node priorities).
template <typename R, int TB> void launch_general(const FluidArgs<R> &a, int first, int g, cudaStream_t s, bool hi) {
    if (!hi) {
        k_face_flux_general<R, TB, false><<<g, TB, 0, s>>>(a, first);
        return;
    }
    int lo = 0, top = 0;
    cudaDeviceGetStreamPriorityRange(&lo, &top);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributePriority;
    attr[0].val.priority = top;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(g);
    cfg.blockDim = dim3(TB);
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_face_flux_general<R, TB, false>, a, first);
}
template <typename R> void launch_fluid_flux_general(const FluidArgs<R> &a, cudaStream_t s) {
    // boundary faces only when the interior faces have a kernel of their own (axis faces, or tiles)
    const bool bc_only = a.axis_aligned || a.flux_tiles;
    const int first = bc_only ? a.ni : 0;
    if (a.nf <= first) return;
    const int tb = a.tb_gen, g = (a.nf - first + tb - 1) / tb;
    const bool hi = bc_only;  // beside the interior-face kernel
    if (tb == 64) launch_general<R, 64>(a, first, g, s, hi);
    else if (tb == 256) launch_general<R, 256>(a, first, g, s, hi);
    else launch_general<R, 128>(a, first, g, s, hi);
}
template <typename R> void launch_fluid_flux(const FluidArgs<R> &a, cudaStream_t s) {
    launch_fluid_flux_axis<R>(a, s);
    launch_fluid_flux_general<R>(a, s);
}
template <typename R, int SUMS> void launch_update(const FluidArgs<R> &a, cudaStream_t s, bool pdl) {
    const int tb = a.tb_update, g = k3_grid(a);
    if (tb == 128) launch_maybe_pdl(k_cell_update<R, 128, SUMS>, g, 128, s, pdl, a);
    else if (tb == 512) launch_maybe_pdl(k_cell_update<R, 512, SUMS>, g, 512, s, pdl, a);
    else launch_maybe_pdl(k_cell_update<R, 256, SUMS>, g, 256, s, pdl, a);
}
template <typename R> void launch_fluid_update(const FluidArgs<R> &a, cudaStream_t s, bool pdl) {
    if constexpr (sizeof(R) == 8) {
        if (a.grid_res) return a.grid_mixed ? launch_update<R, MIXED>(a, s, pdl) : launch_update<R, FUSED>(a, s, pdl);
    }
    launch_update<R, GATHER>(a, s, pdl);
}

template <typename R> void launch_fluid_cfl(const FluidArgs<R> &a, cudaStream_t s) {
    const int g = std::min(kCflBlocks, (a.nc + 255) / 256);
    k_cfl<R><<<g, 256, 0, s>>>(a);
}

template <typename R> void launch_pack_state(const FluidArgs<R> &a, const double *stage, cudaStream_t s) {
    k_pack_state<R><<<(a.nc + 255) / 256, 256, 0, s>>>(a, stage);
}
template <typename R> void launch_unpack_state(const FluidArgs<R> &a, double *stage, cudaStream_t s) {
    k_unpack_state<R><<<(a.nc + 255) / 256, 256, 0, s>>>(a, stage);
}
template void launch_pack_state<double>(const FluidArgs<double> &, const double *, cudaStream_t);
template void launch_pack_state<float>(const FluidArgs<float> &, const double *, cudaStream_t);
template void launch_unpack_state<double>(const FluidArgs<double> &, double *, cudaStream_t);
template void launch_unpack_state<float>(const FluidArgs<float> &, double *, cudaStream_t);

template void launch_fluid_gradients<double>(const FluidArgs<double> &, cudaStream_t);
template void launch_fluid_flux<double>(const FluidArgs<double> &, cudaStream_t);
template void launch_fluid_flux_axis<double>(const FluidArgs<double> &, cudaStream_t, bool);
template void launch_fluid_flux_general<double>(const FluidArgs<double> &, cudaStream_t);
template void launch_fluid_flux_axis<float>(const FluidArgs<float> &, cudaStream_t, bool);
template void launch_fluid_flux_general<float>(const FluidArgs<float> &, cudaStream_t);
template void launch_fluid_update<double>(const FluidArgs<double> &, cudaStream_t, bool);
template void launch_fluid_gradients<float>(const FluidArgs<float> &, cudaStream_t);
template void launch_fluid_flux<float>(const FluidArgs<float> &, cudaStream_t);
template void launch_fluid_update<float>(const FluidArgs<float> &, cudaStream_t, bool);
template void launch_fluid_cfl<double>(const FluidArgs<double> &, cudaStream_t);
template void launch_fluid_gradients_range<double>(const FluidArgs<double> &, int, int, cudaStream_t);
template void launch_fluid_gradients_range<float>(const FluidArgs<float> &, int, int, cudaStream_t);
template void launch_fluid_flux_axis_ranges<double>(const FluidArgs<double> &, const FaceRanges &, cudaStream_t);
template void launch_fluid_flux_axis_ranges<float>(const FluidArgs<float> &, const FaceRanges &, cudaStream_t);
template void launch_fluid_flux_tiles<double>(const FluidArgs<double> &, int, int, cudaStream_t, bool);
template void launch_fluid_flux_tiles<float>(const FluidArgs<float> &, int, int, cudaStream_t, bool);
template void launch_fluid_cfl<float>(const FluidArgs<float> &, cudaStream_t);

}  // namespace lbfs
