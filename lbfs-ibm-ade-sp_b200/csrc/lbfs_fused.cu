// The fluid step of uniform grids in one pass over the state; see lbfs_fused.h
// for the plan's conditions and data.
//
// What the separate kernels move per cell (FP64): gradients out and in (96 B
// each), three face fluxes out and in (96 B each), state and accumulator twice
// -- 578 B against the 128 B a step cannot do without -- and their face kernel
// spends about 400 FP64 instructions a face.  Here a block walks a tile of
// columns plane by plane with the states in shared memory.  A gradient component
// times dt is a constant times the difference of two neighbours, so a face takes
// its slopes straight from the states, and the populations of a side's four
// corner directions are not formed one by one: the equilibrium is a cubic
// polynomial in the displaced state, so their sum and first moments come in
// closed form from six dot products (uniform_side), about 250 FP64 instructions a
// face.  A step reads the state and writes the cell sums (and the state it
// started from, from which the gradient and flux fields are formed on request).
#include <cuda_runtime.h>

#include <cstdint>

#include "lbfs_face.cuh"
#include "lbfs_fluid.cuh"
#include "lbfs_fused.h"
#include "lbfs_internal.h"
#include "lbfs_kernels.h"

namespace lbfs {
namespace {

__device__ __forceinline__ double relaxation(const FluidArgs<double> &a, double vf, double dt) {
    return (a.testcase == 8) ? 0.0 : (a.visc * vf * 3.0 / dt * a.gamma_inv);
}

// The ghost of a cell (state s: rho, u, v, w) across a side with record gs, in place of s.
__device__ __forceinline__ void side_ghost(const FluidArgs<double> &a, const GridSide &gs, double (&s)[4]) {
    const double v[4] = {gs.val.rho, gs.val.u, gs.val.v, gs.val.w};
#pragma unroll
    for (int m = 0; m < 4; m++)
        if (gs.flags & (m == 0 ? 1 : 2)) s[m] = v[m] - (s[m] - v[m]);
    if (gs.flags & 12) {
        const Vec4<double> q = a.state[gs.partner];
        const double qv[4] = {q.rho, q.u, q.v, q.w};
#pragma unroll
        for (int m = 0; m < 4; m++)
            if (gs.flags & (m == 0 ? 4 : 8)) s[m] = qv[m];
    }
}

// Boundary blocks among the first `block` blocks of the launch: spread evenly, so
// that each runs beside a tile's block (all of them first were one latency-bound
// wave before the tiles: 40 us of 275 at 128^3).
__device__ __forceinline__ int bnd_before(const GridArgs &ga, unsigned block) {
    return (int)((unsigned long long)block * (unsigned)ga.bnd_blocks / (unsigned)(ga.bnd_blocks + ga.n_tiles));
}

// ---- the tiles -------------------------------------------------------------------
//
// Four planes (k - 1 .. k + 1 in use, k + 2 in flight) of the tile with its ring
// are in shared memory, brought in by asynchronous 16-byte copies, so no thread
// waits for global memory inside the walk.  Every thread owns a column and forms
// the three low faces of its cells, so all lanes work on every face; the high
// faces of a tile and the upper ones of a walk are another block's low ones, which
// it also leaves in ga.edge for the update to subtract (forming them here too, by a
// warp of their own, cost a fifth: 265 against 203 us at 128^3 FP64).  A walk
// subtracts a cell's upper z flux last and scales nothing, and the update goes on
// from there: the order of a cell's sum does not depend on where its walk ends,
// which follows from all grids of the handle.  Ghosts are
// cells of the ring: copied from the cell beside them (zero gradient) and, where
// they are not, set from the side's record after the copy's arrival by the thread
// that issued it.  Bound by FP64 issue inside the walk (of its cycles about three
// quarters); blocks of four warps, four to an SM at 128 registers, keep a walk's
// start and the short waits of one block under the others' faces.  Gradients kept
// in shared memory instead (two planes of 13 values, two blocks of 256 threads an
// SM) took 362 us: their loads were waited for.
constexpr int kSlots = 4;

__device__ __forceinline__ void copy16(void *smem, const void *g) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(g) : "memory");
}
__device__ __forceinline__ void copy8(void *smem, const void *g) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(a), "l"(g) : "memory");
}

struct State4 {
    double s[4];  // rho, u, v, w
};

// The staged planes: the halves of slot t's states at h[(2 t + half) Q + position].
struct Planes {
    double2 *h;
    int Q;
    __device__ __forceinline__ void get(int at, double (&s)[4]) const {  // at = 2 slot Q + position; rho, u, v, w
        const double2 p = h[at], q = h[at + Q];
        s[1] = p.x; s[2] = p.y; s[3] = q.x; s[0] = q.y;
    }
    __device__ __forceinline__ State4 at(int i) const {
        State4 q;
        get(i, q.s);
        return q;
    }
    __device__ __forceinline__ void put(int at, const double (&s)[4]) const {
        h[at] = make_double2(s[1], s[2]);
        h[at + Q] = make_double2(s[3], s[0]);
    }
};

// A cell's state and its neighbours' differences along each axis (upper - lower).
struct CellSlopes {
    double s[4], d[3][4];
};

// Lattice moments of one side of a face.  Its nodes in the directions e = (s e_A,
// e_B, e_C), e_B, e_C = +-1, hold L = a - e_B b - e_C c: a the value at the node of
// direction s e_A, which is the cell's centre, b and c its gradients along B and C
// times dt.  In velocities times 3 (v = 3 u) the population over its weight is g =
// rho (1 + X), 1 + X = (1 + (1 + e.v)^2 - |v|^2 / 3) / 2, and with
//   1 + e.v = al + e_B be + e_C ga + e_B e_C de,
//   |v|^2 = (aa + bb + cc) - 2 e_B ab - 2 e_C ac + 2 e_B e_C bc
// it has the form q0 + e_B XB + e_C XC + e_B e_C XBC, so that the sums over the four
// corners are products of these with rho's three terms.  A quarter of each sum:
// S = sum g, YB = sum e_B g, YC = sum e_C g; ga0 is twice g of direction s e_A alone.
// The slopes' weight w (dt x gradient weight, its multiples in GridWeights) is
// applied to sums and not to the twelve differences.  rho, a: the cell's density
// and v; db, dc: its neighbours' differences along B and C (velocities not scaled).
struct SideSums {
    double S, YB, YC, ga0;
};
template <int A, int SGN>
__device__ __forceinline__ SideSums uniform_side(double rho, const double (&a)[3], const double (&db)[4],
                                                 const double (&dc)[4], const GridWeights &g) {
    constexpr int B = A == 0 ? 1 : 0, C = A == 2 ? 1 : 2;
    constexpr double s = SGN;
    const double be = SGN > 0 ? a[B] - g.w3 * db[1 + A] : a[B] + g.w3 * db[1 + A];
    const double ga = SGN > 0 ? a[C] - g.w3 * dc[1 + A] : a[C] + g.w3 * dc[1 + A];
    const double de = -g.w3 * (db[1 + C] + dc[1 + B]);
    const double sl = db[1 + B] + dc[1 + C];
    const double aa = a[0] * a[0] + a[1] * a[1] + a[2] * a[2];
    const double nn = (db[1] * db[1] + db[2] * db[2] + db[3] * db[3]) + (dc[1] * dc[1] + dc[2] * dc[2] + dc[3] * dc[3]);
    const double ab = a[0] * db[1] + a[1] * db[2] + a[2] * db[3];
    const double ac = a[0] * dc[1] + a[1] * dc[2] + a[2] * dc[3];
    const double bc = db[1] * dc[1] + db[2] * dc[2] + db[3] * dc[3];
    const double b0 = g.w * db[0], c0 = g.w * dc[0];
    SideSums r;
    const double ea = 1.0 + s * a[A];
    const double al = ea - g.w3 * sl;
    const double Ka = 1.0 - (1.0 / 3.0) * aa;
    const double q0 = 0.5 * ((Ka + al * al + be * be) + (ga * ga + de * de - g.ww3 * nn));
    const double XB = g.w * ab + (al * be + ga * de), XC = g.w * ac + (al * ga + be * de);
    const double XBC = (al * de + be * ga) - g.ww3 * bc;
    r.S = rho * q0 - b0 * XB - c0 * XC;
    r.YB = rho * XB - b0 * q0 - c0 * XBC;
    r.YC = rho * XC - c0 * q0 - b0 * XBC;
    r.ga0 = rho * (Ka + ea * ea);
    return r;
}

// Half the sum and half the difference of the populations (over their weight) of
// the opposite directions +-e_X at the face centre, in the same variables: rho, p
// its density and v, K = 1 - |v|^2 / 3; ds the sum of both cells' differences along
// X, w / 2 times which is the displacement (L = p -+ b).
template <int X>
__device__ __forceinline__ void uniform_pair(double rho, const double (&p)[3], double K, const double (&ds)[4],
                                             const GridWeights &g, double &sum, double &dif) {
    const double bb = ds[1] * ds[1] + ds[2] * ds[2] + ds[3] * ds[3];
    const double pb = p[0] * ds[1] + p[1] * ds[2] + p[2] * ds[3];
    const double b0 = g.h * ds[0], px = p[X];
    const double c = 1.0 - g.h3 * ds[1 + X];
    const double q0 = 0.5 * ((K + c * c) + (px * px - g.hh3 * bb));
    const double odd = g.h * pb + c * px;
    sum = rho * q0 - b0 * odd;
    dif = rho * odd - b0 * q0;
}

// Flux per unit area (rho, u, v, w) through an axis-A face: its density p0 and v at
// the centre, the sums of both cells' differences along B and C and the sides' sums.
template <int A>
__device__ __forceinline__ Vec4<double> face_flux(const GridWeights &g, double p0, const double (&p)[3],
                                                  const double (&bs)[4], const double (&cs)[4], const SideSums &o,
                                                  const SideSums &n, double tau) {
    constexpr int B = A == 0 ? 1 : 0, C = A == 2 ? 1 : 2;
    // the rest and tangential directions from the face centre
    const double pp = (-1.0 / 3.0) * (p[0] * p[0] + p[1] * p[1] + p[2] * p[2]);
    const double K = 1.0 + pp;
    double sB, dB, sC, dC;
    uniform_pair<B>(p0, p, K, bs, g, sB, dB);
    uniform_pair<C>(p0, p, K, cs, g, sC, dC);
    const double gz0 = p0 * (1.0 + 0.5 * pp);
    constexpr double w0 = 2.0 / 9.0, wh = 1.0 / 18.0;
    // moments, relaxation and the axis-A flux (interface_flux): with u = m_A / rho the relaxed second
    // moments are (1 - tau) (u m_q + d_Aq rho / 3) + tau F_q
    const double So = wh * (o.ga0 + o.S), Sn = wh * (n.ga0 + n.S);  // 1/9 of ga0 / 2, four corners of 1/72
    const double rho = (So + Sn) + w0 * (gz0 + (sB + sC));
    const double mA = So - Sn, mB = wh * (o.YB + n.YB) + w0 * dB, mC = wh * (o.YC + n.YC) + w0 * dC;
    const double keep = 1.0 - tau;
    const double ku = keep * (mA / rho), th = tau * wh;
    Vec4<double> r;
    r.rho = mA;
    const double fA = ku * mA + (keep * (1.0 / 3.0)) * rho + tau * (So + Sn);
    const double fB = ku * mB + th * (o.YB - n.YB), fC = ku * mC + th * (o.YC - n.YC);
    r.u = A == 0 ? fA : fB;
    r.v = A == 1 ? fA : (A == 0 ? fB : fC);
    r.w = A == 2 ? fA : fC;
    return r;
}

// Flux per unit area (rho, u, v, w) through the low axis-A face of the cell hi:
// the lower cell at lo, its lower neighbour's state lm and its neighbours lbm, lbp
// along B and lcm, lcp along C.
template <int A>
__device__ __forceinline__ Vec4<double> uniform_flux(const GridWeights &g, const Planes &pl, const CellSlopes &hi, int lo,
                                                     const State4 &lm, int lbm, int lbp, int lcm, int lcp, double tau) {
    constexpr int B = A == 0 ? 1 : 0, C = A == 2 ? 1 : 2;
    double s1[4], p0, p[3];
    pl.get(lo, s1);
    {
        const double(&q)[4] = lm.s;
        p0 = 0.5 * (s1[0] + hi.s[0]) + g.h * ((hi.s[0] - q[0]) - hi.d[A][0]);
#pragma unroll
        for (int m = 0; m < 3; m++)
            p[m] = 1.5 * (s1[1 + m] + hi.s[1 + m]) + g.h3 * ((hi.s[1 + m] - q[1 + m]) - hi.d[A][1 + m]);
    }
    double b[4], c[4];
    {
        double q0[4], q1[4];
        pl.get(lbm, q0);
        pl.get(lbp, q1);
#pragma unroll
        for (int m = 0; m < 4; m++) b[m] = q1[m] - q0[m];
        pl.get(lcm, q0);
        pl.get(lcp, q1);
#pragma unroll
        for (int m = 0; m < 4; m++) c[m] = q1[m] - q0[m];
    }
    const double v1[3] = {3.0 * s1[1], 3.0 * s1[2], 3.0 * s1[3]};
    const SideSums o = uniform_side<A, 1>(s1[0], v1, b, c, g);
    const double v2[3] = {3.0 * hi.s[1], 3.0 * hi.s[2], 3.0 * hi.s[3]};
    const SideSums n = uniform_side<A, -1>(hi.s[0], v2, hi.d[B], hi.d[C], g);
    double bs[4], cs[4];
#pragma unroll
    for (int m = 0; m < 4; m++) { bs[m] = b[m] + hi.d[B][m]; cs[m] = c[m] + hi.d[C][m]; }
    return face_flux<A>(g, p0, p, bs, cs, o, n, tau);
}

// ---- boundary faces ----------------------------------------------------------------
// The same face forms in the frame of the outward normal (axis 0; the components
// are turned and, on the lower sides, reflected into it; calc_face_flux_bc,
// LBFS.cu:2691-2810).  A boundary face takes every direction from the face state p0
// with the ghost's gradients, so its sides' nodes are p0 -+ w D_n; the first ghost's
// face is an interior face between the cell and the ghost.  In the differences' units
// the ghost's gradients are the cell's without their normal part (zero gradient),
// bnd_k times ghost - cell along the normal (Dirichlet), or the partner cell's
// (periodic).  One thread per face, two dependent loads deep; with the gradients and
// the flux of the general-normal kernel (five deep, about 900 instructions) these
// faces were 30 us of the pass at 128^3 FP64 and half of it on 48,000 cells.

// Differences (upper - lower) along x, y, z around the cell of boundary face f.
__device__ __forceinline__ void boundary_slopes(const FluidArgs<double> &a, const GridArgs &ga, const GridBnd &f,
                                                const GridSide &rec, const double (&own)[4], double (&d)[3][4]) {
    const unsigned at[3] = {(unsigned)f.info & 7u, (unsigned)(f.info >> 3) & 7u, (unsigned)(f.info >> 6) & 7u};
    const unsigned miss = 1u << at[0] | 1u << at[1] | 1u << at[2];  // bit 7: none
    const Vec4<double> *st = a.state + f.cell;
    const int step[3] = {1, f.sy, f.sz};
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const Vec4<double> lo = st[(miss >> (2 * q) & 1u) ? 0 : -step[q]], hi = st[(miss >> (2 * q + 1) & 1u) ? 0 : step[q]];
        d[q][0] = hi.rho - lo.rho;
        d[q][1] = hi.u - lo.u;
        d[q][2] = hi.v - lo.v;
        d[q][3] = hi.w - lo.w;
    }
#pragma unroll
    for (int e = 0; e < 3; e++) {
        if (at[e] > 5u) continue;
        double gs[4] = {own[0], own[1], own[2], own[3]};
        side_ghost(a, e == 0 ? rec : ga.bnd_side[f.more[e - 1]], gs);
        const double sg = (at[e] & 1u) ? 1.0 : -1.0;
#pragma unroll
        for (int q = 0; q < 3; q++)
#pragma unroll
            for (int m = 0; m < 4; m++)
                if ((int)(at[e] >> 1) == q) d[q][m] = d[q][m] + sg * (gs[m] - own[m]);
    }
}

__device__ __forceinline__ void grid_boundary(const FluidArgs<double> &a, const GridArgs &ga, const GridSet &gs,
                                              const GridBnd &f, int b) {
    const GridSide rec = ga.bnd_side[b];
    const int side = f.info & 7, axis = side >> 1;
    double d[3][4], dp[3][4];
    State4 own, ghost;
    {
        const Vec4<double> s = a.state[f.cell];
        own = {{s.rho, s.u, s.v, s.w}};
    }
    boundary_slopes(a, ga, f, rec, own.s, d);
    ghost = own;
    side_ghost(a, rec, ghost.s);
    if (rec.flags & 12) {  // the partner's slopes
        const Vec4<double> s = a.state[rec.partner];
        const double q[4] = {s.rho, s.u, s.v, s.w};
        boundary_slopes(a, ga, ga.bnd[f.partner], ga.bnd_side[f.partner], q, dp);
    } else {
#pragma unroll
        for (int q = 0; q < 3; q++)
#pragma unroll
            for (int m = 0; m < 4; m++) dp[q][m] = 0.0;
    }
    // into the frame: components (n, t1, t2) = (axis, the other two in order), n outward
    const double sn = (side & 1) ? 1.0 : -1.0;
    auto turn = [&](double x, double y, double z, double (&o)[3]) {
        o[0] = sn * (axis == 0 ? x : (axis == 1 ? y : z));
        o[1] = axis == 0 ? y : x;
        o[2] = axis == 2 ? y : z;
    };
    auto turned = [&](const double (&v)[4]) {
        State4 o;
        o.s[0] = v[0];
        double t[3];
        turn(v[1], v[2], v[3], t);
        o.s[1] = t[0]; o.s[2] = t[1]; o.s[3] = t[2];
        return o;
    };
    double e[3][4], ep[3][4];  // differences along n, t1, t2 with turned components
    auto turn_slopes = [&](const double (&v)[3][4], double (&o)[3][4]) {
        const State4 x = turned(v[0]), y = turned(v[1]), z = turned(v[2]);
#pragma unroll
        for (int m = 0; m < 4; m++) {
            double t[3];
            turn(x.s[m], y.s[m], z.s[m], t);
            o[0][m] = t[0]; o[1][m] = t[1]; o[2][m] = t[2];
        }
    };
    turn_slopes(d, e);
    turn_slopes(dp, ep);
    const State4 S1 = turned(own.s), S2 = turned(ghost.s), V = turned({rec.val.rho, rec.val.u, rec.val.v, rec.val.w});
    const GridWeights &g = gs.cw;
    const bool first = (f.info & 1024) != 0;
    double p[4], a1[4], a2[4];
    double b1[4], c1[4], b2[4], c2[4];
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const bool dir = (rec.flags & (m == 0 ? 1 : 2)) != 0;
        const bool per = (rec.flags & (m == 0 ? 4 : 8)) != 0;
        const double Dn = dir ? gs.bnd_k * (S2.s[m] - S1.s[m]) : (per ? ep[0][m] : 0.0);  // ghost's differences
        b2[m] = dir ? 0.0 : (per ? ep[1][m] : e[1][m]);
        c2[m] = dir ? 0.0 : (per ? ep[2][m] : e[2][m]);
        const double wD = g.w * Dn;
        const bool set = (rec.flags & (m == 0 ? 1 : 16)) != 0;
        const double h = g.h * (e[0][m] - Dn), hd = 0.5 * (S1.s[m] - S2.s[m]);
        p[m] = first ? S1.s[m] - (hd - h) : (set ? V.s[m] : S1.s[m] + wD);
        a1[m] = first ? S1.s[m] : p[m] - wD;
        a2[m] = first ? S2.s[m] : p[m] + wD;
        b1[m] = first ? e[1][m] : b2[m];
        c1[m] = first ? e[2][m] : c2[m];
    }
    const double v1[3] = {3.0 * a1[1], 3.0 * a1[2], 3.0 * a1[3]}, v2[3] = {3.0 * a2[1], 3.0 * a2[2], 3.0 * a2[3]};
    const double pv[3] = {3.0 * p[1], 3.0 * p[2], 3.0 * p[3]};
    const SideSums o = uniform_side<0, 1>(a1[0], v1, b1, c1, g);
    const SideSums n = uniform_side<0, -1>(a2[0], v2, b2, c2, g);
#pragma unroll
    for (int m = 0; m < 4; m++) { b1[m] = b1[m] + b2[m]; c1[m] = c1[m] + c2[m]; }
    const Vec4<double> t = face_flux<0>(g, p[0], pv, b1, c1, o, n, relaxation(a, 1.0, gs.dt));
    const double fn = sn * t.u;
    Vec4<double> out;
    out.rho = t.rho * gs.area;
    out.u = (axis == 0 ? fn : t.v) * gs.area;
    out.v = (axis == 1 ? fn : (axis == 0 ? t.v : t.w)) * gs.area;
    out.w = (axis == 2 ? fn : t.w) * gs.area;
    a.flux[a.ni + f.face] = out;
}

// SETS: grids of several spacings, whose constants a block loads (one spacing: kernel parameters).
template <bool SETS>
__global__ void __launch_bounds__(kUniformThreads, kUniformBlocks) k_uniform_step(FluidArgs<double> a, GridArgs ga) {
    extern __shared__ __align__(16) unsigned char raw[];
    constexpr int H = 2, TB = kUniformThreads;  // H 16-byte pieces of a state record
    pdl_trigger();
    const int bnd = bnd_before(ga, blockIdx.x);
    if (bnd_before(ga, blockIdx.x + 1) > bnd) {
        const int b = bnd * TB + threadIdx.x;
        if (b >= ga.n_bnd) return;
        const GridBnd f = ga.bnd[b];
        if constexpr (SETS) grid_boundary(a, ga, ga.sets[f.info >> 11], f, b);
        else grid_boundary(a, ga, ga.set, f, b);
        return;
    }
    const GridTile t = ga.tiles[blockIdx.x - bnd];
    const GridInst gi = ga.inst[t.inst];
    const GridSet &gs = SETS ? ga.sets[t.set] : ga.set;
    const int Q = ga.plane_stride;
    Planes pl;
    pl.h = reinterpret_cast<double2 *>(raw);
    pl.Q = Q;
    double *sum = reinterpret_cast<double *>(pl.h + (size_t)kSlots * H * Q);  // [4][TB] the columns' sums
    GridSide *stage = reinterpret_cast<GridSide *>(sum + 4 * TB);       // [stage_max] ghosts' records
    double *vis = reinterpret_cast<double *>(stage + ga.stage_max);                     // [3][Q]
    double *fx = vis + 3 * Q, *fy = fx + 4 * TB, *below = fy + 4 * TB;             // [4][TB]: the plane's fluxes, states two planes down
    const int tid = threadIdx.x, W = t.w + 3;
    const int nxy = gi.nx * gi.ny;
    const int z_end = t.z0 + t.d;

    // what this thread brings in of every plane: up to two cells of the tile with its ring, and one ghost
    int load_c[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int p = tid + q * TB;
        const int y = p / W, x = p - y * W;
        const int gx = t.x0 + x - 2, gy = t.y0 + y - 2;
        const bool on = y < t.h + 3 && gx >= 0 && gx < gi.nx && gy >= 0 && gy < gi.ny;
        load_c[q] = on ? gi.cell0 + gx + gi.nx * gy : -1;
    }
    int ghost_at = -1, ghost_c = 0, ghost_rec = 0, ghost_step = 0;
    bool ghost_set = false;
    {
        // the grid's edges -x, +x (rows -1 .. h), -y, +y (columns -1 .. w) where they cross the tile's ring
        int g = tid, x = 0, y = 0, d = -1;
        if (g < t.h + 2) { d = 0; x = -1 - t.x0; y = g - 1; }
        else if ((g -= t.h + 2) < t.h + 2) { d = 1; x = gi.nx - t.x0; y = g - 1; }
        else if ((g -= t.h + 2) < t.w + 2) { d = 2; y = -1 - t.y0; x = g - 1; }
        else if ((g -= t.w + 2) < t.w + 2) { d = 3; y = gi.ny - t.y0; x = g - 1; }
        const int gx = t.x0 + x, gy = t.y0 + y;
        const bool along = d < 2 ? (x >= -2 && x <= t.w && gy >= 0 && gy < gi.ny)
                                 : (y >= -2 && y <= t.h && gx >= 0 && gx < gi.nx);
        if (d >= 0 && along) {
            ghost_at = (y + 2) * W + x + 2;
            ghost_c = gi.cell0 + min(max(gx, 0), gi.nx - 1) + gi.nx * min(max(gy, 0), gi.ny - 1);
            ghost_rec = gi.side0[d] + (d < 2 ? gy : gx);
            ghost_step = d < 2 ? gi.ny : gi.nx;
            ghost_set = (gi.active >> d & 1) != 0;
        }
    }
    // starts bringing in plane k (-1 and nz: the ghosts of the first and last plane), and the viscosity
    // factors of plane k - 1
    auto bring = [&](int k, bool staged) {
        const int base = H * (k & (kSlots - 1)) * Q;
        const int kc = min(max(k, 0), gi.nz - 1);
        const int side = k < 0 ? 4 : (k >= gi.nz ? 5 : -1);
        const bool set = side >= 0 && (gi.active >> side & 1);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            if (load_c[q] < 0) continue;
            const int p = tid + q * TB;
            const int c = load_c[q] + nxy * kc;
            if (set) {  // the ghost of cell c across the grid's first or last plane
                const Vec4<double> own = a.state[c];
                double s[4] = {own.rho, own.u, own.v, own.w};
                side_ghost(a, ga.side[gi.side0[side] + load_c[q] - gi.cell0], s);
                pl.put(base + p, s);
            } else {
                const char *src = reinterpret_cast<const char *>(a.state + c);
#pragma unroll
                for (int e = 0; e < H; e++) copy16(pl.h + base + e * Q + p, src + 16 * e);
            }
            if (k > 0) copy8(vis + ((k - 1) % 3) * Q + p, a.visc_factor + load_c[q] + nxy * (k - 1));
        }
        if (ghost_at >= 0 && side < 0) {
            const char *src = reinterpret_cast<const char *>(a.state + ghost_c + nxy * k);
#pragma unroll
            for (int e = 0; e < H; e++) copy16(pl.h + base + e * Q + ghost_at, src + 16 * e);
            if (ghost_set && staged) {
                const char *rec = reinterpret_cast<const char *>(ga.side + ghost_rec + (size_t)ghost_step * k);
#pragma unroll
                for (int e = 0; e < (int)(sizeof(GridSide) / 16); e++)
                    copy16(reinterpret_cast<char *>(stage + tid) + 16 * e, rec + 16 * e);
            }
        }
    };
    // this thread's copies have arrived; its ghost of plane k is set where it is not zero-gradient
    auto landed = [&]() { asm volatile("cp.async.wait_all;" ::: "memory"); };
    auto set_ghost = [&](int k, const GridSide &rec) {
        const int at = H * (k & (kSlots - 1)) * Q + ghost_at;
        double s[4];
        pl.get(at, s);
        side_ghost(a, rec, s);
        pl.put(at, s);
    };

    const int ly = tid / t.w, lx = tid - ly * t.w;
    const bool own = ly < t.h;
    const int gx = t.x0 + lx, gy = t.y0 + ly;
    const int at = (ly + 2) * W + lx + 2;
    const int c00 = gi.cell0 + gx + gi.nx * gy;
    const double tau1 = relaxation(a, 1.0, gs.dt);  // at a viscosity factor of 1
    const size_t n = (size_t)a.nc;

    for (int k = t.z0 - 1; k <= t.z0 + 1; k++) bring(k, false);
    if (own && t.z0 > 0) {  // two planes down: the plane's cell, or the ghost of the first plane's
        const Vec4<double> q = a.state[c00 + nxy * max(t.z0 - 2, 0)];
        double s[4] = {q.rho, q.u, q.v, q.w};
        if (t.z0 == 1 && (gi.active & 16)) side_ghost(a, ga.side[gi.side0[4] + c00 - gi.cell0], s);
#pragma unroll
        for (int m = 0; m < 4; m++) below[m * TB + tid] = s[m];
    }
    landed();
    if (ghost_set)
        for (int k = max(t.z0 - 1, 0); k <= min(t.z0 + 1, gi.nz - 1); k++)
            set_ghost(k, ga.side[ghost_rec + (size_t)ghost_step * k]);
    for (int k = t.z0; k < z_end; k++) {
        if (k > t.z0) {
            landed();
            if (ghost_set && k + 1 < gi.nz) set_ghost(k + 1, stage[tid]);
        }
        __syncthreads();  // plane k + 1 is complete, and everyone is done with plane k - 1's fluxes
        const int o = H * Q;
        const int pm = o * ((k - 1) & (kSlots - 1)), pk = o * (k & (kSlots - 1)), pp = o * ((k + 1) & (kSlots - 1));
        if (k + 1 < z_end) bring(k + 2, true);  // over plane k - 2, last read before the barrier
        const int c = c00 + nxy * k;
        CellSlopes cell;
        if (own) {
            pl.get(pk + at, cell.s);
            auto diff = [&](int m0, int p1, double (&d)[4]) {
                double q0[4], q1[4];
                pl.get(m0, q0);
                pl.get(p1, q1);
#pragma unroll
                for (int m = 0; m < 4; m++) d[m] = q1[m] - q0[m];
            };
            diff(pk + at - 1, pk + at + 1, cell.d[0]);
            diff(pk + at - W, pk + at + W, cell.d[1]);
            diff(pm + at, pp + at, cell.d[2]);
            ga.prev[c] = {cell.s[1], cell.s[2], cell.s[3], cell.s[0]};
            const double *vis0 = vis + (k % 3) * Q + at;
            if (gx > 0) {
                const int l = pk + at - 1;
                const Vec4<double> v = uniform_flux<0>(gs.cw, pl, cell, l, pl.at(l - 1), l - W, l + W, pm + at - 1,
                                                     pp + at - 1, tau1 * vis0[-1]);
                double *f = fx + tid;
                f[0] = v.rho; f[TB] = v.u; f[2 * TB] = v.v; f[3 * TB] = v.w;
                if (lx == 0) ga.edge[c] = v;
            }
            if (gy > 0) {
                const int l = pk + at - W;
                const Vec4<double> v = uniform_flux<1>(gs.cw, pl, cell, l, pl.at(l - W), l - 1, l + 1, pm + at - W,
                                                     pp + at - W, tau1 * vis0[-W]);
                double *f = fy + tid;
                f[0] = v.rho; f[TB] = v.u; f[2 * TB] = v.v; f[3 * TB] = v.w;
                if (ly == 0) ga.edge[n + c] = v;
            }
        }
        __syncthreads();
        if (own) {
            Vec4<double> z{};
            if (k > 0) {
                const int l = pm + at;
                State4 two;  // of plane k - 2
#pragma unroll
                for (int m = 0; m < 4; m++) two.s[m] = below[m * TB + tid];
                z = uniform_flux<2>(gs.cw, pl, cell, l, two, l - 1, l + 1, l - W, l + W, tau1 * vis[((k - 1) % 3) * Q + at]);
                if (k == t.z0) ga.edge[2 * n + c] = z;
            }
            double lo[4];
            pl.get(pm + at, lo);
#pragma unroll
            for (int m = 0; m < 4; m++) below[m * TB + tid] = lo[m];
            const double zl[4] = {z.rho, z.u, z.v, z.w};
            double below_sum[4];
#pragma unroll
            for (int m = 0; m < 4; m++) {
                below_sum[m] = sum[m * TB + tid] - (double)zl[m];
                double v = (double)zl[m];
                if (gx > 0) v = v + (double)fx[m * TB + tid];
                if (lx + 1 < t.w) v = v - (double)fx[m * TB + tid + 1];
                if (gy > 0) v = v + (double)fy[m * TB + tid];
                if (ly + 1 < t.h) v = v - (double)fy[m * TB + tid + t.w];
                sum[m * TB + tid] = v;
            }
            if (k > t.z0)  // the cell below is complete
                ga.res[c - nxy] = make_double4(below_sum[0], below_sum[1], below_sum[2], below_sum[3]);
        }
    }
    if (own) {  // the last cell's upper face belongs to the walk above (or there is none)
        ga.res[c00 + nxy * (z_end - 1)] = make_double4(sum[tid], sum[TB + tid], sum[2 * TB + tid], sum[3 * TB + tid]);
    }
}

}  // namespace

size_t grid_smem_bytes(const GridArgs &ga) {
    return sizeof(double) * ((kSlots * 4 + 3) * (size_t)ga.plane_stride + 12 * (size_t)kUniformThreads) +
           32 * (size_t)kUniformThreads + ga.stage_max * sizeof(GridSide);
}
// The limit is the kernel's, shared by every handle: always the largest.
cudaError_t grid_prepare() {
    const cudaError_t e = cudaFuncSetAttribute(k_uniform_step<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_uniform_step<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
}
static_assert(sizeof(double) * ((kSlots * 4 + 3) * kUniformPlaneMax + 12 * kUniformThreads) +
                      kUniformThreads * (32 + sizeof(GridSide)) <= 64 * 1024,
              "a tile's shared memory");
void launch_grid_step(const FluidArgs<double> &a, const GridArgs &ga, cudaStream_t s) {
    const int blocks = ga.bnd_blocks + ga.n_tiles;
    if (ga.n_sets > 1) k_uniform_step<true><<<blocks, kUniformThreads, grid_smem_bytes(ga), s>>>(a, ga);
    else k_uniform_step<false><<<blocks, kUniformThreads, grid_smem_bytes(ga), s>>>(a, ga);
}

}  // namespace lbfs
