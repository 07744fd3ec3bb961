// Device functions of the fluid kernels: ghost states, cell gradients, lattice
// populations and face fluxes, shared by the separate kernels (lbfs_fluid.cu)
// and the fused step of structured grids (lbfs_fused.cu).
#pragma once

#include "lbfs_fluid.cuh"

namespace lbfs {

// Ghost-cell macros from the owner state (update_unstructured_bcs,
// LBFS.cu:1868-1918).  Type 3 (periodic) takes the partner cell's state, as
// the reference's CPU solver does (Solution::update_unstructured_bcs,
// Solution.cpp:777-803).  Types outside {1,2,3} / {1,2,3,9,10} are rejected at
// creation, so every branch here assigns.
template <typename R>
__device__ __forceinline__ Vec4<R> ghost_state(const FluidArgs<R> &a, int b, const Vec4<R> &own) {
    const Vec4<R> bc = a.bc_val[b];
    Vec4<R> g;
    const int rt = a.bc_rho_type[b], vt = a.bc_vel_type[b];
    const Vec4<R> p = (rt == 3 || vt == 3) ? a.state[a.bc_periodic[b]] : own;
    if (rt == 1) g.rho = bc.rho - (own.rho - bc.rho);
    else if (rt == 2) g.rho = own.rho;
    else g.rho = p.rho;
    if (vt == 3) {
        g.u = p.u; g.v = p.v; g.w = p.w;
    } else if (vt == 2) {
        g.u = own.u; g.v = own.v; g.w = own.w;
    } else {
        R ut = bc.u;
        if (vt == 9) {
            const BcRec<R> r = a.bc_rec[b];
            ut = (R)(16 * (double)bc.u * (a.H2 + r.gy) * (a.H2 - r.gy) * (a.H2 + r.gz) * (a.H2 - r.gz) / a.H4);
        } else if (vt == 10) {
            ut = a.bc_rec[b].gy * bc.u;
        }
        g.u = ut - (own.u - ut);
        g.v = bc.v - (own.v - bc.v);
        g.w = bc.w - (own.w - bc.w);
    }
    return g;
}

// Least-squares gradients of cell i (state own) over its stencil, ghost states
// formed from the cell's own (K1).
template <typename R>
__device__ __forceinline__ void cell_gradient(const FluidArgs<R> &a, int i, const Vec4<R> &own, R (&g)[12]) {
    int st[6];
#pragma unroll
    for (int q = 0; q < 3; q++) {
        const int2 p = __ldg(a.stencil + 3 * i + q);
        st[2 * q] = p.x;
        st[2 * q + 1] = p.y;
    }
    LsW<R> W;
    if (a.lsw_code) {  // the weights from the per-mesh table by the cell's six 3-bit codes
        const unsigned code = __ldg(a.lsw_code + i);
#pragma unroll
        for (int q = 0; q < 6; q++) {
            const unsigned k = (code >> (3 * q)) & 7u;
#pragma unroll
            for (int r = 0; r < 3; r++) {
                R v = a.lsw_tab[0][r];
#pragma unroll
                for (unsigned t = 1; t < 8; t++) v = (k == t) ? a.lsw_tab[t][r] : v;
                W.w[3 * q + r] = v;
            }
        }
    } else {
        W = a.lsw[i];
    }
#pragma unroll
    for (int t = 0; t < 12; t++) g[t] = R(0);
#pragma unroll
    for (int q = 0; q < 6; q++) {
        const int j = st[q];
        Vec4<R> s;
        if (j < a.nc) {
            s = a.state[j];
        } else {
            s = ghost_state(a, j - a.nc, own);
        }
        // add_LS_contributions (LBFS.cu:2051-2083) with LHS^-1 folded in
        const R d[4] = {s.rho - own.rho, s.u - own.u, s.v - own.v, s.w - own.w};
#pragma unroll
        for (int m = 0; m < 4; m++)
#pragma unroll
            for (int r = 0; r < 3; r++) g[3 * m + r] = g[3 * m + r] + W.w[3 * q + r] * d[m];
    }
}

// Density offset of the stored state: 0 in FP64 (a compile-time zero, so no
// add is spent on it), rho0 in the FP32-bulk form.
template <typename R> __device__ __forceinline__ R rho0_of(const FluidArgs<R> &a) {
    if constexpr (sizeof(R) == 8) return R(0);
    else return a.rho0;
}

// Lattice population divided by its weight, g_k = f_k / w_k, at a reconstructed
// state L = (rho', u, v, w):  g = rho' + (rho' + rho0) X,
// X = 3 e.u + q (4.5 (e.u)^2 - 1.5 |u|^2).  The reference's equilibrium
// w_k rho (1 + X) (populate_feq_lattice_explicit, LBFS.cu:1041-1354; populate_feq,
// LBFS.cu:940-1036 with the preconditioning factor q) with the weight applied
// later, once per group of directions that share it.
template <typename R>
__device__ __forceinline__ R pop_g(const R (&L)[4], R eu, R rho0, R q) {
    const R usq = L[1] * L[1] + L[2] * L[2] + L[3] * L[3];
    const R X = R(3) * eu + q * (R(4.5) * eu * eu - R(1.5) * usq);
    if constexpr (sizeof(R) == 8) return L[0] + L[0] * X;
    else return L[0] + (L[0] + rho0) * X;
}

// FP32-bulk (deviation) form of pop_g at a reconstructed state written as
// L = p0 + d, p0 the face-centre state and d the direction's small offset
// from it.  The population's term 3 rho0 e.p0_u is large (the velocity
// itself) and the same for every direction, so that summing the populations
// over directions would cancel it and leave its FP32 rounding in the
// cross-stream moments; it is left out here, and its moments (rho0 p0_u in
// the first moment, zero in every other) are added once, exactly, by the
// caller.  The rest is formed from small terms only:
//   g~ = rho' (1 + X) + rho0 (3 e.d_u + q (4.5 (e.u)^2 - 1.5 |u|^2)).
// eu = e.u at L, edu = e.d_u.
__device__ __forceinline__ float pop_dev(const float (&L)[4], float eu, float edu, float rho0, float q) {
    const float usq = L[1] * L[1] + L[2] * L[2] + L[3] * L[3];
    const float Q = q * (4.5f * eu * eu - 1.5f * usq);
    const float X = 3.0f * eu + Q;
    return (L[0] + L[0] * X) + rho0 * (3.0f * edu + Q);
}

// Moments of the reconstructed lattice populations that the interface flux
// needs: rho = sum f, m_c = sum e_c f, d_c = sum_{e_c != 0} f (= sum e_c e_c f),
// o_xy, o_xz, o_yz = sum e_c e_m f.  Formed from sums and differences of
// opposite directions (the D3Q15 set is symmetric), then weighted once per
// group: a few dozen adds instead of one accumulation per direction and moment.
template <typename R> struct LatMoments {
    R rho, m[3], d[3], o[3];  // o: xy, xz, yz
};
template <typename R> __device__ __forceinline__ R o_of(const LatMoments<R> &M, int c, int q) {
    // symmetric second moment e_c e_q for c != q
    return (c + q == 1) ? M.o[0] : ((c + q == 2) ? M.o[1] : M.o[2]);
}

// Interface equilibrium, BGK relaxation towards the lattice populations and
// the flux through the face: calculate_flux_at_interface (LBFS.cu:1462-1648)
// and its axis-aligned forms (LBFS.cu:3648-4092).  The relaxed populations are
// f_k - tau (f_k - fl_k), f_k the interface equilibrium, so the flux tensor is
// (1 - tau) F_eq + tau F_fl, F_fl the moments of the lattice populations fl_k.
// The D3Q15 weights make the equilibrium moments exact closed forms
// (sum w e = 0, sum w e e = I / 3, sum w e e e e = (dd + dd + dd) / 9):
//   sum_k e_c f_k = rho u_c = m_c,  sum_k e_c e_q f_k = q_s m_c m_q / rho + d_cq rho' / 3
// (q_s the preconditioning factor; in the deviation form the d_cq term is
// rho' / 3).  So the mass flux is m . n exactly, and the momentum flux is
// formed from the six distinct second moments.  The reference sums the 15
// equilibria explicitly; the closed form is the same quantity with fewer
// roundings.  `axis` >= 0: only the face-normal component (axis-aligned faces,
// n = e_axis); `axis` < 0: all three with the face normal.
template <typename R>
__device__ __forceinline__ Vec4<R> interface_flux(const LatMoments<R> &M, R rho0, R tau, R qscale, R area, int axis,
                                                  R nx, R ny, R nz) {
    const R rho_i = M.rho + rho0;
    const R inv = R(1) / rho_i;
    const R keep = R(1) - tau;
    const R third = M.rho * R(1.0 / 3.0);
    // relaxed second moment c, q
    auto T = [&](int c, int q) -> R {
        R eq = qscale * (M.m[c] * inv) * M.m[q];
        R fl;
        if (c == q) {
            eq = eq + third;
            fl = M.d[c];
        } else {
            fl = o_of(M, c, q);
        }
        return keep * eq + tau * fl;
    };
    Vec4<R> out;
    if (axis >= 0) {
        out.rho = M.m[axis] * area;
        out.u = T(axis, 0) * area;
        out.v = T(axis, 1) * area;
        out.w = T(axis, 2) * area;
    } else {
        const R Txx = T(0, 0), Tyy = T(1, 1), Tzz = T(2, 2), Txy = T(0, 1), Txz = T(0, 2), Tyz = T(1, 2);
        out.rho = (M.m[0] * nx + M.m[1] * ny + M.m[2] * nz) * area;
        out.u = (Txx * nx + Txy * ny + Txz * nz) * area;
        out.v = (Txy * nx + Tyy * ny + Tyz * nz) * area;
        out.w = (Txz * nx + Tyz * ny + Tzz * nz) * area;
    }
    return out;
}

struct Dir {
    int ex, ey, ez;
};
__device__ __forceinline__ Dir dir_of(int k) { return {c_ex(k), c_ey(k), c_ez(k)}; }

template <typename R> __device__ __forceinline__ void load_grad(const R *g, R (&o)[12]) {
    const GradRec<R> r = *reinterpret_cast<const GradRec<R> *>(g);
#pragma unroll
    for (int t = 0; t < 12; t++) o[t] = r.g[t];
}

// The five directions of one side of a face: e_A = s (s = SGN: +1 owner side, -1
// neighbour side) with (e_B, e_C) in {(0,0), (+,+), (+,-), (-,+), (-,-)} (B < C the
// other two axes).  populate_lattice_macros_uniform_{x,y,z} (LBFS.cu:2939-3644): the
// lattice node sits at x_f - e dt and is extrapolated from the side's cell, L =
// a - e_B b - e_C c with a the state at the node of direction s e_A and b, c the
// gradients along B and C times dt.  With
//   e.u  = al + e_B be + e_C ga + e_B e_C de,
//   |u|^2 = (aa + bb + cc) - 2 e_B ab - 2 e_C ac + 2 e_B e_C bc,
// the population over its weight g = rho (1 + X), X = 3 e.u + q (4.5 (e.u)^2 -
// 1.5 |u|^2), has X = X0 + e_B XB + e_C XC + e_B e_C XBC, and the sums over the
// four corners are products of these four with rho's three terms: about two thirds
// of the operations of the five nodes one by one (57x45x33 FP32: 22.0 us a step, 20.9 with it).  Returned: a quarter of each sum,
// S = sum g, YB = sum e_B g, YC = sum e_C g, Z = sum e_B e_C g, and ga0 = g of
// direction s e_A alone.  FP32 (rho the deviation from rho0): the term 3 rho0 e.p0
// of the face centre's velocity is left out as in pop_dev and added once by the
// caller; ad = a - p0 there.
template <typename R> struct LatticeSide {
    R S, YB, YC, Z, ga0;
};
template <typename R, int A, int SGN, bool WITH_Z>
__device__ __forceinline__ LatticeSide<R> lattice_side(const R (&a)[4], const R (&b)[4], const R (&c)[4],
                                                    const R (&ad)[4], R rho0, R q) {
    constexpr int B = A == 0 ? 1 : 0, C = A == 2 ? 1 : 2;
    constexpr R s = R(SGN);
    const R bc_ = b[1 + B] + c[1 + C];
    const R al = s * a[1 + A] - bc_;
    const R be = a[1 + B] - s * b[1 + A], ga = a[1 + C] - s * c[1 + A];
    const R de = -(b[1 + C] + c[1 + B]);
    const R aa = a[1] * a[1] + a[2] * a[2] + a[3] * a[3];
    const R nn = aa + (b[1] * b[1] + b[2] * b[2] + b[3] * b[3]) + (c[1] * c[1] + c[2] * c[2] + c[3] * c[3]);
    const R ab = a[1] * b[1] + a[2] * b[2] + a[3] * b[3];
    const R ac = a[1] * c[1] + a[2] * c[2] + a[3] * c[3];
    const R bc = b[1] * c[1] + b[2] * c[2] + b[3] * c[3];
    const R k45 = R(4.5) * q, k15 = R(1.5) * q, k9 = R(9) * q, k3 = R(3) * q;
    const R E0 = k45 * (al * al + be * be + ga * ga + de * de) - k15 * nn;
    const R EB = k9 * (al * be + ga * de) + k3 * ab;
    const R EC = k9 * (al * ga + be * de) + k3 * ac;
    const R X0 = R(3) * al + E0, XB = R(3) * be + EB, XC = R(3) * ga + EC;
    const R XBC = R(3) * de + (k9 * (al * de + be * ga) - k3 * bc);
    const R Ea = k45 * (a[1 + A] * a[1 + A]) - k15 * aa;
    const R Xa = R(3) * (s * a[1 + A]) + Ea;
    LatticeSide<R> r;
    r.Z = R(0);
    if constexpr (sizeof(R) == 8) {
        const R q0 = R(1) + X0;
        r.S = a[0] * q0 - b[0] * XB - c[0] * XC;
        r.YB = a[0] * XB - b[0] * q0 - c[0] * XBC;
        r.YC = a[0] * XC - c[0] * q0 - b[0] * XBC;
        if constexpr (WITH_Z) r.Z = a[0] * XBC - b[0] * XC - c[0] * XB;
        r.ga0 = a[0] + a[0] * Xa;
    } else {
        const R ald = s * ad[1 + A] - bc_, bed = ad[1 + B] - s * b[1 + A], gad = ad[1 + C] - s * c[1 + A];
        r.S = a[0] + (a[0] * X0 - b[0] * XB - c[0] * XC + rho0 * (R(3) * ald + E0));
        r.YB = (a[0] * XB - b[0] * X0 - c[0] * XBC + rho0 * (R(3) * bed + EB)) - b[0];
        r.YC = (a[0] * XC - c[0] * X0 - b[0] * XBC + rho0 * (R(3) * gad + EC)) - c[0];
        if constexpr (WITH_Z) r.Z = a[0] * XBC - b[0] * XC - c[0] * XB + rho0 * XBC;
        r.ga0 = a[0] + (a[0] * Xa + rho0 * (R(3) * (s * ad[1 + A]) + Ea));
    }
    return r;
}

// Half the sum and half the difference of the populations (over their weight)
// of the opposite directions +-e_X at a face centre p with displacement b (L =
// p -+ b); pp = |p|^2.  FP32: in the deviation form.
template <typename R, int X>
__device__ __forceinline__ void centre_pair(const R (&p)[4], const R (&b)[4], R pp, R rho0, R &sum, R &dif) {
    const R bb = b[1] * b[1] + b[2] * b[2] + b[3] * b[3];
    const R pb = p[1] * b[1] + p[2] * b[2] + p[3] * b[3];
    const R px = p[1 + X], bx = b[1 + X];
    const R even = R(4.5) * (px * px + bx * bx) - R(1.5) * (pp + bb) - R(3) * bx;
    const R odd2 = R(3) * pb - R(9) * (px * bx);
    const R odd = odd2 + R(3) * px;
    if constexpr (sizeof(R) == 8) {
        const R q0 = R(1) + even;
        sum = p[0] * q0 - b[0] * odd;
        dif = p[0] * odd - b[0] * q0;
    } else {
        sum = p[0] + (p[0] * even - b[0] * odd + rho0 * even);
        dif = (p[0] * odd - b[0] * even + rho0 * odd2) - b[0];
    }
}

template <typename R> __device__ __forceinline__ R one_pop(const R (&L)[4], R eu, R edu, R rho0, R q) {
    if constexpr (sizeof(R) == 8) return pop_g<R>(L, eu, rho0, q);
    else return pop_dev(L, eu, edu, rho0, q);
}

// Axis-aligned interior face of axis A (calc_face_flux_x/_y/_z, LBFS.cu:2283-2569):
// directions with e_A = +1 extrapolate from the owner, -1 from the neighbour,
// 0 from the face centre with the distance-weighted gradient.
template <typename R, int A>
__device__ __forceinline__ Vec4<R> axis_face_flux(const FluidArgs<R> &a, int f) {
    constexpr int B = A == 0 ? 1 : 0, C = A == 2 ? 1 : 2;
    const int2 oc = __ldg(a.face_cells + f);
    AxisFace<R> geo;
    R wa, wb;
    if (a.axis_uniform) {
        geo = {a.axis_geo[A][0], a.axis_geo[A][1], a.axis_geo[A][2], a.axis_geo[A][3]};
        wa = a.axis_wa[A];
        wb = a.axis_wb[A];
    } else {
        geo = a.axis_face[f];
        const R ic = R(1) / (geo.t2 - geo.t1);
        wa = fabs(geo.t2 * ic);
        wb = fabs(geo.t1 * ic);
    }
    const Vec4<R> s1 = a.state[oc.x], s2 = a.state[oc.y];
    R g1[12], g2[12];
    load_grad(a.grad + (size_t)12 * oc.x, g1);
    load_grad(a.grad + (size_t)12 * oc.y, g2);
    const R rho0 = rho0_of(a);
    const R dt = geo.dt, t1 = geo.t1, t2 = geo.t2;
    const R S1[4] = {s1.rho, s1.u, s1.v, s1.w}, S2[4] = {s2.rho, s2.u, s2.v, s2.w};
    R pi[4], pn[4], p0[4];
#pragma unroll
    for (int m = 0; m < 4; m++) {
        pi[m] = S1[m] - t1 * g1[3 * m + A];
        pn[m] = S2[m] - t2 * g2[3 * m + A];
        p0[m] = (pi[m] + pn[m]) * R(0.5);
    }
    R a1[4], a2[4], b1[4], c1[4], b2[4], c2[4];
    R ad1[4] = {R(0), R(0), R(0), R(0)}, ad2[4] = {R(0), R(0), R(0), R(0)};
#pragma unroll
    for (int m = 0; m < 4; m++) {
        b1[m] = dt * g1[3 * m + B]; c1[m] = dt * g1[3 * m + C];
        b2[m] = dt * g2[3 * m + B]; c2[m] = dt * g2[3 * m + C];
        if constexpr (sizeof(R) == 8) {
            a1[m] = pi[m] - dt * g1[3 * m + A];
            a2[m] = pn[m] + dt * g2[3 * m + A];
        } else {
            // half the owner-neighbour difference, from the states' difference (exact for close values)
            const R hdp = ((S1[m] - S2[m]) - (t1 * g1[3 * m + A] - t2 * g2[3 * m + A])) * R(0.5);
            ad1[m] = hdp - dt * g1[3 * m + A];
            ad2[m] = dt * g2[3 * m + A] - hdp;
            a1[m] = p0[m] + ad1[m];
            a2[m] = p0[m] + ad2[m];
        }
    }
    const LatticeSide<R> o = lattice_side<R, A, 1, false>(a1, b1, c1, ad1, rho0, R(1));
    const LatticeSide<R> n = lattice_side<R, A, -1, false>(a2, b2, c2, ad2, rho0, R(1));
    // centre directions (e_A = 0): rest, +-B, +-C, from p0 with the distance-weighted gradient
    R bv[4], cv[4];
#pragma unroll
    for (int m = 0; m < 4; m++) {
        bv[m] = b1[m] * wa + b2[m] * wb;
        cv[m] = c1[m] * wa + c2[m] * wb;
    }
    const R pp = p0[1] * p0[1] + p0[2] * p0[2] + p0[3] * p0[3];
    const R gz0 = p0[0] + (p0[0] + rho0) * (R(-1.5) * pp);
    R sB, dB, sC, dC;
    centre_pair<R, B>(p0, bv, pp, rho0, sB, dB);
    centre_pair<R, C>(p0, cv, pp, rho0, sC, dC);
    // weights 2/9, 1/9 and 1/72; the sides' sums are quarters, the pairs' halves
    constexpr R w0 = R(2.0 / 9.0), w1 = R(1.0 / 9.0), w2 = R(1.0 / 18.0);
    const R So = w1 * o.ga0 + w2 * o.S, Sn = w1 * n.ga0 + w2 * n.S;
    LatMoments<R> M;
    M.rho = (So + Sn) + w0 * (gz0 + (sB + sC));
    M.m[A] = So - Sn;
    M.d[A] = So + Sn;
    M.m[B] = w2 * (o.YB + n.YB) + w0 * dB;
    M.m[C] = w2 * (o.YC + n.YC) + w0 * dC;
    M.o[A + B - 1] = w2 * (o.YB - n.YB);  // o index of the pair (A, B): xy 0, xz 1, yz 2
    M.o[A + C - 1] = w2 * (o.YC - n.YC);
    M.d[B] = M.d[C] = M.o[B + C - 1] = R(0);  // not read by the axis-A flux
    if constexpr (sizeof(R) == 4) {
        // first moments of the left-out term 3 rho0 e.p0_u (pop_dev)
#pragma unroll
        for (int c = 0; c < 3; c++) M.m[c] = M.m[c] + rho0 * p0[1 + c];
    }
    const R vf = a.visc_factor[oc.x];
    const R tau = (a.testcase == 8) ? R(0) : (a.visc * vf * R(3) / dt * a.gamma_inv);
    return interface_flux<R>(M, rho0, tau, R(1), geo.area, A, 0, 0, 0);
}

// General face: populate_lattice_macros (LBFS.cu:323-936).  Boundary faces
// take the boundary branch except the face of the first ghost (LBFS.cu tests
// neighbour > n_cells), which the host marks per instance in bc_branch.
// Ghost of boundary face f (ghost cell g = its neighbour): its state
// (update_unstructured_bcs, LBFS.cu:1843-1928) and its gradients
// (get_bc_gradients, LBFS.cu:1933-2048): Dirichlet components the difference
// to the owner over the owner-ghost distance along that direction, the others
// the owner's gradient without its face-normal part; a periodic component
// (type 3) the partner cell's gradient gp (gradients::Get_LS_Gradients,
// gradients.cpp:428-440).
template <typename R>
__device__ __forceinline__ void boundary_ghost(const FluidArgs<R> &a, int b, const Vec4<R> &own, const R (&go)[12],
                                               const R (&gp)[12], Vec4<R> &gs, R (&gg)[12]) {
    gs = ghost_state(a, b, own);
    const BcRec<R> r = a.bc_rec[b];
    const int rt = a.bc_rho_type[b], vt = a.bc_vel_type[b];
    const R d[4] = {gs.rho - own.rho, gs.u - own.u, gs.v - own.v, gs.w - own.w};
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const bool dirichlet = (m == 0) ? rt == 1 : (vt != 2 && vt != 3);
        if (dirichlet) {
            gg[3 * m + 0] = d[m] / r.dmag * r.dnx;
            gg[3 * m + 1] = d[m] / r.dmag * r.dny;
            gg[3 * m + 2] = d[m] / r.dmag * r.dnz;
        } else {
            gg[3 * m + 0] = go[3 * m + 0] * r.mx;
            gg[3 * m + 1] = go[3 * m + 1] * r.my;
            gg[3 * m + 2] = go[3 * m + 2] * r.mz;
        }
    }
    if (rt == 3 || vt == 3) {
#pragma unroll
        for (int t = 0; t < 12; t++)
            if ((t < 3) ? rt == 3 : vt == 3) gg[t] = gp[t];
    }
}

// Flux through a general face with owner state s1 and gradients g1, neighbour
// (or ghost) state s2 and gradients g2; b: its boundary index where geo.bc_branch
// is set, vf the viscosity factor.
template <typename R>
__device__ __forceinline__ Vec4<R> general_flux(const FluidArgs<R> &a, const GenFace<R> &geo, const Vec4<R> &s1,
                                                const Vec4<R> &s2, R (&g1)[12], const R (&g2)[12], int b, R vf) {
    const R rho0 = rho0_of(a);
    const R dt = geo.dt;
    const R S1[4] = {s1.rho, s1.u, s1.v, s1.w}, S2[4] = {s2.rho, s2.u, s2.v, s2.w};
    R pi[4], pn[4], p0[4];
    if (geo.bc_branch != R(0)) {
        const Vec4<R> bc = a.bc_val[b];
        const bool rd = a.bc_rho_type[b] == 1, vd = a.bc_vel_type[b] == 1;
        const R bcv[4] = {bc.rho, bc.u, bc.v, bc.w};
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const bool dir = (m == 0) ? rd : vd;
            p0[m] = dir ? bcv[m]
                        : S1[m] - (geo.t1x * g2[3 * m] + geo.t1y * g2[3 * m + 1] + geo.t1z * g2[3 * m + 2]);
            pi[m] = p0[m];
            pn[m] = p0[m];
        }
#pragma unroll
        for (int t = 0; t < 12; t++) g1[t] = g2[t];
    } else {
#pragma unroll
        for (int m = 0; m < 4; m++) {
            pi[m] = S1[m] - (geo.t1x * g1[3 * m] + geo.t1y * g1[3 * m + 1] + geo.t1z * g1[3 * m + 2]);
            pn[m] = S2[m] - (geo.t2x * g2[3 * m] + geo.t2y * g2[3 * m + 1] + geo.t2z * g2[3 * m + 2]);
            p0[m] = (pi[m] + pn[m]) * R(0.5);
        }
    }
    // FP32 deviation form: offsets from the face centre (pop_dev); hdp is half
    // the owner-neighbour difference of the reconstructed states
    R hdp[4] = {R(0), R(0), R(0), R(0)};
    if constexpr (sizeof(R) == 4) {
        if (geo.bc_branch == R(0)) {
#pragma unroll
            for (int m = 0; m < 4; m++)
                hdp[m] = ((S1[m] - S2[m]) - ((geo.t1x * g1[3 * m] + geo.t1y * g1[3 * m + 1] + geo.t1z * g1[3 * m + 2]) -
                                             (geo.t2x * g2[3 * m] + geo.t2y * g2[3 * m + 1] + geo.t2z * g2[3 * m + 2]))) *
                         R(0.5);
        }
    }
    // Upwind selection by the sign of n.e_k with the threshold 0.001 dt
    // (LBFS.cu:351-352 override the sin(pi/14) arguments).  Directions come in
    // opposite pairs (k, k + 1): sum and difference of the pair's populations
    // feed the moments.
    const R thr = R(0.001) * dt;
    const R q = a.recon_q;
    R g0;
    if constexpr (sizeof(R) == 4) g0 = pop_dev(p0, R(0), R(0), rho0, q);
    else g0 = pop_g<R>(p0, R(0), rho0, q);
    R sax[3], dax[3];          // axis pairs (+e_c, -e_c): sum and difference
    R sc, mcor[3], ocor[3];    // corner pairs: sum of sums; sum of e_c x difference; of e_c e_q x sum
#pragma unroll
    for (int k = 1; k < 15; k += 2) {
        const Dir e = dir_of(k);  // odd k: e_k; k + 1: -e_k
        const int ee[3] = {e.ex, e.ey, e.ez};
        const R s = (k < 7) ? (e.ex ? geo.nx : (e.ey ? geo.ny : geo.nz))
                            : (R(e.ex) * geo.nx + R(e.ey) * geo.ny + R(e.ez) * geo.nz);
        // Upwind sides.  With sg = -1 where n.e < -thr and +1 otherwise, the population of
        // direction sg e comes from the owner and that of -sg e from the neighbour, each
        // extrapolated along its own direction: Lo = p_owner - sg dt (e . g_owner),
        // Ln = p_neighbour + sg dt (e . g_neighbour).  Where |n.e| <= thr (cen) both come from
        // the face centre with the mean gradient C (sg = +1: +e at Lo, -e at Ln).  Only warps
        // with such a lane take the selects; in the others the side is a sign of dt.
        const bool neg = s < -thr, cen = !(s > thr) && !neg;
        const R sg = neg ? R(-1) : R(1);
        const R sdt = sg * dt;
        R A[4], B[4];  // e . gradient per component, owner (A) and neighbour (B)
#pragma unroll
        for (int m = 0; m < 4; m++) {
            bool first = true;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                if (!ee[d]) continue;
                const R ga = ee[d] > 0 ? g1[3 * m + d] : -g1[3 * m + d];
                const R gb = ee[d] > 0 ? g2[3 * m + d] : -g2[3 * m + d];
                A[m] = first ? ga : A[m] + ga;
                B[m] = first ? gb : B[m] + gb;
                first = false;
            }
        }
        R Lo[4], Ln[4], Do[4], Dn[4];
        if (__any_sync(__activemask(), cen)) {
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const R C = (A[m] + B[m]) * R(0.5);
                const R Xo = cen ? C : A[m], Xn = cen ? C : B[m];
                if constexpr (sizeof(R) == 8) {
                    Lo[m] = (cen ? p0[m] : pi[m]) - sdt * Xo;
                    Ln[m] = (cen ? p0[m] : pn[m]) + sdt * Xn;
                } else {
                    // FP32: offsets from the face centre (+hdp owner, -hdp neighbour, 0 centre)
                    Do[m] = (cen ? R(0) : hdp[m]) - sdt * Xo;
                    Dn[m] = (cen ? R(0) : -hdp[m]) + sdt * Xn;
                    Lo[m] = p0[m] + Do[m];
                    Ln[m] = p0[m] + Dn[m];
                }
            }
        } else {
#pragma unroll
            for (int m = 0; m < 4; m++) {
                if constexpr (sizeof(R) == 8) {
                    Lo[m] = pi[m] - sdt * A[m];
                    Ln[m] = pn[m] + sdt * B[m];
                } else {
                    Do[m] = hdp[m] - sdt * A[m];
                    Dn[m] = -hdp[m] + sdt * B[m];
                    Lo[m] = p0[m] + Do[m];
                    Ln[m] = p0[m] + Dn[m];
                }
            }
        }
        // e . u at both states (and e . d, FP32); the owner's direction is sg e, the neighbour's -sg e
        R Eo, En, Edo = R(0), Edn = R(0);
        {
            bool first = true;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                if (!ee[d]) continue;
                const R uo = ee[d] > 0 ? Lo[1 + d] : -Lo[1 + d], un = ee[d] > 0 ? Ln[1 + d] : -Ln[1 + d];
                Eo = first ? uo : Eo + uo;
                En = first ? un : En + un;
                if constexpr (sizeof(R) == 4) {
                    const R dO = ee[d] > 0 ? Do[1 + d] : -Do[1 + d], dN = ee[d] > 0 ? Dn[1 + d] : -Dn[1 + d];
                    Edo = first ? dO : Edo + dO;
                    Edn = first ? dN : Edn + dN;
                }
                first = false;
            }
        }
        R go, gn;
        if constexpr (sizeof(R) == 4) {
            go = pop_dev(Lo, sg * Eo, sg * Edo, rho0, q);
            gn = pop_dev(Ln, -sg * En, -sg * Edn, rho0, q);
        } else {
            go = pop_g<R>(Lo, sg * Eo, rho0, q);
            gn = pop_g<R>(Ln, -sg * En, rho0, q);
        }
        // the pair's sum and its (+e) - (-e) difference
        const R sig = go + gn, del = sg * (go - gn);
        if (k < 7) {
            const int c = e.ex ? 0 : (e.ey ? 1 : 2);
            sax[c] = sig;
            dax[c] = del;
        } else if (k == 7) {  // (+,+,+): first corner pair
            sc = sig;
#pragma unroll
            for (int d = 0; d < 3; d++) { mcor[d] = del; ocor[d] = sig; }
        } else {
            sc = sc + sig;
#pragma unroll
            for (int d = 0; d < 3; d++) mcor[d] = (ee[d] > 0) ? mcor[d] + del : mcor[d] - del;
            ocor[0] = (ee[0] * ee[1] > 0) ? ocor[0] + sig : ocor[0] - sig;
            ocor[1] = (ee[0] * ee[2] > 0) ? ocor[1] + sig : ocor[1] - sig;
            ocor[2] = (ee[1] * ee[2] > 0) ? ocor[2] + sig : ocor[2] - sig;
        }
    }
    constexpr R w_rest = R(2.0 / 9.0), w_axis = R(1.0 / 9.0), w_corner = R(1.0 / 72.0);
    LatMoments<R> M;
    M.rho = w_rest * g0 + w_axis * ((sax[0] + sax[1]) + sax[2]) + w_corner * sc;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        M.m[c] = w_axis * dax[c] + w_corner * mcor[c];
        M.d[c] = w_axis * sax[c] + w_corner * sc;
        M.o[c] = w_corner * ocor[c];
        if constexpr (sizeof(R) == 4) M.m[c] = M.m[c] + rho0 * p0[1 + c];  // the term pop_dev leaves out
    }
    const R tau = (a.testcase == 8) ? R(0) : (a.visc * vf * R(3) / dt * a.gamma_inv);
    return interface_flux<R>(M, rho0, tau, a.gamma_inv, geo.area, -1, geo.nx, geo.ny, geo.nz);
}

// The same flux for an interior face whose normal lies within its axis' cone, n_A -
// |n_B| - |n_C| > 0.001 dt: every direction with e_A = +1 then comes from the owner
// and every one with e_A = -1 from the neighbour, so the two sides take the closed
// form of the axis-aligned faces and only the pairs +-e_B, +-e_C choose by n's signs
// (us per step without / with: 128.6 / 118.4 jittered at 72^3 FP64, 367 / 346 at 128^3 FP32).
template <typename R, int A>
__device__ __forceinline__ Vec4<R> cone_flux(const FluidArgs<R> &args, const GenFace<R> &geo, const Vec4<R> &s1,
                                             const Vec4<R> &s2, const R (&g1)[12], const R (&g2)[12], R vf) {
    constexpr int B = A == 0 ? 1 : 0, C = A == 2 ? 1 : 2;
    const R rho0 = rho0_of(args), q = args.recon_q, dt = geo.dt, thr = R(0.001) * dt;
    const R nv[3] = {geo.nx, geo.ny, geo.nz};
    const R S1[4] = {s1.rho, s1.u, s1.v, s1.w}, S2[4] = {s2.rho, s2.u, s2.v, s2.w};
    R p0[4], hd[4], a1[4], a2[4], b1[4], c1[4], b2[4], c2[4], pi[4], pn[4];
    R ad1[4] = {R(0), R(0), R(0), R(0)}, ad2[4] = {R(0), R(0), R(0), R(0)};
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const R r1 = geo.t1x * g1[3 * m] + geo.t1y * g1[3 * m + 1] + geo.t1z * g1[3 * m + 2];
        const R r2 = geo.t2x * g2[3 * m] + geo.t2y * g2[3 * m + 1] + geo.t2z * g2[3 * m + 2];
        pi[m] = S1[m] - r1;
        pn[m] = S2[m] - r2;
        p0[m] = (pi[m] + pn[m]) * R(0.5);
        hd[m] = R(0);
        const R gA1 = dt * g1[3 * m + A], gA2 = dt * g2[3 * m + A];
        b1[m] = dt * g1[3 * m + B]; c1[m] = dt * g1[3 * m + C];
        b2[m] = dt * g2[3 * m + B]; c2[m] = dt * g2[3 * m + C];
        if constexpr (sizeof(R) == 8) {
            a1[m] = pi[m] - gA1;
            a2[m] = pn[m] + gA2;
        } else {
            hd[m] = ((S1[m] - S2[m]) - (r1 - r2)) * R(0.5);
            ad1[m] = hd[m] - gA1;
            ad2[m] = gA2 - hd[m];
            a1[m] = p0[m] + ad1[m];
            a2[m] = p0[m] + ad2[m];
        }
    }
    const LatticeSide<R> o = lattice_side<R, A, 1, true>(a1, b1, c1, ad1, rho0, q);
    const LatticeSide<R> n = lattice_side<R, A, -1, true>(a2, b2, c2, ad2, rho0, q);
    // the pairs +-e_X, X = B, C: direction sg e_X from the owner, -sg e_X from the neighbour, or both from
    // the face centre with the mean gradient
    const unsigned lanes = __activemask();
    auto tangent = [&](const R(&x1)[4], const R(&x2)[4], R nx, int X, R &sig, R &del) {
        const bool neg = nx < -thr, cen = !(nx > thr) && !neg;
        const R sg = neg ? R(-1) : R(1);
        R Lo[4], Ln[4], Do[4] = {R(0), R(0), R(0), R(0)}, Dn[4] = {R(0), R(0), R(0), R(0)};
        const bool any = __any_sync(lanes, cen);
#pragma unroll
        for (int m = 0; m < 4; m++) {
            R xo = x1[m], xn = x2[m];
            if constexpr (sizeof(R) == 8) {
                R bo = pi[m], bn = pn[m];
                if (any) {
                    const R xm = (x1[m] + x2[m]) * R(0.5);
                    xo = cen ? xm : xo; xn = cen ? xm : xn;
                    bo = cen ? p0[m] : bo; bn = cen ? p0[m] : bn;
                }
                Lo[m] = bo - sg * xo;
                Ln[m] = bn + sg * xn;
            } else {
                R h = hd[m];
                if (any) {
                    const R xm = (x1[m] + x2[m]) * R(0.5);
                    xo = cen ? xm : xo; xn = cen ? xm : xn;
                    h = cen ? R(0) : h;
                }
                Do[m] = h - sg * xo;
                Dn[m] = sg * xn - h;
                Lo[m] = p0[m] + Do[m];
                Ln[m] = p0[m] + Dn[m];
            }
        }
        const R go = one_pop<R>(Lo, sg * Lo[1 + X], sg * Do[1 + X], rho0, q);
        const R gn = one_pop<R>(Ln, -sg * Ln[1 + X], -sg * Dn[1 + X], rho0, q);
        sig = go + gn;
        del = sg * (go - gn);
    };
    R sB, dB, sC, dC;
    tangent(b1, b2, nv[B], B, sB, dB);
    tangent(c1, c2, nv[C], C, sC, dC);
    const R x0 = R(-1.5) * q * (p0[1] * p0[1] + p0[2] * p0[2] + p0[3] * p0[3]);
    const R g0 = p0[0] + (p0[0] + rho0) * x0;
    constexpr R w0 = R(2.0 / 9.0), w1 = R(1.0 / 9.0), w2 = R(1.0 / 18.0);
    const R So = w1 * o.ga0 + w2 * o.S, Sn = w1 * n.ga0 + w2 * n.S, Sc = w2 * (o.S + n.S);
    LatMoments<R> M;
    M.rho = (So + Sn) + (w0 * g0 + w1 * (sB + sC));
    M.m[A] = So - Sn;
    M.d[A] = So + Sn;
    M.m[B] = w2 * (o.YB + n.YB) + w1 * dB;
    M.m[C] = w2 * (o.YC + n.YC) + w1 * dC;
    M.d[B] = Sc + w1 * sB;
    M.d[C] = Sc + w1 * sC;
    M.o[A + B - 1] = w2 * (o.YB - n.YB);
    M.o[A + C - 1] = w2 * (o.YC - n.YC);
    M.o[B + C - 1] = w2 * (o.Z + n.Z);
    if constexpr (sizeof(R) == 4) {
#pragma unroll
        for (int d = 0; d < 3; d++) M.m[d] = M.m[d] + rho0 * p0[1 + d];
    }
    const R tau = (args.testcase == 8) ? R(0) : (args.visc * vf * R(3) / dt * args.gamma_inv);
    return interface_flux<R>(M, rho0, tau, args.gamma_inv, geo.area, -1, nv[0], nv[1], nv[2]);
}

// CONE: the axis whose cone the (interior) face's normal lies in, -1: none is known.
template <typename R, int CONE>
__device__ __forceinline__ Vec4<R> general_face_flux(const FluidArgs<R> &a, int f, bool is_bc) {
    const int2 oc = __ldg(a.face_cells + f);
    const GenFace<R> geo = a.gen_face[a.axis_aligned ? f - a.ni : f];
    const Vec4<R> s1 = a.state[oc.x];
    Vec4<R> s2;
    R g1[12], g2[12];
    load_grad(a.grad + (size_t)12 * oc.x, g1);
    if (is_bc) {
        R gp[12];
        const int b = oc.y - a.nc;
        if (a.bc_rho_type[b] == 3 || a.bc_vel_type[b] == 3) load_grad(a.grad + (size_t)12 * a.bc_periodic[b], gp);
        boundary_ghost(a, b, s1, g1, gp, s2, g2);
        a.state[oc.y] = s2;
        GradRec<R> gr;
#pragma unroll
        for (int t = 0; t < 12; t++) gr.g[t] = g2[t];
        reinterpret_cast<GradRec<R> *>(a.grad)[oc.y] = gr;
    } else {
        s2 = a.state[oc.y];
        load_grad(a.grad + (size_t)12 * oc.y, g2);
        if constexpr (CONE >= 0) return cone_flux<R, CONE>(a, geo, s1, s2, g1, g2, a.visc_factor[oc.x]);
    }
    return general_flux<R>(a, geo, s1, s2, g1, g2, oc.y - a.nc, is_bc ? R(1) : a.visc_factor[oc.x]);
}

}  // namespace lbfs
