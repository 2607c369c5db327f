// Atomic-free element assembly (a3-a9). A block owns a tile of consecutive rows and computes each
// element that touches them once, into shared memory (elemtile.cuh); its threads then sum every
// CSR entry and right-hand side entry from there, in ascending element order, and write every value
// once, entries coalesced. Where that is not the better form (et_better) or a tile's elements do not fit
// (a node of very many elements), one thread per matrix row gathers the contributions of the row's
// elements from the sorted node -> element incidence, in the same order and with the same roundings:
// a mesh's bits do not depend on the form. Compared with the reference's one-thread-per-element kernels with FP64
// atomicAdd into a binary-searched CSR slot (src/cfa/fem_kernels.cuh:40-282, :697-909), there
// are no atomics and no searches, the result is deterministic, and each CSR value is written
// exactly once (coalesced along the row).
#include <mutex>

#include "internal.cuh"
#include "mesh.cuh"

namespace cfa {

struct Geom {
    double area, dNdx[3], dNdy[3];
    bool ok;
};

// Element geometry exactly as the reference kernels compute it (fem_kernels.cuh:77-87)
__device__ __forceinline__ Geom elem_geom(const int* nd, const double* __restrict__ x, const double* __restrict__ y) {
    Geom g;
    const double x0 = x[nd[0]], y0 = y[nd[0]], x1 = x[nd[1]], y1 = y[nd[1]], x2 = x[nd[2]], y2 = y[nd[2]];
    const double detJ = __fma_rn(x1 - x0, y2 - y0, -__dmul_rn(x2 - x0, y1 - y0));
    g.area = 0.5 * fabs(detJ);
    g.ok = !(g.area < 1.0e-14);
    const double inv2A = 1.0 / (2.0 * g.area);
    g.dNdx[0] = (y1 - y2) * inv2A; g.dNdx[1] = (y2 - y0) * inv2A; g.dNdx[2] = (y0 - y1) * inv2A;
    g.dNdy[0] = (x2 - x1) * inv2A; g.dNdy[1] = (x0 - x2) * inv2A; g.dNdy[2] = (x1 - x0) * inv2A;
    return g;
}

__device__ __forceinline__ void load_elem(const int* __restrict__ ev, int e, int* nd) {
    nd[0] = ev[3 * e]; nd[1] = ev[3 * e + 1]; nd[2] = ev[3 * e + 2];
}

struct MomParams {
    double dt, nu, rho, a0, a1, a2, c1, c2, tau_time, skew_coef;
};

// Dirichlet rows of the momentum system (k_apply_bc_momentum, fem_kernels.cuh:431-441)
__device__ __forceinline__ bool momentum_dirichlet(int tag, const OutletBc& bc) {
    return tag == BC_INLET || tag == BC_WALL || tag == BC_CYLINDER || (tag == BC_OUTLET && bc.outlet_dirichlet);
}
__device__ __forceinline__ double momentum_bc_u(int tag, double yi, double u_max, double H, const OutletBc& bc) {
    if (tag == BC_INLET || tag == BC_OUTLET)
        return 4.0 * u_max * yi * (H - yi) / (H * H) * (tag == BC_OUTLET ? bc.outlet_scale : 1.0);
    return 0.0;
}

// Element terms of the momentum system (fem_kernels.cuh:88-176). Every product that meets a sum is
// rounded explicitly: the two kernels below hold the same expressions in different surroundings, where
// the compiler would contract them differently, and a last digit of A moves a mixed-precision solve
// of some 500k vertices by up to 1e-8 (the ILU sweeps round their input to FP32).
struct MomElem {
    double area, area3, nu, tau, area_tau, area3_tau, skew_div, dpdx, dpdy;
    double u_h[3], v_h[3];
};
__device__ __forceinline__ MomElem momentum_element(const int* nd, const Geom& g, const double* __restrict__ u_old,
                                                    const double* __restrict__ v_old,
                                                    const double* __restrict__ u_prev,
                                                    const double* __restrict__ v_prev,
                                                    const double* __restrict__ p_old,
                                                    const double* __restrict__ nu_node, const MomParams& P,
                                                    double inv_rho, double term_t, double (&ugN)[3]) {
    // reciprocals of the constant and per-launch divisors, taken once (the products differ from
    // the quotients in the last bit at most; the element formula is division-bound in FP64)
    constexpr double kThird = 1.0 / 3.0;
    MomElem m;
    m.area = g.area;
    m.area3 = __dmul_rn(g.area, kThird);
    double w_u = 0.0, w_v = 0.0, div_w = 0.0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double un = u_old[nd[k]], vn = v_old[nd[k]], um = u_prev[nd[k]], vm = v_prev[nd[k]];
        m.u_h[k] = __fma_rn(P.a1, un, __dmul_rn(P.a2, um));
        m.v_h[k] = __fma_rn(P.a1, vn, __dmul_rn(P.a2, vm));
        const double wu = __fma_rn(P.c1, un, __dmul_rn(P.c2, um)), wv = __fma_rn(P.c1, vn, __dmul_rn(P.c2, vm));
        w_u = __fma_rn(wu, kThird, w_u);
        w_v = __fma_rn(wv, kThird, w_v);
        div_w = __dadd_rn(div_w, __fma_rn(wu, g.dNdx[k], __dmul_rn(wv, g.dNdy[k])));
    }
    const double vel_mag = sqrt(__fma_rn(w_u, w_u, __dmul_rn(w_v, w_v))) + 1.0e-12;
    const double h_K = sqrt(2.0 * g.area);
    // element viscosity: the scalar nu, or the mean of a nodal field
    m.nu = nu_node ? __dmul_rn(nu_node[nd[0]] + nu_node[nd[1]] + nu_node[nd[2]], kThird) : P.nu;
    const double term_c = 2.0 * vel_mag / h_K;
    const double term_d = 4.0 * m.nu / __dmul_rn(h_K, h_K);
    m.tau = 1.0 / sqrt(__fma_rn(__dmul_rn(9.0, term_d), term_d, __fma_rn(term_c, term_c, __dmul_rn(term_t, term_t))));
    m.area_tau = __dmul_rn(g.area, m.tau);
    m.area3_tau = __dmul_rn(m.area3, m.tau);
    m.skew_div = __dmul_rn(P.skew_coef, div_w);
    const double p0 = p_old[nd[0]], p1 = p_old[nd[1]], p2 = p_old[nd[2]];
    m.dpdx = __dmul_rn(__fma_rn(p2, g.dNdx[2], __fma_rn(p0, g.dNdx[0], __dmul_rn(p1, g.dNdx[1]))), inv_rho);
    m.dpdy = __dmul_rn(__fma_rn(p2, g.dNdy[2], __fma_rn(p0, g.dNdy[0], __dmul_rn(p1, g.dNdy[1]))), inv_rho);
#pragma unroll
    for (int k = 0; k < 3; ++k) ugN[k] = __fma_rn(w_u, g.dNdx[k], __dmul_rn(w_v, g.dNdy[k]));
    return m;
}
// A_aj of one element; f_u, f_v take its (M + Ms) u_h
__device__ __forceinline__ double momentum_entry(const MomElem& m, double dNdx_a, double dNdy_a, double ugN_a,
                                                 bool diag, int j, const Geom& g, double ugN_j, double a0,
                                                 double& f_u, double& f_v) {
    constexpr double kSixth = 1.0 / 6.0, kTwelfth = 1.0 / 12.0;
    const double M_ij = __dmul_rn(m.area, diag ? kSixth : kTwelfth);
    const double MM = __dadd_rn(M_ij, __dmul_rn(m.area3_tau, ugN_a));
    const double K_ij = __dmul_rn(m.area, __fma_rn(dNdx_a, g.dNdx[j], __dmul_rn(dNdy_a, g.dNdy[j])));
    const double C_ij = __fma_rn(m.skew_div, M_ij, __dmul_rn(m.area3, ugN_j));
    f_u = __fma_rn(MM, m.u_h[j], f_u);
    f_v = __fma_rn(MM, m.v_h[j], f_v);
    return __fma_rn(__dmul_rn(m.area_tau, ugN_a), ugN_j,
                    __dadd_rn(__fma_rn(m.nu, K_ij, __dmul_rn(a0, MM)), C_ij));
}
// the pressure gradient's share of f_u, f_v
__device__ __forceinline__ void momentum_pressure(const MomElem& m, double ugN_a, double& f_u, double& f_v) {
    const double tw = __dadd_rn(m.area3, __dmul_rn(m.area_tau, ugN_a));
    f_u = __fma_rn(-tw, m.dpdx, f_u);
    f_v = __fma_rn(-tw, m.dpdy, f_v);
}

// Momentum rows: k_assemble_momentum_fem (fem_kernels.cuh:40-181) gathered per row, lumped mass,
// and (with_bc) the Dirichlet rows of k_apply_bc_momentum (:411-453) on A and the RHS. A row of
// up to kMomCap entries accumulates in shared memory laid out [slot][thread] (conflict-free for
// any slot a thread adds to); longer rows in place in global memory. Same addition order.
constexpr int kMomCap = 16;
constexpr size_t kMomSmem = (size_t)kMomCap * kThreads * sizeof(double);

__global__ void __launch_bounds__(kThreads)
k_momentum_rows(int n, const int* __restrict__ ev, const double* __restrict__ x, const double* __restrict__ y,
                const int* __restrict__ tag, const int* __restrict__ inc_ptr, const int* __restrict__ inc,
                const int* __restrict__ pos, const int* __restrict__ rp, const int* __restrict__ ci,
                const double* __restrict__ u_old, const double* __restrict__ v_old,
                const double* __restrict__ u_prev, const double* __restrict__ v_prev,
                const double* __restrict__ p_old, const double* __restrict__ nu_node, MomParams P, int with_bc,
                double u_max, double H, OutletBc bc, double* __restrict__ A_val, double* __restrict__ rhs_u,
                double* __restrict__ rhs_v, double* __restrict__ mass) {
    CFA_GRID_DEP();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int r0 = rp[i], len = rp[i + 1] - r0;
    const bool dir = with_bc && momentum_dirichlet(tag[i], bc);
    const bool local = len <= kMomCap;
    extern __shared__ double mom_sm[];   // [kMomCap][blockDim.x]
    const int T = blockDim.x;
    double* acc = mom_sm + threadIdx.x;  // acc[q * T]: entry q of this row
    if (!dir) {
        if (local) {
            for (int q = 0; q < len; ++q) acc[q * T] = 0.0;
        } else {
            for (int q = 0; q < len; ++q) A_val[r0 + q] = 0.0;
        }
    }
    double f_u_row = 0.0, f_v_row = 0.0, m_row = 0.0;
    const double inv_rho = 1.0 / P.rho, term_t = 2.0 / P.tau_time;
    for (int s = inc_ptr[i]; s < inc_ptr[i + 1]; ++s) {
        const int e = inc[s] >> 2, a = inc[s] & 3;
        int nd[3];
        load_elem(ev, e, nd);
        const Geom g = elem_geom(nd, x, y);
        if (!g.ok) continue;
        m_row = __dadd_rn(m_row, __dmul_rn(g.area, 1.0 / 3.0));
        if (dir) continue;
        double ugN[3];
        const MomElem m =
            momentum_element(nd, g, u_old, v_old, u_prev, v_prev, p_old, nu_node, P, inv_rho, term_t, ugN);
        double f_u = 0.0, f_v = 0.0;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double A_ij = momentum_entry(m, g.dNdx[a], g.dNdy[a], ugN[a], a == j, j, g, ugN[j], P.a0, f_u, f_v);
            const int p = pos[3 * s + j];
            if (local) acc[(p - r0) * T] += A_ij; else A_val[p] += A_ij;
        }
        momentum_pressure(m, ugN[a], f_u, f_v);
        f_u_row += f_u;
        f_v_row += f_v;
    }
    mass[i] = m_row;
    if (dir) {
        const int t = tag[i];
        const double ub = momentum_bc_u(t, y[i], u_max, H, bc);
        for (int q = 0; q < len; ++q) A_val[r0 + q] = (ci[r0 + q] == i) ? 1.0 : 0.0;
        rhs_u[i] = ub;
        rhs_v[i] = 0.0;
        return;
    }
    if (local)
        for (int q = 0; q < len; ++q) A_val[r0 + q] = acc[q * T];
    rhs_u[i] = f_u_row;
    rhs_v[i] = f_v_row;
}

// Momentum rows on element tiles: the element matrix and right-hand side of every element of the
// tile (16 doubles an element: A_ab, f_u, f_v, area / 3), then the entries, the rows and the
// Dirichlet rows. Bound by latency: each block's chain of plan, vertices and fields, the divisions
// and square roots of the element formula, then the entries' codes (issue 28%, DRAM 7%, LSU 32% busy at
// 402k vertices). Gathers -> tiles, the L2 flushed first: 149 -> 144 us at 402k vertices (77 MB of DRAM),
// 29.7 -> 20.0 us at 22k, 27.7 -> 19.5 us at 7k.
// Three blocks per SM (80 registers) matter: at 92 registers, two blocks, 189 against 144 us at 402k
// vertices, each with the L2 flushed first. A wave of tiles (3 x 148 of 96 rows) takes some 14 us, one of
// gathers (2 x 148 of 256 rows) some 24, so tiles run up to 5/3 of the gathers' waves. Tiles / gathers in
// us: 37k vertices 26 / 28, 56k 36 / 34, 76k 38 / 45, 113k 50 / 57, 135k 61 / 58, 156k 65 / 73, 317k
// 118 / 123, 402k 144 / 149, 642k 220 / 221, 1.3M 427 / 419, 4.2M 1350 / 1317. A tile of some 260
// elements is usual, one of 576 shares none: 402k vertices with 1% of them appended in random order
// 204 / 159, 76k with 5% 55 / 54; a 22k mesh of 64-row tiles 24 / 36.
constexpr EtForm kMomForm = {3, 2, 5, 3, 5 * kEtRows};
__global__ void __launch_bounds__(kEtThreads, 3)
k_momentum_tiles(ElemTileView tv, int n, const int* __restrict__ ev, const double* __restrict__ x,
                 const double* __restrict__ y, const int* __restrict__ tag, const int* __restrict__ rp,
                 const int* __restrict__ ci, const double* __restrict__ u_old, const double* __restrict__ v_old,
                 const double* __restrict__ u_prev, const double* __restrict__ v_prev,
                 const double* __restrict__ p_old, const double* __restrict__ nu_node, MomParams P, int with_bc,
                 double u_max, double H, OutletBc bc, double* __restrict__ A_val, double* __restrict__ rhs_u,
                 double* __restrict__ rhs_v, double* __restrict__ mass) {
    extern __shared__ __align__(16) double et_rec[];   // [16][tv.stride]
    const EtBlock b = et_block(tv, n);
    const int S = tv.stride;
    CFA_GRID_DEP();
    const double inv_rho = 1.0 / P.rho, term_t = 2.0 / P.tau_time;
    for (int le = threadIdx.x; le < b.ne; le += kEtThreads) {
        int nd[3];
        load_elem(ev, tv.elems[b.i0 + le], nd);
        const Geom g = elem_geom(nd, x, y);
        double* rec = et_rec + le;
        if (!g.ok) {
#pragma unroll
            for (int q = 0; q < 16; ++q) rec[q * S] = 0.0;
            continue;
        }
        double ugN[3];
        const MomElem m =
            momentum_element(nd, g, u_old, v_old, u_prev, v_prev, p_old, nu_node, P, inv_rho, term_t, ugN);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            double f_u = 0.0, f_v = 0.0;
#pragma unroll
            for (int j = 0; j < 3; ++j)
                rec[(3 * a + j) * S] =
                    momentum_entry(m, g.dNdx[a], g.dNdy[a], ugN[a], a == j, j, g, ugN[j], P.a0, f_u, f_v);
            momentum_pressure(m, ugN[a], f_u, f_v);
            rec[(9 + a) * S] = f_u;
            rec[(12 + a) * S] = f_v;
        }
        rec[15 * S] = m.area3;
    }
    __syncthreads();
    const int p0 = rp[b.r0], p1 = rp[b.r1];
    const unsigned short* code = tv.ecode + 3 * (size_t)b.i0;
    auto entry = [&](int p, int c0, int c1) {
        double v = 0.0;
        for (int c = c0; c < c1; ++c) {
            const int q = code[c];
            v += et_rec[(3 * ((q >> 2) & 3) + (q & 3)) * S + (q >> 4)];
        }
        A_val[p] = v;
    };
    for (int p = p0 + threadIdx.x; p < p1; p += kEtThreads)
        entry(p, tv.eoff[p], p + 1 < p1 ? (int)tv.eoff[p + 1] : 3 * (b.i1 - b.i0));
    if (with_bc) __syncthreads();   // the Dirichlet rows below follow the entries' values
    for (int i = b.r0 + threadIdx.x; i < b.r1; i += kEtThreads) {
        double f_u = 0.0, f_v = 0.0, m = 0.0;
        for (int s = tv.inc_ptr[i]; s < tv.inc_ptr[i + 1]; ++s) {
            const int q = tv.rcode[s], le = q >> 2, a = q & 3;
            f_u += et_rec[(9 + a) * S + le];
            f_v += et_rec[(12 + a) * S + le];
            m += et_rec[15 * S + le];
        }
        mass[i] = m;
        const int t = tag[i];
        if (with_bc && momentum_dirichlet(t, bc)) {
            for (int q = rp[i]; q < rp[i + 1]; ++q) A_val[q] = (ci[q] == i) ? 1.0 : 0.0;
            f_u = momentum_bc_u(t, y[i], u_max, H, bc);
            f_v = 0.0;
        }
        rhs_u[i] = f_u;
        rhs_v[i] = f_v;
    }
}

// Dirichlet rows of the momentum system alone (k_apply_bc_momentum, fem_kernels.cuh:411-453);
// rows_too writes the A rows and RHS as well, otherwise only the solution values.
__global__ void k_momentum_bc(int n, const int* __restrict__ tag, const double* __restrict__ y,
                              const int* __restrict__ rp, const int* __restrict__ ci, double u_max, double H,
                              OutletBc bc, int rows_too, double* __restrict__ A_val, double* __restrict__ rhs_u,
                              double* __restrict__ rhs_v, double* __restrict__ u, double* __restrict__ v) {
    CFA_GRID_DEP();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int t = tag[i];
    if (!momentum_dirichlet(t, bc)) return;
    const double ub = momentum_bc_u(t, y[i], u_max, H, bc);
    if (rows_too) {
        for (int q = rp[i]; q < rp[i + 1]; ++q) A_val[q] = (ci[q] == i) ? 1.0 : 0.0;
        rhs_u[i] = ub;
        rhs_v[i] = 0.0;
    }
    if (u) u[i] = ub;
    if (v) v[i] = 0.0;
}

// k_assemble_lumped_mass (fem_kernels.cuh:890-909), per row
__global__ void k_lumped_mass_rows(int n, const int* __restrict__ ev, const double* __restrict__ x,
                                   const double* __restrict__ y, const int* __restrict__ inc_ptr,
                                   const int* __restrict__ inc, double* __restrict__ m) {
    CFA_GRID_DEP();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = 0.0;
    for (int k = inc_ptr[i]; k < inc_ptr[i + 1]; ++k) {
        int nd[3];
        load_elem(ev, inc[k] >> 2, nd);
        const double detJ = (x[nd[1]] - x[nd[0]]) * (y[nd[2]] - y[nd[0]]) - (x[nd[2]] - x[nd[0]]) * (y[nd[1]] - y[nd[0]]);
        s += fabs(detJ) / 6.0;
    }
    m[i] = s;
}

// k_compute_oss_weights (fem_kernels.cuh:697-719), one thread per element
__global__ void k_oss_weights(int ne, const int* __restrict__ ev, const double* __restrict__ x,
                              const double* __restrict__ y, const double* __restrict__ us,
                              const double* __restrict__ vs, double dt, double rho, double nu, double stab,
                              double* __restrict__ elem_s) {
    CFA_GRID_DEP();
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    const int n0 = ev[3 * e], n1 = ev[3 * e + 1], n2 = ev[3 * e + 2];
    const double area = 0.5 * fabs((x[n1] - x[n0]) * (y[n2] - y[n0]) - (x[n2] - x[n0]) * (y[n1] - y[n0]));
    const double h = sqrt(2.0 * area);
    const double ub = (us[n0] + us[n1] + us[n2]) / 3.0;
    const double vb = (vs[n0] + vs[n1] + vs[n2]) / 3.0;
    const double tau = stab / (rho * (4.0 * nu / (h * h) + 2.0 * sqrt(ub * ub + vb * vb) / h) + 1.0e-300);
    elem_s[e] = rho * tau / dt;
}

// Area and grad f of one element (fem_kernels.cuh:735-752), rounded explicitly as the momentum's terms
// are; false for a degenerate element. Its weight is gradient_weight.
__device__ __forceinline__ bool gradient_element(double x0, double y0, double x1, double y1, double x2, double y2,
                                                 double f0, double f1, double f2, double& area, double& gx,
                                                 double& gy) {
    area = 0.5 * fabs(__fma_rn(x1 - x0, y2 - y0, -__dmul_rn(x2 - x0, y1 - y0)));
    if (area < 1.0e-14) return false;
    const double inv2A = 1.0 / (2.0 * area);
    gx = __dmul_rn(__fma_rn(f2, y0 - y1, __fma_rn(f0, y1 - y2, __dmul_rn(f1, y2 - y0))), inv2A);
    gy = __dmul_rn(__fma_rn(f2, x1 - x0, __fma_rn(f0, x2 - x1, __dmul_rn(f1, x0 - x2))), inv2A);
    return true;
}
__device__ __forceinline__ double gradient_weight(double rs, double area) { return __dmul_rn(rs, area) / 3.0; }

// k_accumulate_scalar_gradient (fem_kernels.cuh:726-757), per row: G_i(f) numerators
__global__ void k_scalar_gradient_rows(int n, const int* __restrict__ ev, const double* __restrict__ x,
                                       const double* __restrict__ y, const int* __restrict__ inc_ptr,
                                       const int* __restrict__ inc, const double* __restrict__ f,
                                       const double* __restrict__ elem_s, double* __restrict__ gx_out,
                                       double* __restrict__ gy_out) {
    CFA_GRID_DEP();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double sx = 0.0, sy = 0.0;
    for (int k = inc_ptr[i]; k < inc_ptr[i + 1]; ++k) {
        const int e = inc[k] >> 2;
        int nd[3];
        load_elem(ev, e, nd);
        const double x0 = x[nd[0]], y0 = y[nd[0]], x1 = x[nd[1]], y1 = y[nd[1]], x2 = x[nd[2]], y2 = y[nd[2]];
        double area, gx, gy;
        if (!gradient_element(x0, y0, x1, y1, x2, y2, f[nd[0]], f[nd[1]], f[nd[2]], area, gx, gy)) continue;
        const double w = gradient_weight(elem_s ? sqrt(elem_s[e]) : 1.0, area);
        sx = __fma_rn(w, gx, sx);
        sy = __fma_rn(w, gy, sy);
    }
    gx_out[i] = sx;
    gy_out[i] = sy;
}

// Element terms of the pressure system (fem_kernels.cuh:230-270), rounded explicitly as the momentum's
// are: the row gather and the element tiles give the same bits whatever the compiler contracts.
__device__ __forceinline__ double pressure_divergence(const int* nd, const Geom& g, const double* __restrict__ us,
                                                      const double* __restrict__ vs) {
    double d = __fma_rn(us[nd[0]], g.dNdx[0], __dmul_rn(us[nd[1]], g.dNdx[1]));
    d = __fma_rn(us[nd[2]], g.dNdx[2], d);
#pragma unroll
    for (int q = 0; q < 3; ++q) d = __fma_rn(vs[nd[q]], g.dNdy[q], d);
    return d;
}
// grad p and the projected gradient of one element
__device__ __forceinline__ void pressure_gradients(const int* nd, const Geom& g, const double* __restrict__ p_old,
                                                   const double* __restrict__ gpx, const double* __restrict__ gpy,
                                                   const double* __restrict__ mass, double s, double& gx, double& gy,
                                                   double& sx, double& sy) {
    const double p0 = p_old[nd[0]], p1 = p_old[nd[1]], p2 = p_old[nd[2]], third = sqrt(s) / 3.0;
    gx = __fma_rn(p2, g.dNdx[2], __fma_rn(p0, g.dNdx[0], __dmul_rn(p1, g.dNdx[1])));
    gy = __fma_rn(p2, g.dNdy[2], __fma_rn(p0, g.dNdy[0], __dmul_rn(p1, g.dNdy[1])));
    sx = sy = 0.0;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double im = 1.0 / fmax(mass[nd[q]], 1.0e-14);
        sx = __fma_rn(gpx[nd[q]], im, sx);
        sy = __fma_rn(gpy[nd[q]], im, sy);
    }
    sx = __dmul_rn(sx, third);
    sy = __dmul_rn(sy, third);
}
// -(rho / dt) (area / 3) div u - (s area (grad N . grad p) - area (grad N . the projected gradient))
__device__ __forceinline__ double pressure_rhs(double area, double s, double rho_dt, double div_u, double dNdx_a,
                                               double dNdy_a, double gx, double gy, double sx, double sy) {
    const double stab_i = __fma_rn(__dmul_rn(s, area), __fma_rn(dNdx_a, gx, __dmul_rn(dNdy_a, gy)),
                                   -__dmul_rn(area, __fma_rn(dNdy_a, sy, __dmul_rn(dNdx_a, sx))));
    return __fma_rn(__dmul_rn(-rho_dt, area / 3.0), div_u, -stab_i);
}
__device__ __forceinline__ double pressure_entry(double area, double xa, double ya, double xb, double yb) {
    return __dmul_rn(area, __fma_rn(xa, xb, __dmul_rn(ya, yb)));
}

// Pressure rows: k_assemble_pressure_poisson (fem_kernels.cuh:201-282) gathered per row; with
// oss_val the rows of B and B^T of k_assemble_oss_operator (:807-847) and inv_m (:849-852) in
// the same pass; with with_bc the Dirichlet rows/columns of k_apply_bc_pressure (:460-490).
// A row of up to kPressCap entries accumulates K, Bx, By, B^T x, B^T y in shared memory laid out
// [array][slot][thread], so that threads adding to different slots of their rows hit different
// banks; longer rows accumulate in place in global memory. Every entry takes its terms in the
// element order of the incidence either way.
constexpr int kPressThreads = 128;
constexpr int kPressCap = 16;
constexpr size_t kPressSmem = (size_t)5 * kPressCap * kPressThreads * sizeof(double);

__global__ void __launch_bounds__(kPressThreads)
k_pressure_rows(int n, int nnz, const int* __restrict__ ev, const double* __restrict__ x,
                const double* __restrict__ y, const int* __restrict__ tag, const int* __restrict__ inc_ptr,
                const int* __restrict__ inc, const int* __restrict__ pos, const int* __restrict__ rp,
                const int* __restrict__ ci, const double* __restrict__ us, const double* __restrict__ vs,
                const double* __restrict__ p_old, const double* __restrict__ gpx, const double* __restrict__ gpy,
                const double* __restrict__ mass, const double* __restrict__ elem_s, double dt, double rho,
                double stab, int with_bc, OutletBc bc, double* __restrict__ Kp_val, double* __restrict__ rhs_p,
                double* __restrict__ div_num, double* __restrict__ dp, double* __restrict__ oss_val,
                double* __restrict__ inv_m) {
    CFA_GRID_DEP();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int r0 = rp[i], len = rp[i + 1] - r0;
    const bool local = len <= kPressCap;
    const bool want_oss = oss_val != nullptr;
    extern __shared__ double press_sm[];   // [5][kPressCap][blockDim.x]
    const int T = blockDim.x, tt = threadIdx.x;
    double* sK = press_sm + tt;                          // sK[q * T]: K entry q of this row
    double* sBx = press_sm + 1 * kPressCap * T + tt;
    double* sBy = press_sm + 2 * kPressCap * T + tt;
    double* sTx = press_sm + 3 * kPressCap * T + tt;
    double* sTy = press_sm + 4 * kPressCap * T + tt;
    double *Bx = oss_val, *By = oss_val + (size_t)nnz, *BTx = oss_val + 2 * (size_t)nnz, *BTy = oss_val + 3 * (size_t)nnz;
    if (local) {
        for (int q = 0; q < len; ++q) {
            sK[q * T] = 0.0;
            if (want_oss) { sBx[q * T] = 0.0; sBy[q * T] = 0.0; sTx[q * T] = 0.0; sTy[q * T] = 0.0; }
        }
    } else {
        for (int q = 0; q < len; ++q) Kp_val[r0 + q] = 0.0;
        if (want_oss)
            for (int q = 0; q < len; ++q) { Bx[r0 + q] = 0.0; By[r0 + q] = 0.0; BTx[r0 + q] = 0.0; BTy[r0 + q] = 0.0; }
    }
    double rhs_row = 0.0, div_row = 0.0;
    for (int k = inc_ptr[i]; k < inc_ptr[i + 1]; ++k) {
        const int e = inc[k] >> 2, a = inc[k] & 3;
        int nd[3];
        load_elem(ev, e, nd);
        const Geom g = elem_geom(nd, x, y);
        if (!g.ok) continue;
        const double area = g.area;
        const double div_u = pressure_divergence(nd, g, us, vs);
        double s = 0.0, sx = 0.0, sy = 0.0, gx = 0.0, gy = 0.0;
        if (stab > 0.0) {
            s = elem_s[e];
            pressure_gradients(nd, g, p_old, gpx, gpy, mass, s, gx, gy, sx, sy);
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double K_ij = pressure_entry(area, g.dNdx[a], g.dNdy[a], g.dNdx[j], g.dNdy[j]);
            const int p = pos[3 * k + j];
            if (local) sK[(p - r0) * T] = __fma_rn(1.0 + s, K_ij, sK[(p - r0) * T]);
            else Kp_val[p] = __fma_rn(1.0 + s, K_ij, Kp_val[p]);
        }
        rhs_row += pressure_rhs(area, s, rho / dt, div_u, g.dNdx[a], g.dNdy[a], gx, gy, sx, sy);
        div_row = __fma_rn(area / 3.0, div_u, div_row);
        if (want_oss) {
            const double w = __dmul_rn(sqrt(elem_s[e]), area) / 3.0;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int p = pos[3 * k + j];
                // B_ij = sum_K w_K grad N_j|K (row i, column j); B^T_ij = B_ji = sum_K w_K grad N_i|K
                if (local) {
                    const int q = (p - r0) * T;
                    sBx[q] = __fma_rn(w, g.dNdx[j], sBx[q]);
                    sBy[q] = __fma_rn(w, g.dNdy[j], sBy[q]);
                    sTx[q] = __fma_rn(w, g.dNdx[a], sTx[q]);
                    sTy[q] = __fma_rn(w, g.dNdy[a], sTy[q]);
                } else {
                    Bx[p] = __fma_rn(w, g.dNdx[j], Bx[p]);
                    By[p] = __fma_rn(w, g.dNdy[j], By[p]);
                    BTx[p] = __fma_rn(w, g.dNdx[a], BTx[p]);
                    BTy[p] = __fma_rn(w, g.dNdy[a], BTy[p]);
                }
            }
        }
    }
    if (want_oss) {
        inv_m[i] = 1.0 / fmax(mass[i], 1.0e-14);
        if (local)
            for (int q = 0; q < len; ++q) {
                Bx[r0 + q] = sBx[q * T];
                By[r0 + q] = sBy[q * T];
                BTx[r0 + q] = sTx[q * T];
                BTy[r0 + q] = sTy[q * T];
            }
    }
    div_num[i] = div_row;
    if (with_bc && pressure_dirichlet(i, tag[i], bc)) {
        for (int q = 0; q < len; ++q) Kp_val[r0 + q] = (ci[r0 + q] == i) ? 1.0 : 0.0;
        rhs_p[i] = 0.0;
        if (dp) dp[i] = 0.0;
        return;
    }
    for (int q = 0; q < len; ++q) {
        double v = local ? sK[q * T] : Kp_val[r0 + q];
        if (with_bc) {
            const int c = ci[r0 + q];
            if (c != i && pressure_dirichlet(c, tag[c], bc)) v = 0.0;
        }
        Kp_val[r0 + q] = v;
    }
    rhs_p[i] = rhs_row;
}

// Scalar gradient on element tiles: grad f and the weight (area / 3) sqrt(s) of every element
// once, then the rows. The tile's plan is as many bytes as it saves, so the form pays while it is one
// wave (5 blocks of 96 rows an SM, 71k vertices). Tiles / gathers in us, the L2 flushed first: 7k vertices
// 10.2 / 18.5, 22k 10.3 / 18.0, 66k 14.3 / 18.6, 76k 18.4 / 18.4, 100k 20.5 / 19.5, 135k 22.3 / 20.5.
constexpr EtForm kGradForm = {5, 5, 1, 1};

__global__ void __launch_bounds__(kEtThreads)
k_scalar_gradient_tiles(ElemTileView tv, int n, const int* __restrict__ ev, const double* __restrict__ x,
                        const double* __restrict__ y, const double* __restrict__ f, const double* __restrict__ elem_s,
                        double* __restrict__ gx_out, double* __restrict__ gy_out) {
    extern __shared__ __align__(16) double et_rec[];   // [3][tv.stride]
    const EtBlock b = et_block(tv, n);
    const int S = tv.stride;
    CFA_GRID_DEP();
    for (int le = threadIdx.x; le < b.ne; le += kEtThreads) {
        int nd[3];
        load_elem(ev, tv.elems[b.i0 + le], nd);
        const double es = elem_s ? elem_s[tv.elems[b.i0 + le]] : 1.0;
        const double x0 = x[nd[0]], y0 = y[nd[0]], x1 = x[nd[1]], y1 = y[nd[1]], x2 = x[nd[2]], y2 = y[nd[2]];
        double area, gx = 0.0, gy = 0.0, w = 0.0;
        if (gradient_element(x0, y0, x1, y1, x2, y2, f[nd[0]], f[nd[1]], f[nd[2]], area, gx, gy))
            w = gradient_weight(elem_s ? sqrt(es) : 1.0, area);
        et_rec[le] = gx;
        et_rec[S + le] = gy;
        et_rec[2 * S + le] = w;
    }
    __syncthreads();
    for (int i = b.r0 + threadIdx.x; i < b.r1; i += kEtThreads) {
        double sx = 0.0, sy = 0.0;
        for (int s = tv.inc_ptr[i]; s < tv.inc_ptr[i + 1]; ++s) {
            const int le = tv.rcode[s] >> 2;
            const double w = et_rec[2 * S + le];
            sx = __fma_rn(w, et_rec[le], sx);
            sy = __fma_rn(w, et_rec[S + le], sy);
        }
        gx_out[i] = sx;
        gy_out[i] = sy;
    }
}

// Pressure rows on element tiles, 19 doubles an element: the symmetric K (6), grad N (6), w, 1 + s,
// the right-hand side of each vertex (3), area / 3 and div u. The weights enter the sums by fused
// multiply-adds, as in the row gather. Bound by latency (half of a warp's wait between instructions is
// on global loads, DRAM 13% busy) with the LSU data pipe next (56% busy, two thirds of it the records'
// shared-memory reads, seven a contribution and 2.6 contributions an entry); registers and records
// leave four blocks an SM. Staging the codes in shared memory and loading offsets ahead was slower (152
// us), as were blocks of 384 threads (177 us). Gathers -> tiles, the L2 flushed first: 373 -> 150 us at
// 402k vertices (162 MB of DRAM, 1.1 TB/s), 3738 -> 1430 us at 4.2M, 41 -> 20.5 us at 22k, 35 -> 18.4 us at 7k.
__global__ void __launch_bounds__(kEtThreads)
k_pressure_tiles(ElemTileView tv, int n, int nnz, const int* __restrict__ ev, const double* __restrict__ x,
                 const double* __restrict__ y, const int* __restrict__ tag, const int* __restrict__ rp,
                 const int* __restrict__ ci, const double* __restrict__ us, const double* __restrict__ vs,
                 const double* __restrict__ p_old, const double* __restrict__ gpx, const double* __restrict__ gpy,
                 const double* __restrict__ mass, const double* __restrict__ elem_s, double dt, double rho,
                 double stab, int with_bc, OutletBc bc, double* __restrict__ Kp_val, double* __restrict__ rhs_p,
                 double* __restrict__ div_num, double* __restrict__ dp, double* __restrict__ oss_val,
                 double* __restrict__ inv_m) {
    extern __shared__ __align__(16) double et_rec[];   // [19][tv.stride]
    const EtBlock b = et_block(tv, n);
    const int S = tv.stride;
    const bool want_oss = oss_val != nullptr;
    CFA_GRID_DEP();
    for (int le = threadIdx.x; le < b.ne; le += kEtThreads) {
        int nd[3];
        load_elem(ev, tv.elems[b.i0 + le], nd);
        const double es = stab > 0.0 || want_oss ? elem_s[tv.elems[b.i0 + le]] : 0.0;
        const Geom g = elem_geom(nd, x, y);
        double* rec = et_rec + le;
        if (!g.ok) {
#pragma unroll
            for (int q = 0; q < 19; ++q) rec[q * S] = 0.0;
            continue;
        }
        const double area = g.area;
        const double div_u = pressure_divergence(nd, g, us, vs);
        double s = 0.0, sx = 0.0, sy = 0.0, gx = 0.0, gy = 0.0;
        if (stab > 0.0) {
            s = es;
            pressure_gradients(nd, g, p_old, gpx, gpy, mass, s, gx, gy, sx, sy);
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
#pragma unroll
            for (int j = a; j < 3; ++j)   // 00 01 02 11 12 22
                rec[(a + j + (a > 0 ? 1 : 0)) * S] = pressure_entry(area, g.dNdx[a], g.dNdy[a], g.dNdx[j], g.dNdy[j]);
            rec[(6 + a) * S] = g.dNdx[a];
            rec[(9 + a) * S] = g.dNdy[a];
            rec[(14 + a) * S] = pressure_rhs(area, s, rho / dt, div_u, g.dNdx[a], g.dNdy[a], gx, gy, sx, sy);
        }
        rec[12 * S] = __dmul_rn(sqrt(es), area) / 3.0;
        rec[13 * S] = 1.0 + s;
        rec[17 * S] = area / 3.0;
        rec[18 * S] = div_u;
    }
    __syncthreads();
    double *Bx = oss_val, *By = oss_val + (size_t)nnz, *BTx = oss_val + 2 * (size_t)nnz, *BTy = oss_val + 3 * (size_t)nnz;
    const int p0 = rp[b.r0], p1 = rp[b.r1];
    const unsigned short* code = tv.ecode + 3 * (size_t)b.i0;
    auto entry = [&](int p, int c0, int c1) {
        double k = 0.0, bx = 0.0, by = 0.0, tx = 0.0, ty = 0.0;
        for (int c = c0; c < c1; ++c) {
            const int q = code[c], a = (q >> 2) & 3, j = q & 3;
            const double* rec = et_rec + (q >> 4);
            k = __fma_rn(rec[13 * S], rec[(a + j + (a > 0 && j > 0 ? 1 : 0)) * S], k);
            if (want_oss) {
                // B_ij = sum_K w_K grad N_j|K (row i, column j); B^T_ij = B_ji = sum_K w_K grad N_i|K
                const double w = rec[12 * S];
                bx = __fma_rn(w, rec[(6 + j) * S], bx);
                by = __fma_rn(w, rec[(9 + j) * S], by);
                tx = __fma_rn(w, rec[(6 + a) * S], tx);
                ty = __fma_rn(w, rec[(9 + a) * S], ty);
            }
        }
        if (with_bc) {   // a Dirichlet column; its own row is written below
            const int col = ci[p];
            if (pressure_dirichlet(col, tag[col], bc)) k = 0.0;
        }
        Kp_val[p] = k;
        if (want_oss) {
            Bx[p] = bx;
            By[p] = by;
            BTx[p] = tx;
            BTy[p] = ty;
        }
    };
    for (int p = p0 + threadIdx.x; p < p1; p += kEtThreads)
        entry(p, tv.eoff[p], p + 1 < p1 ? (int)tv.eoff[p + 1] : 3 * (b.i1 - b.i0));
    if (with_bc) __syncthreads();   // the Dirichlet rows below follow the entries' values
    for (int i = b.r0 + threadIdx.x; i < b.r1; i += kEtThreads) {
        double r = 0.0, d = 0.0;
        for (int s = tv.inc_ptr[i]; s < tv.inc_ptr[i + 1]; ++s) {
            const int q = tv.rcode[s], le = q >> 2;
            r += et_rec[(14 + (q & 3)) * S + le];
            d = __fma_rn(et_rec[17 * S + le], et_rec[18 * S + le], d);
        }
        if (want_oss) inv_m[i] = 1.0 / fmax(mass[i], 1.0e-14);
        div_num[i] = d;
        if (with_bc && pressure_dirichlet(i, tag[i], bc)) {
            for (int q = rp[i]; q < rp[i + 1]; ++q) Kp_val[q] = (ci[q] == i) ? 1.0 : 0.0;
            r = 0.0;
            if (dp) dp[i] = 0.0;
        }
        rhs_p[i] = r;
    }
}

// k_apply_bc_pressure (fem_kernels.cuh:460-490) alone; with mean removal first when pinned
// (k_sum / k_subtract_mean, :493-510, summed here in a fixed order).
__global__ void k_pressure_bc(int n, const int* __restrict__ tag, const int* __restrict__ rp,
                              const int* __restrict__ ci, OutletBc bc, const double* __restrict__ sums,
                              const double* __restrict__ mass, double* __restrict__ Kp_val,
                              double* __restrict__ rhs, double* __restrict__ dp) {
    CFA_GRID_DEP();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (sums) rhs[i] -= sums[0] / sums[1] * mass[i];
    if (pressure_dirichlet(i, tag[i], bc)) {
        for (int q = rp[i]; q < rp[i + 1]; ++q) Kp_val[q] = (ci[q] == i) ? 1.0 : 0.0;
        rhs[i] = 0.0;
        if (dp) dp[i] = 0.0;
    } else {
        for (int q = rp[i]; q < rp[i + 1]; ++q) {
            const int c = ci[q];
            if (c != i && pressure_dirichlet(c, tag[c], bc)) Kp_val[q] = 0.0;
        }
    }
}

// Sums of rhs and mass in a fixed order (deterministic), into out[0], out[1]
__global__ void __launch_bounds__(kThreads)
k_sum2(int n, const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ part,
       unsigned int* __restrict__ counter, double* __restrict__ out) {
    CFA_GRID_DEP();
    __shared__ double sh[2 * kWarps];
    double v[2] = {0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        v[0] += a[i];
        v[1] += b[i];
    }
    block_sum<2>(v, sh);
    if (publish_partials<2>(v, part, counter)) {
        reduce_partials<2>(v, part, counter, sh);
        if (threadIdx.x == 0) { out[0] = v[0]; out[1] = v[1]; }
    }
}

static cfa_status mean_removal_sums(cfa_ctx* ctx, int n, const double* rhs, const double* mass, double* out2) {
    const int grid = row_grid(ctx, n, 1);
    CFA_PROPAGATE(ensure_partials(ctx, 2 * (size_t)grid + 2));
    CFA_LAUNCH(ctx, k_sum2, grid, kThreads, 0, n, rhs, mass, ctx->d_part, ctx->d_counters, out2);
    return CFA_OK;
}

static void allow_et_kernels() {
    static std::once_flag once;
    std::call_once(once, [] {
        cudaFuncSetAttribute(k_momentum_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, kEtMaxSmem);
        cudaFuncSetAttribute(k_pressure_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, kEtMaxSmem);
        cudaFuncSetAttribute(k_scalar_gradient_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, kEtMaxSmem);
    });
}

}  // namespace cfa

using namespace cfa;

extern "C" {

cfa_status cfa_assemble_momentum_nu(cfa_ctx* ctx, const cfa_mesh* m, const double* u_old, const double* v_old,
                                    const double* u_prev, const double* v_prev, const double* p_old,
                                    const cfa_momentum_params* prm, const double* nu_node,
                                    const cfa_momentum_bc* bcp, double* A_val, double* rhs_u, double* rhs_v,
                                    double* mass, double* u, double* v);

cfa_status cfa_assemble_momentum(cfa_ctx* ctx, const cfa_mesh* m, const double* u_old, const double* v_old,
                                 const double* u_prev, const double* v_prev, const double* p_old,
                                 const cfa_momentum_params* prm, const cfa_momentum_bc* bcp, double* A_val,
                                 double* rhs_u, double* rhs_v, double* mass, double* u, double* v) {
    return cfa_assemble_momentum_nu(ctx, m, u_old, v_old, u_prev, v_prev, p_old, prm, nullptr, bcp, A_val, rhs_u,
                                    rhs_v, mass, u, v);
}

cfa_status cfa_assemble_momentum_nu(cfa_ctx* ctx, const cfa_mesh* m, const double* u_old, const double* v_old,
                                    const double* u_prev, const double* v_prev, const double* p_old,
                                    const cfa_momentum_params* prm, const double* nu_node,
                                    const cfa_momentum_bc* bcp, double* A_val, double* rhs_u, double* rhs_v,
                                    double* mass, double* u, double* v) {
    CFA_ENTER(ctx);
    CFA_ARG(m && u_old && v_old && u_prev && v_prev && p_old && prm && A_val && rhs_u && rhs_v && mass);
    CFA_ARG(!bcp || (u && v));
    MomParams P{prm->dt, prm->nu, prm->rho, prm->a0, prm->a1, prm->a2, prm->c1, prm->c2, prm->tau_time, prm->skew_coef};
    const double u_max = bcp ? bcp->u_max : 0.0, H = bcp ? bcp->H : 1.0;
    allow_et_kernels();
    if (et_better(m->et, m->n, ctx->num_sms, kMomForm))
        CFA_LAUNCH(ctx, k_momentum_tiles, m->et.ntiles, kEtThreads, et_smem_bytes(m->et, 16), m->tiles(), m->n, m->ev,
                   m->x, m->y, m->tag, m->rp, m->ci, u_old, v_old, u_prev, v_prev, p_old, nu_node, P, bcp ? 1 : 0, u_max, H, m->bc,
                   A_val, rhs_u, rhs_v, mass);
    else
        CFA_LAUNCH(ctx, k_momentum_rows, ceil_div(m->n, kThreads), kThreads, kMomSmem, m->n, m->ev, m->x, m->y, m->tag,
                   m->inc_ptr.p, m->inc.p, m->pos.p, m->rp, m->ci, u_old, v_old, u_prev, v_prev, p_old, nu_node, P,
                   bcp ? 1 : 0, u_max, H, m->bc, A_val, rhs_u, rhs_v, mass);
    if (bcp)   // solution values on Dirichlet nodes after the rows (u may alias u_old)
        CFA_LAUNCH(ctx, k_momentum_bc, ceil_div(m->n, kThreads), kThreads, 0, m->n, m->tag, m->y, m->rp, m->ci,
                   u_max, H, m->bc, 0, A_val, rhs_u, rhs_v, u, v);
    CFA_CHECK_LAUNCH();
    return CFA_OK;
}

cfa_status cfa_apply_bc_momentum(cfa_ctx* ctx, const cfa_mesh* m, const cfa_momentum_bc* bcp, double* A_val,
                                 double* rhs_u, double* rhs_v, double* u, double* v) {
    CFA_ENTER(ctx);
    CFA_ARG(m && bcp && A_val && rhs_u && rhs_v);
    CFA_LAUNCH(ctx, k_momentum_bc, ceil_div(m->n, kThreads), kThreads, 0, m->n, m->tag, m->y, m->rp, m->ci,
               bcp->u_max, bcp->H, m->bc, 1, A_val, rhs_u, rhs_v, u, v);
    CFA_CHECK_LAUNCH();
    return CFA_OK;
}

cfa_status cfa_lumped_mass(cfa_ctx* ctx, const cfa_mesh* m, double* mass) {
    CFA_ENTER(ctx);
    CFA_ARG(m && mass);
    CFA_LAUNCH(ctx, k_lumped_mass_rows, ceil_div(m->n, kThreads), kThreads, 0, m->n, m->ev, m->x, m->y,
               m->inc_ptr.p, m->inc.p, mass);
    CFA_CHECK_LAUNCH();
    return CFA_OK;
}

cfa_status cfa_oss_weights(cfa_ctx* ctx, const cfa_mesh* m, const double* us, const double* vs, double dt,
                           double rho, double nu, double stab, double* elem_s) {
    CFA_ENTER(ctx);
    CFA_ARG(m && us && vs && elem_s);
    CFA_LAUNCH(ctx, k_oss_weights, ceil_div(m->ne, kThreads), kThreads, 0, m->ne, m->ev, m->x, m->y, us, vs, dt,
               rho, nu, stab, elem_s);
    CFA_CHECK_LAUNCH();
    return CFA_OK;
}

cfa_status cfa_scalar_gradient(cfa_ctx* ctx, const cfa_mesh* m, const double* f, const double* elem_s, double* gx,
                               double* gy) {
    CFA_ENTER(ctx);
    CFA_ARG(m && f && gx && gy);
    allow_et_kernels();
    if (et_better(m->et, m->n, ctx->num_sms, kGradForm))
        CFA_LAUNCH(ctx, k_scalar_gradient_tiles, m->et.ntiles, kEtThreads, et_smem_bytes(m->et, 3), m->tiles(), m->n,
                   m->ev, m->x, m->y, f, elem_s, gx, gy);
    else
        CFA_LAUNCH(ctx, k_scalar_gradient_rows, ceil_div(m->n, kThreads), kThreads, 0, m->n, m->ev, m->x, m->y,
                   m->inc_ptr.p, m->inc.p, f, elem_s, gx, gy);
    CFA_CHECK_LAUNCH();
    return CFA_OK;
}

static cfa_status assemble_pressure(cfa_ctx* ctx, const cfa_mesh* m, const double* us, const double* vs,
                                    const double* p_old, const double* gpx, const double* gpy, const double* mass,
                                    const double* elem_s, double dt, double rho, double stab, int apply_bc,
                                    double* Kp, double* rhs, double* div, double* dp, double* oss_val,
                                    double* inv_m) {
    // With the pinned outlet the RHS loses its mean before the BC rows (apply_bc_pressure,
    // fem_kernels.cuh:519-531): assemble without BC, then sums, then the BC kernel.
    const bool split = apply_bc && m->bc.outlet_dirichlet;
    static std::once_flag press_once;
    std::call_once(press_once, [] {
        cudaFuncSetAttribute(k_pressure_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPressSmem);
    });
    allow_et_kernels();
    const int with_bc = (apply_bc && !split) ? 1 : 0;
    if (m->et.ok)
        CFA_LAUNCH(ctx, k_pressure_tiles, m->et.ntiles, kEtThreads, et_smem_bytes(m->et, 19), m->tiles(), m->n,
                   m->nnz, m->ev, m->x, m->y, m->tag, m->rp, m->ci, us, vs, p_old, gpx, gpy, mass, elem_s, dt, rho, stab, with_bc,
                   m->bc, Kp, rhs, div, dp, oss_val, inv_m);
    else
        CFA_LAUNCH(ctx, k_pressure_rows, ceil_div(m->n, kPressThreads), kPressThreads, kPressSmem, m->n, m->nnz, m->ev,
                   m->x, m->y, m->tag, m->inc_ptr.p, m->inc.p, m->pos.p, m->rp, m->ci, us, vs, p_old, gpx, gpy, mass,
                   elem_s, dt, rho, stab, with_bc, m->bc, Kp, rhs, div, dp, oss_val, inv_m);
    if (split) {
        double* sums = ctx->d_part;   // after the partials region
        CFA_PROPAGATE(ensure_partials(ctx, 2 * (size_t)row_grid(ctx, m->n, 1) + 4));
        sums = ctx->d_part + ctx->part_cap - 2;
        CFA_PROPAGATE(mean_removal_sums(ctx, m->n, rhs, mass, sums));
        CFA_LAUNCH(ctx, k_pressure_bc, ceil_div(m->n, kThreads), kThreads, 0, m->n, m->tag, m->rp, m->ci, m->bc,
                   (const double*)sums, mass, Kp, rhs, dp);
    }
    CFA_CHECK_LAUNCH();
    return CFA_OK;
}

cfa_status cfa_assemble_ppe(cfa_ctx* ctx, const cfa_mesh* m, const double* us, const double* vs, const double* p_old,
                            const double* gpx, const double* gpy, const double* mass, const double* elem_s, double dt,
                            double rho, double stab, int apply_bc, double* Kp, double* rhs, double* div, double* dp) {
    CFA_ENTER(ctx);
    CFA_ARG(m && us && vs && Kp && rhs && div);
    CFA_ARG(!(stab > 0.0) || (p_old && gpx && gpy && mass && elem_s));
    return assemble_pressure(ctx, m, us, vs, p_old, gpx, gpy, mass, elem_s, dt, rho, stab, apply_bc, Kp, rhs, div,
                             dp, nullptr, nullptr);
}

cfa_status cfa_apply_bc_pressure(cfa_ctx* ctx, const cfa_mesh* m, double* Kp, double* rhs, double* dp,
                                 const double* mass) {
    CFA_ENTER(ctx);
    CFA_ARG(m && Kp && rhs);
    const double* sums = nullptr;
    if (m->bc.outlet_dirichlet) {
        CFA_ARG(mass);
        CFA_PROPAGATE(ensure_partials(ctx, 2 * (size_t)row_grid(ctx, m->n, 1) + 4));
        double* s = ctx->d_part + ctx->part_cap - 2;
        CFA_PROPAGATE(mean_removal_sums(ctx, m->n, rhs, mass, s));
        sums = s;
    }
    CFA_LAUNCH(ctx, k_pressure_bc, ceil_div(m->n, kThreads), kThreads, 0, m->n, m->tag, m->rp, m->ci, m->bc, sums,
               mass, Kp, rhs, dp);
    CFA_CHECK_LAUNCH();
    return CFA_OK;
}

cfa_status cfa_assemble_oss(cfa_ctx* ctx, const cfa_mesh* m, const double* elem_s, const double* mass,
                            double* oss_val, double* inv_m) {
    CFA_ENTER(ctx);
    CFA_ARG(m && elem_s && mass && oss_val && inv_m);
    // The B/B^T rows are produced by the pressure-row pass; K, RHS and div go to scratch here.
    DevBuf<double> scratch;
    CFA_CUDA(scratch.ensure((size_t)m->nnz + 2 * (size_t)m->n));
    double* K = scratch.p;
    double* rhs = K + m->nnz;
    double* div = rhs + m->n;
    CFA_PROPAGATE(assemble_pressure(ctx, m, m->x, m->y, m->x, m->x, m->y, mass, elem_s, 1.0, 1.0, 0.0, 0, K, rhs,
                                    div, nullptr, oss_val, inv_m));
    CFA_CUDA(cudaStreamSynchronize(ctx->stream));   // scratch is released on return
    return CFA_OK;
}

// Fused pressure system: PPE (+ BCs) and the OSS operator in one row pass.
cfa_status cfa_assemble_pressure_system(cfa_ctx* ctx, const cfa_mesh* m, const double* us, const double* vs,
                                        const double* p_old, const double* gpx, const double* gpy,
                                        const double* mass, const double* elem_s, double dt, double rho,
                                        double stab, double* Kp, double* rhs, double* div, double* dp,
                                        double* oss_val, double* inv_m) {
    CFA_ENTER(ctx);
    CFA_ARG(m && us && vs && Kp && rhs && div);
    CFA_ARG(!(stab > 0.0) || (p_old && gpx && gpy && mass && elem_s && oss_val && inv_m));
    return assemble_pressure(ctx, m, us, vs, p_old, gpx, gpy, mass, elem_s, dt, rho, stab, 1, Kp, rhs, div, dp,
                             stab > 0.0 ? oss_val : nullptr, inv_m);
}

}  // extern "C"
