// des_adjoint.cu -- hand-written reverse mode of the 3D FP64 step.
//
// Every kernel here is the adjoint (transpose of the derivative) of one
// forward stage of des_kernels.cu, evaluated at the forward values recorded
// on the tape.  Branches (yield, EVP choice, clamps, damping signs, Dirichlet
// and velocity BCs) follow the forward's decisions, so each adjoint is the
// derivative of the branch the forward took: a subgradient at the kinks.
// Where the forward's map is discontinuous in its input -- the eigenbasis
// of repeated principal stresses, the sign of a zero force under damping --
// the term of the discontinuity is dropped.  Adjoints are checked against
// finite differences, not bit for bit: divisions by 3 are div3, and the
// reciprocals of the common paths are recip_newton (~1e-14 relative), each
// a few FP64 instructions instead of an FP64 division.
#include <algorithm>
#include <cfloat>

#include "des_adjoint.cuh"
#include "des_bc.cuh"
#include "des_gather.cuh"
#include "des_kernels.cuh"
#include "des_rheology.cuh"

namespace des {

constexpr int TPB_A = BLOCK_MOST;   // the element and facet kernels' largest block

__device__ __forceinline__ double tshp(const TapeStep &t, size_t ne, int k, int i, int e)
{
    return t.shp[((size_t)k * 4 + i) * ne + e];
}

// the stress after NMD_stress (geometry.cxx:182-236), as k_elem_force forms
// it, from the tape's stress after update_stress and its pressure changes:
// the same operations in the same order, so the same bits (the division by
// 4 is exact, with or without a fused multiply-add)
__device__ __forceinline__ void tape_sss(const KP &p, const TapeStep &t, int e, double *s)
{
    const size_t ne = p.ne;
    double dpn = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) dpn += t.dpn[conn_at(p, i, e)];
    const double corr = divnd<3>(-t.dp[e] + dpn / 4);
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) s[cc] = t.sstar[cc * ne + e];
#pragma unroll
    for (int i = 0; i < 3; ++i) s[i] += corr;
}

__device__ __forceinline__ void tload3(const double *a, size_t nn, int n, double *o)
{
    o[0] = a[n];
    o[1] = a[nn + n];
    o[2] = a[2 * nn + n];
}

// ------------------------------------------------------------------
// geometry: volume (geometry.cxx:29-49) and shape functions
// (geometry.cxx:368-455) of one tet, reversed.  Given the adjoints gvol of
// the volume and gs[k][i] of g_i,k = dN_i/dx_k, writes the coordinate
// adjoints gc.  Moving the nodes by d_j changes the volume by
// V sum_j g_j . d_j and the gradients of the linear functions by
// dg_i = -sum_j (d_j . g_i) g_j (the first-order change of the inverse of
// the element's deformation), so with M_ab = sum_i g_i,a gs_b,i
//   gc_j,a = sum_b (gvol V delta_ab - M_ab) g_j,b:
// 75 multiply-adds on the shape functions alone, in place of the reversed
// cofactor expressions of the coordinates (about 250 FP64 operations).
// ------------------------------------------------------------------
__device__ __forceinline__ void geom_reverse(const double (*g)[4], double vol, const double (*gs)[4], double gvol,
                                             double (*gc)[3])
{
    double m[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            double acc = a == b ? gvol * vol : 0.0;
#pragma unroll
            for (int i = 0; i < 4; ++i) acc -= g[a][i] * gs[b][i];
            m[a][b] = acc;
        }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int a = 0; a < 3; ++a) gc[j][a] = m[a][0] * g[0][j] + m[a][1] * g[1][j] + m[a][2] * g[2][j];
}

// mass, tmass and volume_n of the element's four nodes (geometry.cxx:313-365),
// reversed: adds to gvol and returns the element density adjoint
__device__ __forceinline__ double mass_reverse(const KP &p, int e, const double *gm, const double *gtm,
                                               const double *gvn, double vol, double rho_e, double &gvol)
{
    const bool quasi = p.prm.is_quasi_static, thermal = p.prm.has_thermal_diffusion;
    const double rho = quasi ? p.mat.rho_pseudo : rho_e;
    const double cp = m_cp(p, e);
    const double sm = (gm[0] + gm[1]) + (gm[2] + gm[3]);
    gvol += rho / 4 * sm + ((gvn[0] + gvn[1]) + (gvn[2] + gvn[3]));
    double grho = quasi ? 0.0 : vol / 4 * sm;
    if (thermal) {
        const double st = cp / 4 * ((gtm[0] + gtm[1]) + (gtm[2] + gtm[3]));
        gvol += rho_e * st;
        grho += vol * st;
    }
    return grho;
}

// ------------------------------------------------------------------
// end of the step: mass (at the new volumes), rotate_stress
// (fields.cxx:411-483, Jaumann rate with the new velocities and shape
// functions) and the geometry of the new coordinates, reversed.
// In: as = adjoint of the rotated stress, avol/ashp = adjoints of the new
// volume and shape functions, am/atm/avn = adjoints of the new nodal mass,
// tmass, volume_n.  Out: as = adjoint of the stress before the rotation,
// arho = element density adjoint (mass share), slot3 = new-velocity
// contributions, slotx = new-coordinate contributions.
// ------------------------------------------------------------------
__global__ void __launch_bounds__(TPB_A) k_adj_end_geometry(KP p, AdjBufs a, TapeStep t, TapeStep t1, double dt)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= p.ne) return;
    const size_t ne = p.ne, nn = p.nn;
    int nodes[4];
    double v[4][3], sh[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        nodes[i] = conn_at(p, i, e);
        tload3(t1.v, nn, nodes[i], v[i]);
    }
    const double vol = t1.vol[e];
    double gvol = a.avol[e];
    double gs[3][4];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            sh[k][i] = tshp(t1, ne, k, i, e);
            gs[k][i] = a.ashp[((size_t)k * 4 + i) * ne + e];
        }
    {
        double gm[4], gtm[4], gvn[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            gm[i] = a.am[nodes[i]];
            gtm[i] = a.atm[nodes[i]];
            gvn[i] = a.avn[nodes[i]];
        }
        a.arho[e] = mass_reverse(p, e, gm, gtm, gvn, vol, t.rho[e], gvol);
    }
    double h3 = 0, h4 = 0, h5 = 0;   // half the spin's adjoints
    if (p.mat.rheol_type & DES_RH_ELASTIC) {
        double s[6], g[6];
        tape_sss(p, t, e, s);
#pragma unroll
        for (int cc = 0; cc < 6; ++cc) g[cc] = a.as[cc * ne + e];
        double w3 = 0, w4 = 0, w5 = 0;   // dt times the spin
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            w3 += v[i][0] * sh[1][i] - v[i][1] * sh[0][i];
            w4 += v[i][0] * sh[2][i] - v[i][2] * sh[0][i];
            w5 += v[i][1] * sh[2][i] - v[i][2] * sh[1][i];
        }
        const double hdt = 0.5 * dt;
        w3 *= hdt, w4 *= hdt, w5 *= hdt;
        // s_out = s + dt * si(s, w) (jaumann3), bilinear in s and w
        const double d01 = g[1] - g[0], d02 = g[2] - g[0], d12 = g[2] - g[1];
        h3 = hdt * (2 * s[3] * d01 + (s[0] - s[1]) * g[3] - s[5] * g[4] + s[4] * g[5]);
        h4 = hdt * (2 * s[4] * d02 - s[5] * g[3] + (s[0] - s[2]) * g[4] + s[3] * g[5]);
        h5 = hdt * (2 * s[5] * d12 - s[4] * g[3] + s[3] * g[4] + (s[1] - s[2]) * g[5]);
        a.as[0 * ne + e] = g[0] + g[3] * w3 + g[4] * w4;
        a.as[1 * ne + e] = g[1] - g[3] * w3 + g[5] * w5;
        a.as[2 * ne + e] = g[2] - g[4] * w4 - g[5] * w5;
        a.as[3 * ne + e] = g[3] + 2 * w3 * d01 + g[4] * w5 + g[5] * w4;
        a.as[4 * ne + e] = g[4] + 2 * w4 * d02 - g[3] * w5 + g[5] * w3;
        a.as[5 * ne + e] = g[5] + 2 * w5 * d12 - g[3] * w4 - g[4] * w3;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        a.slot3[((size_t)0 * 4 + i) * ne + e] = h3 * sh[1][i] + h4 * sh[2][i];
        a.slot3[((size_t)1 * 4 + i) * ne + e] = h5 * sh[2][i] - h3 * sh[0][i];
        a.slot3[((size_t)2 * 4 + i) * ne + e] = -h4 * sh[0][i] - h5 * sh[1][i];
        gs[0][i] -= h3 * v[i][1] + h4 * v[i][2];
        gs[1][i] += h3 * v[i][0] - h5 * v[i][2];
        gs[2][i] += h4 * v[i][0] + h5 * v[i][1];
    }
    double gc[4][3];
    geom_reverse(sh, vol, gs, gvol, gc);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int d = 0; d < 3; ++d) a.slotx[((size_t)d * 4 + i) * ne + e] = gc[i][d];
}

int launch_adj_end_geometry(const KP &p, const AdjBufs &a, const TapeStep &t, const TapeStep &t1, double dt,
                            cudaStream_t s)
{
    DES_LAUNCH_W(k_adj_end_geometry, p.ne, s, p, a, t, t1, dt);
    return 1;
}

// derivative of the damped force with respect to the undamped one
// (fields.cxx:235-288); the force keeps the sign of the undamped force, and
// the velocity enters only through signs (derivative zero)
__device__ __forceinline__ double damp_deriv(const KP &p, double f, double v)
{
    const double df = p.prm.damping_factor;
    switch (p.prm.damping_option) {
    case 1:
        if (fabs(v) > 1e-13) {
            const double sf = (f > 0) ? 1.0 : ((f < 0) ? -1.0 : 0.0);
            return 1 - df * sf * ((v > 0) ? 1.0 : -1.0);
        }
        return 1;
    case 2: return 1 - df;
    case 3: return ((f < 0) == (v < 0)) ? (1 - df) : (2 - df);
    default: return 1;
    }
}

// ------------------------------------------------------------------
// nodes: gather the end-of-step contributions, then reverse
// update_coordinate (x' = x + v' dt), apply_vbcs (affine in v and the
// prescribed values: its transpose is read off by probing the forward map
// with unit vectors), update_velocity (v' = v + dt f / m), the elastic
// foundation and the damping.  Writes ax (coordinate adjoint, start of the
// step), av (velocity adjoint, before the strain-rate share), af (adjoint
// of the undamped force), am (mass adjoint of the start), clears atm and
// avn, and adds the sums of the prescribed-value adjoints to gvbc.
// ------------------------------------------------------------------
template <bool STAGED>
__global__ void __launch_bounds__(192) k_adj_motion(KP p, AdjBufs a, TapeStep t, TapeStep t1, double dt)
{
    const size_t ne = p.ne, nn = p.nn;
    double sum[6] = {};   // coordinate and velocity contributions
    const int n = node_sums<SumF64, 6, 3, STAGED>(
        p.sup_off, 0, p.nn, 6,
        [&](int q, double *s) {
            const int ent = p.sup_ent[q];
            const int e = ent >> 2, k = ent & 3;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                s[d] = a.slotx[((size_t)d * 4 + k) * ne + e];
                s[3 + d] = a.slot3[((size_t)d * 4 + k) * ne + e];
            }
        },
        [&](int c, int m) { return c < 3 ? a.ax[c * nn + m] : a.av[(c - 3) * nn + m]; }, sum);
    double gva[DES_NBDRYTYPES];
#pragma unroll
    for (int ib = 0; ib < DES_NBDRYTYPES; ++ib) gva[ib] = 0;
    const unsigned flag = n >= 0 ? p.bcflag[n] : 0u;
    if (n >= 0) {
        double gx[3] = {sum[0], sum[1], sum[2]}, gv[3] = {sum[3], sum[4], sum[5]};
        // x' = x + v' dt
#pragma unroll
        for (int d = 0; d < 3; ++d) gv[d] += dt * gx[d];
        // v' = BC(pre): gpre = A^T gv, gva = B^T gv
        double gpre[3] = {gv[0], gv[1], gv[2]};
        if (flag & BOUND_ANY) {
            // the three unit velocities, then a unit value of each of the
            // node's own boundaries (its BCs read no others'): one copy of
            // the BC code, which a small mesh's launch otherwise spends its
            // time fetching
#pragma unroll 1
            for (int q = 0; q < 3 + DES_NBDRYTYPES; ++q) {
                if (q >= 3 && !(flag & (1u << (q - 3)))) continue;
                double col[3], val[DES_NBDRYTYPES];
#pragma unroll
                for (int d = 0; d < 3; ++d) col[d] = d == q ? 1.0 : 0.0;
#pragma unroll
                for (int ib = 0; ib < DES_NBDRYTYPES; ++ib) val[ib] = ib + 3 == q ? 1.0 : 0.0;
                apply_vbcs_node_va<3>(p, flag, col, val);
                const double r = col[0] * gv[0] + col[1] * gv[1] + col[2] * gv[2];
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    if (d == q) gpre[d] = r;
#pragma unroll
                for (int ib = 0; ib < DES_NBDRYTYPES; ++ib)
                    if (ib + 3 == q) gva[ib] = r;
            }
        }
        const double im = recip_newton(t.mass[n]);
        double gm = 0, gf[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double f = t.f[d * nn + n];
            a.av[d * nn + n] = gpre[d];
            gf[d] = dt * gpre[d] * im;
            gm -= gf[d] * f * im;
            double dd = 1;
            if (p.prm.is_quasi_static) dd = damp_deriv(p, f, t.v[d * nn + n]);
            gf[d] *= dd;
            a.af[d * nn + n] = gf[d];
        }
        if (p.prm.has_elastic_foundation && (flag & BOUNDZ0)) gx[2] -= p.prm.elastic_foundation_constant * gf[2];
#pragma unroll
        for (int d = 0; d < 3; ++d) a.ax[d * nn + n] = gx[d];
        a.am[n] = gm;
        a.atm[n] = 0;
        a.avn[n] = 0;
    }
    // fixed-order sums of the prescribed-value adjoints over the warp's nodes
    if (!__any_sync(0xffffffffu, flag & BOUND_ANY)) return;
    const size_t part = STAGED ? blockIdx.x : (blockIdx.x * blockDim.x + threadIdx.x) / 32;
#pragma unroll
    for (int ib = 0; ib < DES_NBDRYTYPES; ++ib) {
        double g = gva[ib];
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) g += __shfl_down_sync(0xffffffffu, g, w);
        if ((threadIdx.x & 31) == 0) a.gvbc[part * DES_NBDRYTYPES + ib] += g;
    }
}

int launch_adj_motion(const KP &p, const AdjBufs &a, const TapeStep &t, const TapeStep &t1, double dt,
                      cudaStream_t s)
{
    DES_NODES(k_adj_motion<STAGED>, p.nn, s, p, a, t, t1, dt);
    return 1;
}

int adj_vbc_parts(const KP &p)
{
    const int nodes = node_staged(p, p.nn) ? NPB : 32;   // a block's, or a warp's
    return (p.nn + nodes - 1) / nodes;
}

// ------------------------------------------------------------------
// stress BCs of one boundary facet (bc.cxx:493-566), reversed.  The facet
// force fv = pr(zcenter, rho) * normal / 3 is subtracted at each of the
// facet's nodes, so its adjoint is minus the sum of their force adjoints.
// Writes the coordinate adjoints of the facet's three nodes to fslot and
// the element density adjoint (Winkler foundation) to frho.
// ------------------------------------------------------------------
__global__ void __launch_bounds__(TPB_A) k_adj_facets(KP p, AdjBufs a, TapeStep t)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= p.nbf) return;
    const size_t nn = p.nn, nbf = p.nbf;
    const int i = p.fac_bdry[q];
    const int ty = p.prm.vbc_types[i];
    const bool active = p.prm.gravity != 0 && (ty == 0 || ty == 2 || ty == 4) &&
                        !(i == 4 && !p.prm.has_winkler_foundation) && !(i == 5 && !p.prm.has_water_loading);
    double gc[3][3] = {};
    double grho = 0;
    if (active) {
        const int e = p.fac_elem[q], f = p.fac_f[q];
        const int F[4][3] = {{1, 2, 3}, {0, 3, 2}, {0, 1, 3}, {0, 2, 1}};
        int nd[3];
        double c[3][3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            nd[j] = conn_at(p, F[f][j], e);
            tload3(t.x, nn, nd[j], c[j]);
        }
        double gfv[3];
#pragma unroll
        for (int d = 0; d < 3; ++d)
            gfv[d] = -(a.af[d * nn + nd[0]] + a.af[d * nn + nd[1]] + a.af[d * nn + nd[2]]);
        double va[3], vb[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            va[d] = c[1][d] - c[0][d];
            vb[d] = c[2][d] - c[0][d];
        }
        const double nrm[3] = {(va[1] * vb[2] - va[2] * vb[1]) / 2, (va[2] * vb[0] - va[0] * vb[2]) / 2,
                               (va[0] * vb[1] - va[1] * vb[0]) / 2};
        const double zc = div3(c[0][2] + c[1][2] + c[2][2]);
        double pr, gzc_per_gpr, grho_per_gpr = 0;
        if (i == 4 && p.prm.has_winkler_foundation) {
            const double rho = t.rho[e];
            pr = p.prm.compensation_pressure - (rho + p.prm.winkler_delta_rho) * p.prm.gravity * (zc + p.prm.zlength);
            gzc_per_gpr = -(rho + p.prm.winkler_delta_rho) * p.prm.gravity;
            grho_per_gpr = -p.prm.gravity * (zc + p.prm.zlength);
        } else if (i == 5 && p.prm.has_water_loading) {
            pr = (zc < 0) ? 1030 * p.prm.gravity * (0 - zc) : 0;
            gzc_per_gpr = (zc < 0) ? -1030 * p.prm.gravity : 0;
        } else {
            pr = ref_pressure_(p, zc);
            gzc_per_gpr = -p.mat.rho0[0] * p.prm.gravity;
        }
        double gpr = 0, gn[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            gpr += div3(gfv[d] * nrm[d]);
            gn[d] = div3(gfv[d] * pr);
        }
        grho = gpr * grho_per_gpr;
        const double gzc = gpr * gzc_per_gpr;
        const double ga[3] = {(-gn[1] * vb[2] + gn[2] * vb[1]) / 2, (gn[0] * vb[2] - gn[2] * vb[0]) / 2,
                              (-gn[0] * vb[1] + gn[1] * vb[0]) / 2};
        const double gb[3] = {(gn[1] * va[2] - gn[2] * va[1]) / 2, (-gn[0] * va[2] + gn[2] * va[0]) / 2,
                              (gn[0] * va[1] - gn[1] * va[0]) / 2};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            gc[0][d] = -ga[d] - gb[d];
            gc[1][d] = ga[d];
            gc[2][d] = gb[d];
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) gc[j][2] += div3(gzc);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int j = 0; j < 3; ++j) a.fslot[((size_t)d * 3 + j) * nbf + q] = gc[j][d];
    a.frho[q] = grho;
}

// ------------------------------------------------------------------
// update_force element terms (fields.cxx:291-340), reversed: per element,
// the four nodes' undamped force adjoints give the adjoints of the NMD
// stress, the start shape functions and volume, and the element density
// (buoyancy; Winkler facets from frho).  Also the first half of NMD_stress
// reversed (geometry.cxx:182-236): the trace of the stress adjoint feeds
// dp directly and, through the nodal average, every node of the element.
// Out: as (stress after update_stress), ashp and avol (start of the step;
// avol also takes the adjoint of volume_old of the next state), arho,
// adp (direct part), slot1[e] = the element's share of the NMD nodal sum.
// ------------------------------------------------------------------
__global__ void __launch_bounds__(TPB_A) k_adj_force(KP p, AdjBufs a, TapeStep t)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= p.ne) return;
    const size_t ne = p.ne, nn = p.nn;
    double s[6], gsig[6];
    tape_sss(p, t, e, s);
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) gsig[cc] = a.as[cc * ne + e];
    const double vol = t.vol[e];
    const double gravity = p.prm.gravity;
    const double buoy = (gravity != 0) ? t.rho[e] * gravity / 4 : 0.0;
    double gvol = a.avolo[e];
    a.avolo[e] = 0;
    double grho = a.arho[e];
    for (int q = a.e2f_off[e]; q < a.e2f_off[e + 1]; ++q) grho += a.frho[a.e2f_ent[q]];
    // with F_lk = sum_i gf_i,l dN_i/dx_k over the nodes' force adjoints: the
    // volume's adjoint is -(sigma : F + buoy sum gf_z), the stress's -vol sym(F)
    // and dN_i/dx_k's -vol sum_l gf_i,l sigma_lk
    double F[3][3] = {}, sv[6], fz = 0;
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) sv[cc] = -vol * s[cc];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        double gf[3];
        tload3(a.af, nn, conn_at(p, i, e), gf);
        const double sh[3] = {tshp(t, ne, 0, i, e), tshp(t, ne, 1, i, e), tshp(t, ne, 2, i, e)};
#pragma unroll
        for (int l = 0; l < 3; ++l)
#pragma unroll
            for (int k = 0; k < 3; ++k) F[l][k] += gf[l] * sh[k];
        a.ashp[((size_t)0 * 4 + i) * ne + e] = gf[0] * sv[0] + gf[1] * sv[3] + gf[2] * sv[4];
        a.ashp[((size_t)1 * 4 + i) * ne + e] = gf[0] * sv[3] + gf[1] * sv[1] + gf[2] * sv[5];
        a.ashp[((size_t)2 * 4 + i) * ne + e] = gf[0] * sv[4] + gf[1] * sv[5] + gf[2] * sv[2];
        fz += gf[2];
    }
    const double f3 = F[0][1] + F[1][0], f4 = F[0][2] + F[2][0], f5 = F[1][2] + F[2][1];
    gvol -= s[0] * F[0][0] + s[1] * F[1][1] + s[2] * F[2][2] + s[3] * f3 + s[4] * f4 + s[5] * f5 + buoy * fz;
    gsig[0] -= vol * F[0][0];
    gsig[1] -= vol * F[1][1];
    gsig[2] -= vol * F[2][2];
    gsig[3] -= vol * f3;
    gsig[4] -= vol * f4;
    gsig[5] -= vol * f5;
    if (gravity != 0) grho -= vol * fz * gravity / 4;
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) a.as[cc * ne + e] = gsig[cc];
    a.avol[e] = gvol;
    a.arho[e] = grho;
    // NMD: stress_ii += (-dp + mean_i dpn_i) / 3
    const double tr = gsig[0] + gsig[1] + gsig[2];
    a.adp[e] = -div3(tr);
    a.slot1[e] = div3(tr) / 4;
}

// nodes: NMD nodal sum reversed (dpn = sum_e dp_e vol_e / volume_n), and the
// facets' coordinate adjoints added to ax.  On a small mesh a boundary node's
// walk over its facets, a chain of dependent loads, was most of the kernel:
// as a sum of its own, staged side by side, 16 -> 11 us at 14,400 tets.
template <bool STAGED>
__global__ void __launch_bounds__(192) k_adj_nmd_nodes(KP p, AdjBufs a, TapeStep t)
{
    const size_t nn = p.nn, nbf = p.nbf;
    double acc, gx[3];
    node_sums<SumF64, 3, 3, STAGED>(
        p.nf_off, 0, p.nn, 3,
        [&](int k, double *s) {
            const int ent = p.nf_ent[k];
#pragma unroll
            for (int d = 0; d < 3; ++d) s[d] = a.fslot[((size_t)d * 3 + (ent & 3)) * nbf + (ent >> 2)];
        },
        FromZero<SumF64>(), gx);
    const int n = node_sums<SumF64, 1, 3, STAGED>(
        p.sup_off, 0, p.nn, 1, [&](int q, double *s) { *s = a.slot1[p.sup_ent[q] >> 2]; }, FromZero<SumF64>(), &acc);
    if (n < 0) return;
    const double ivn = recip_newton(t.voln[n]);
    a.adpn[n] = acc * ivn;
    a.avn[n] -= acc * t.dpn[n] * ivn;
    // the facets' coordinate adjoints
    if (p.nf_off[n] < p.nf_off[n + 1])
#pragma unroll
        for (int d = 0; d < 3; ++d) a.ax[d * nn + n] += gx[d];
}

int launch_adj_force(const KP &p, const AdjBufs &a, const TapeStep &t, cudaStream_t s)
{
    int n = 0;
    if (p.nbf > 0) {
        DES_LAUNCH(k_adj_facets, p.nbf, s, p, a, t);
        ++n;
    }
    DES_LAUNCH_W(k_adj_force, p.ne, s, p, a, t);
    return n + 1;
}

int launch_adj_nmd_nodes(const KP &p, const AdjBufs &a, const TapeStep &t, cudaStream_t s)
{
    DES_NODES(k_adj_nmd_nodes<STAGED>, p.nn, s, p, a, t);
    return 1;
}

// ------------------------------------------------------------------
// rheology, reversed (rheology.cxx:105-299, matprops.cxx:264-373).  Each
// *_reverse adds to the adjoints it is given; forward values are recomputed
// with the forward's own functions, so every branch matches the forward.
// ------------------------------------------------------------------
// elastic: out = s + E(de), out_i = s_i + 2G de_i + (K - 2G/3) tr(de), out_c = s_c + 2G de_c
__device__ __forceinline__ void elastic_reverse(double K, double G, const double *de, const double *go, double *gs,
                                                double *gde, double &gG)
{
    const double lambda = K - 2. / 3 * G;
    const double trde = de[0] + de[1] + de[2], tg = go[0] + go[1] + go[2];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        gs[i] += go[i];
        gde[i] += 2 * G * go[i] + lambda * tg;
        gG += 2 * de[i] * go[i];
    }
    gG -= 2. / 3 * trde * tg;
#pragma unroll
    for (int c = 3; c < 6; ++c) {
        gs[c] += go[c];
        gde[c] += 2 * G * go[c];
        gG += 2 * de[c] * go[c];
    }
}

// maxwell: out_i = ((s_i - s0) f1 + 2G (de_i - dev)) f2 + s0 + K dv, out_c = (s_c f1 + 2G de_c) f2,
// f1 = 1 - tmp, f2 = 1 / (1 + tmp), tmp = dt G / (2 visc)
__device__ __forceinline__ void maxwell_reverse(double K, double G, double visc, double dt, const double *de,
                                                const double *s, const double *go, double *gs, double *gde,
                                                double &gG, double &gvisc, double &gdv)
{
    // with the deviators x = s - s0, y = de - dev: out = (x f1 + 2G y) f2 (+ s0 + K dv)
    const double ivisc = recip_newton(visc);
    const double tmp = 0.5 * dt * G * ivisc;
    const double f1 = 1 - tmp, f2 = recip_newton(1 + tmp);
    const double dev = div3(de[0] + de[1] + de[2]), s0 = div3(s[0] + s[1] + s[2]);
    const double c = f1 * f2, d = 2 * G * f2;
    double A = 0, B = 0;   // <go, x>, <go, y>
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        A += go[i] * (s[i] - s0);
        B += go[i] * (de[i] - dev);
    }
#pragma unroll
    for (int k = 3; k < 6; ++k) {
        A += go[k] * s[k];
        B += go[k] * de[k];
    }
    const double tg = go[0] + go[1] + go[2], tg3 = div3(tg);
    gdv += K * tg;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        gs[i] += c * go[i] + (tg3 - c * tg3);
        gde[i] += d * (go[i] - tg3);
    }
#pragma unroll
    for (int k = 3; k < 6; ++k) {
        gs[k] += c * go[k];
        gde[k] += d * go[k];
    }
    const double gtmp = -f2 * A - (f1 * A + 2 * G * B) * f2 * f2;
    gG += 2 * f2 * B + gtmp * 0.5 * dt * ivisc;
    gvisc -= gtmp * tmp * ivisc;
}

// MatProps::visc for one material without markers, at an explicit mean
// temperature T (the forward reads it from the nodes at that time)
__device__ double visc_eval(const KP &p, int e, const double *edot, double T, double &raw, double &ed)
{
    ed = 0;
    if (p.ef[DES_EF_LOG10_VISC]) {
        raw = pow(10.0, p.ef[DES_EF_LOG10_VISC][e]);
    } else {
        const double gas_constant = 8.3144;
        ed = dmax_(second_invariant_<3>(edot), 1e-30);
        const double visc0 = 0.25 * pow(ed, p.mat.visc_pw[0]) * p.mat.visc_coef[0]
            * exp(p.mat.visc_activation_energy[0] / (p.mat.visc_exponent[0] * gas_constant * T)) * 1e6;
        raw = 1 / (1 / visc0);
    }
    return dmin_(dmax_(raw, p.mat.visc_min), p.mat.visc_max);
}

// adjoint of the viscosity -> strain rate (corrected), mean temperature, log10
// viscosity; raw is the unclamped viscosity and ed the strain-rate invariant
// of visc_eval for the same element (ed < 0: not known yet)
__device__ void visc_reverse(const KP &p, int e, const double *edot, double T, double raw, double ed, double gvisc,
                             double *gedot, double &gT, double &glv)
{
    if (!(raw > p.mat.visc_min && raw < p.mat.visc_max)) return;   // clamped: no sensitivity
    if (p.ef[DES_EF_LOG10_VISC]) {
        glv += gvisc * raw * 2.302585092994046;   // d 10^x / dx = 10^x ln 10
        return;
    }
    const double gas_constant = 8.3144;
    const double q = p.mat.visc_activation_energy[0] / (p.mat.visc_exponent[0] * gas_constant);
    const double iT = recip_newton(T);
    gT -= gvisc * raw * q * iT * iT;
    if (ed < 0) ed = dmax_(second_invariant_<3>(edot), 1e-30);   // as visc_eval forms it
    if (ed > 1e-30) {
        const double ied = recip_newton(ed);
        const double ged = gvisc * raw * p.mat.visc_pw[0] * ied;
        const double gj2 = 0.5 * ged * ied;
        const double a = div3(edot[0] + edot[1] + edot[2]);
#pragma unroll
        for (int i = 0; i < 3; ++i) gedot[i] += gj2 * (edot[i] - a);
#pragma unroll
        for (int c = 3; c < 6; ++c) gedot[c] += gj2 * 2 * edot[c];
    }
}

// MatProps::plastic_weakening + plastic_props for one material without
// markers, reversed from the adjoints of (amc, anphi, anpsi, hardn,
// ten_max) to the per-element cohesion and friction angles and plstrain
__device__ void plastic_props_reverse(const KP &p, int e, double pls, double gamc, double ganphi, double ganpsi,
                                      double ghardn, double gtmax, double *gpar, double &gpls)
{
    // an element whose return map was inactive passes zero adjoints: its
    // contributions below are all zero, and the transcendentals are skipped
    if (gamc == 0 && ganphi == 0 && ganpsi == 0 && ghardn == 0 && gtmax == 0) return;
    const double c0 = p.ef[DES_EF_COHESION0] ? p.ef[DES_EF_COHESION0][e] : p.mat.cohesion0[0];
    const double c1 = p.ef[DES_EF_COHESION1] ? p.ef[DES_EF_COHESION1][e] : p.mat.cohesion1[0];
    const double f0 = p.ef[DES_EF_FRICTION0] ? p.ef[DES_EF_FRICTION0][e] : p.mat.friction_angle0[0];
    const double f1 = p.ef[DES_EF_FRICTION1] ? p.ef[DES_EF_FRICTION1][e] : p.mat.friction_angle1[0];
    const double d0 = p.mat.dilation_angle0[0], d1 = p.mat.dilation_angle1[0];
    const double l0 = p.mat.pls0[0], l1 = p.mat.pls1[0];
    int seg;
    double q = 0, c, phi, psi;
    if (pls < l0) {
        seg = 0;
        c = c0; phi = f0; psi = d0;
    } else if (pls < l1) {
        seg = 1;
        q = (pls - l0) / (l1 - l0);
        c = c0 + q * (c1 - c0); phi = f0 + q * (f1 - f0); psi = d0 + q * (d1 - d0);
    } else {
        seg = 2;
        c = c1; phi = f1; psi = d1;
    }
    const double sphi = sin(phi * DEG2RAD), spsi = sin(psi * DEG2RAD);
    const double anphi = (1 + sphi) / (1 - sphi);
    const double sq = sqrt(anphi), tn = tan(phi * DEG2RAD);
    double gc = 2 * sq * gamc;
    ganphi += 2 * c * gamc / (2 * sq);
    double gtn = 0;
    if (phi != 0 && c / tn < p.mat.tension_max) {
        gc += gtmax / tn;
        gtn = -gtmax * c / (tn * tn);
    }
    const double gphi = ganphi * 2 / ((1 - sphi) * (1 - sphi)) * cos(phi * DEG2RAD) * DEG2RAD
        + gtn * (1 + tn * tn) * DEG2RAD;
    const double gpsi = ganpsi * 2 / ((1 - spsi) * (1 - spsi)) * cos(psi * DEG2RAD) * DEG2RAD;
    if (seg == 0) {
        gpar[DES_EF_COHESION0] += gc;
        gpar[DES_EF_FRICTION0] += gphi;
    } else if (seg == 1) {
        const double il = 1 / (l1 - l0);
        gpar[DES_EF_COHESION0] += gc * (1 - q) - ghardn * il;
        gpar[DES_EF_COHESION1] += gc * q + ghardn * il;
        gpar[DES_EF_FRICTION0] += gphi * (1 - q);
        gpar[DES_EF_FRICTION1] += gphi * q;
        gpls += (gc * (c1 - c0) + gphi * (f1 - f0) + gpsi * (d1 - d0)) * il;
    } else {
        gpar[DES_EF_COHESION1] += gc;
        gpar[DES_EF_FRICTION1] += gphi;
    }
}

// Mohr-Coulomb return map in principal space (rheology.cxx:163-299),
// reversed.  S' = sum_k (p_k - alpha c_k) v_k v_k^T = S - alpha M.  With G_o
// the symmetric matrix of the output adjoint and g_ab = v_a^T G_o v_b, the
// adjoint of the trial stress is
//   H = G_o + sum_k dp_k v_k v_k^T - sum_{a<b} g_ab alpha (c_a - c_b) / (p_a - p_b) (v_a v_b^T + v_b v_a^T),
// (first-order perturbation of the eigenvalues, v_k^T dS v_k, and of the
// eigenprojectors), dp_k being the eigenvalue adjoints that alpha's
// dependence on the principal stresses contributes.  The identity part is
// applied directly: the analytic eigenvectors of near-repeated principal
// stresses are not orthonormal to working precision, so only the plastic
// correction goes through them, and an element that does not yield takes
// the identity exactly.  When p_a and p_b (nearly) coincide the eigenbasis,
// and with it the direction of the correction, is discontinuous in S: the
// term of that pair is dropped (a subgradient).
__device__ void mc_return_reverse(double K, double G, double amc, double anphi, double anpsi, double hardn,
                                  double tmax, const double *S, const double *go, double gdepls, double *gS,
                                  double &gG, double &gamc, double &ganphi, double &ganpsi, double &ghardn,
                                  double &gtmax)
{
    if (clearly_elastic3(amc, anphi, tmax, S)) {   // S' = S (the forward skipped the eigen-solve too)
#pragma unroll
        for (int cc = 0; cc < 6; ++cc) gS[cc] += go[cc];
        return;
    }
    double pr[3], v[3][3];
    principal_stresses3(S, pr, v);
    const double fs = pr[0] - pr[2] * anphi + amc;
    const double ft = pr[2] - tmax;
    double alpha = 0, c[3] = {0, 0, 0}, r = 0, D = 1;
    bool yield = !(fs > 0 && ft < 0), shear = false;
    const double a1 = K + 4. / 3 * G, a2 = K - 2. / 3 * G;
    if (!yield) {   // S' = S
#pragma unroll
        for (int cc = 0; cc < 6; ++cc) gS[cc] += go[cc];
        return;
    }
    {
        const double pa = sqrt(1 + anphi * anphi) + anphi;
        const double ps = tmax * anphi - amc;
        const double h = pr[2] - tmax + pa * (pr[0] - ps);
        shear = h < 0;
        if (shear) {
            D = a1 - a2 * anpsi + a1 * anphi * anpsi - a2 * anphi + 2 * sqrt(anphi) * hardn;
            alpha = fs / D;
            c[0] = a1 - a2 * anpsi;
            c[1] = a2 - a2 * anpsi;
            c[2] = a2 - a1 * anpsi;
            r = sqrt((7 + 4 * anpsi + 7 * anpsi * anpsi) / 18);
        } else {
            alpha = ft / a1;
            c[0] = a2;
            c[1] = a2;
            c[2] = a1;
            r = sqrt(7. / 18);
        }
    }
    // G_o and its eigenbasis components
    const double Go[3][3] = {{go[0], go[3] / 2, go[4] / 2}, {go[3] / 2, go[1], go[5] / 2}, {go[4] / 2, go[5] / 2, go[2]}};
    double gv[3][3];   // G_o v_k
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int m = 0; m < 3; ++m) gv[m][k] = Go[m][0] * v[0][k] + Go[m][1] * v[1][k] + Go[m][2] * v[2][k];
    double g[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b) g[a][b] = v[0][a] * gv[0][b] + v[1][a] * gv[1][b] + v[2][a] * gv[2][b];
    double pb[3] = {g[0][0], g[1][1], g[2][2]};   // adjoints of p'_k, then of p_k
    double w[3][3] = {};   // projector terms beyond the identity
    const double scale = fabs(pr[0]) + fabs(pr[1]) + fabs(pr[2]) + 1e-300;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = a + 1; b < 3; ++b) {
            const double gap = pr[a] - pr[b];
            if (c[a] != c[b] && fabs(gap) > 1e-12 * scale) w[a][b] = -g[a][b] * alpha * (c[a] - c[b]) / gap;
        }
    {
        double galpha = -(pb[0] * c[0] + pb[1] * c[1] + pb[2] * c[2]);
        galpha += gdepls * ((alpha > 0) ? r : ((alpha < 0) ? -r : 0.0));
        double gc[3] = {-alpha * pb[0], -alpha * pb[1], -alpha * pb[2]};
        double ga1 = 0, ga2 = 0;
        if (shear) {
            const double gfs = galpha / D, gD = -galpha * alpha / D;
            pb[0] += gfs;
            pb[2] -= anphi * gfs;
            ganphi -= pr[2] * gfs;
            gamc += gfs;
            const double sqa = sqrt(anphi);
            ga1 += gD * (1 + anphi * anpsi);
            ga2 += gD * (-anpsi - anphi);
            ganpsi += gD * (-a2 + a1 * anphi);
            ganphi += gD * (a1 * anpsi - a2 + hardn / sqa);
            ghardn += gD * 2 * sqa;
            ga1 += gc[0] - gc[2] * anpsi;
            ga2 += -gc[0] * anpsi + gc[1] * (1 - anpsi) + gc[2];
            ganpsi += -gc[0] * a2 - gc[1] * a2 - gc[2] * a1;
            if (alpha != 0) ganpsi += gdepls * fabs(alpha) * (4 + 14 * anpsi) / (36 * r);
        } else {
            const double gft = galpha / a1;
            ga1 -= galpha * alpha / a1;
            pb[2] += gft;
            gtmax -= gft;
            ga2 += gc[0] + gc[1];
            ga1 += gc[2];
        }
        gG += ga1 * 4. / 3 - ga2 * 2. / 3;
    }
    // H - G_o in components (diagonal H_mm, off-diagonal 2 H_mn), plus G_o
    const double dpb[3] = {pb[0] - g[0][0], pb[1] - g[1][1], pb[2] - g[2][2]};
    const int cm[6] = {0, 1, 2, 0, 0, 1}, cn[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) {
        const int m = cm[cc], n = cn[cc];
        double h = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) h += dpb[k] * v[m][k] * v[n][k];
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = a + 1; b < 3; ++b) h += w[a][b] * (v[m][a] * v[n][b] + v[m][b] * v[n][a]);
        gS[cc] += go[cc] + ((cc < 3) ? h : 2 * h);
    }
}

// ------------------------------------------------------------------
// update_stress (rheology.cxx:510-646) of one element, reversed, plus the
// second half of NMD_stress (the dp adjoint gathered from the element's
// nodes) and the element density rho(T) of the step.
// In: as = adjoint of the stress after update_stress, apls = of plstrain
// after the step, adp/adpn/arho/avol.  Out: as, apls = adjoints at the
// start of the step; aedot = adjoint of the strain rate before the
// anti-locking correction; aedv; avol, avolo; slot1 = T' contributions of
// the four nodes; g += the parameter gradients of the element.
// ------------------------------------------------------------------
__global__ void __launch_bounds__(TPB_A) k_adj_stress(KP p, AdjBufs a, TapeStep t, TapeStep t1, double dt)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= p.ne) return;
    const size_t ne = p.ne;
    int nodes[4];
    double sacc = 0, Tsum = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        nodes[i] = conn_at(p, i, e);
        sacc += a.adpn[nodes[i]];
        Tsum += t1.T[nodes[i]];
    }
    const double T = Tsum / 4;   // elem_avg_T of the updated temperature
    const double vol = t.vol[e], volo = t.volo[e];
    const double gdp = a.adp[e] + vol * sacc;
    double gvol = a.avol[e] + t.dp[e] * sacc, gvolo = 0;
    double s0[6], edot[6], go[6];
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) {
        s0[cc] = t.s[cc * ne + e];
        edot[cc] = t.edot[cc * ne + e];
        go[cc] = a.as[cc * ne + e];
    }
    const double pls = t.pls[e];
    // anti-locking correction (rheology.cxx:527-534) and increments
    {
        const double div = edot[0] + edot[1] + edot[2];
        const double corr = divnd<3>(t.edv[e] - div);
#pragma unroll
        for (int i = 0; i < 3; ++i) edot[i] += corr;
    }
    double de[6];
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) de[cc] = edot[cc] * dt;
    const double K = m_bulkm(p, e), G = m_shearm(p, e);
    // dp = tr(s_out) - tr(s0)
#pragma unroll
    for (int i = 0; i < 3; ++i) go[i] += gdp;
    double gs[6] = {-gdp, -gdp, -gdp, 0, 0, 0};
    double gde[6] = {0, 0, 0, 0, 0, 0}, gec[6] = {0, 0, 0, 0, 0, 0};
    double gG = 0, gvisc = 0, gdv = 0, gT = 0, glv = 0, gpls_props = 0;
    double gpar[DES_EF_COUNT] = {};
    const int rt = p.mat.rheol_type;
    // the viscosity and the EVP branch: the forward recompute's, from the
    // tape (else evaluated again, as the forward does)
    double visc = 0, raw = 0, ed = -1;
    const bool viscous = (rt & DES_RH_VISCOUS) != 0;
    if (viscous) {
        if (t.visc) raw = visc = t.visc[e];   // unclamped: raw == visc; clamped: no sensitivity either way
        else visc = visc_eval(p, e, edot, T, raw, ed);
    }
    if (rt == DES_RH_ELASTIC) {
        elastic_reverse(K, G, de, go, gs, gde, gG);
    } else if (rt == DES_RH_MAXWELL) {
        maxwell_reverse(K, G, visc, dt, de, s0, go, gs, gde, gG, gvisc, gdv);
    } else {   // EP or EVP
        double amc, anphi, anpsi, hardn, tmax;
        bool plastic = true;
        if (rt == DES_RH_EVP) {
            if (t.evp) {
                plastic = t.evp[e] != 0;
            } else {
                m_plastic_props(p, e, pls, amc, anphi, anpsi, hardn, tmax);
                const double dv = vol / volo - 1;
                double sv[6], sp[6];
#pragma unroll
                for (int cc = 0; cc < 6; ++cc) sv[cc] = sp[cc] = s0[cc];
                elastic_<3>(K, G, de, sp);
                maxwell_<3>(K, G, visc, dt, dv, de, sv);
                double depls;
                if (!clearly_elastic3(amc, anphi, tmax, sp))
                    mc_return_<3>(K, G, amc, anphi, anpsi, hardn, tmax, depls, sp);
                plastic = !(second_invariant2_<3>(sv) < second_invariant2_<3>(sp));
            }
        }
        if (plastic) {
            m_plastic_props(p, e, pls, amc, anphi, anpsi, hardn, tmax);
            double S[6];   // the elastic trial stress
#pragma unroll
            for (int cc = 0; cc < 6; ++cc) S[cc] = s0[cc];
            elastic_<3>(K, G, de, S);
            double gS[6] = {0, 0, 0, 0, 0, 0};
            double gamc = 0, ganphi = 0, ganpsi = 0, ghardn = 0, gtmax = 0;
            mc_return_reverse(K, G, amc, anphi, anpsi, hardn, tmax, S, go, a.apls[e], gS, gG, gamc, ganphi, ganpsi,
                              ghardn, gtmax);
            elastic_reverse(K, G, de, gS, gs, gde, gG);
            plastic_props_reverse(p, e, pls, gamc, ganphi, ganpsi, ghardn, gtmax, gpar, gpls_props);
        } else {
            maxwell_reverse(K, G, visc, dt, de, s0, go, gs, gde, gG, gvisc, gdv);
        }
    }
    if (viscous && gvisc != 0) visc_reverse(p, e, edot, T, raw, ed, gvisc, gec, gT, glv);
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) gec[cc] += dt * gde[cc];
    const double ivo = recip_newton(volo);
    gvol += gdv * ivo;
    gvolo -= gdv * vol * ivo * ivo;
    // corrected strain rate -> strain rate before the correction, edvoldt
    const double tg = gec[0] + gec[1] + gec[2];
#pragma unroll
    for (int i = 0; i < 3; ++i) a.aedot[i * ne + e] = gec[i] - div3(tg);
#pragma unroll
    for (int cc = 3; cc < 6; ++cc) a.aedot[cc * ne + e] = gec[cc];
    a.aedv[e] = div3(tg);
    // element density of the step: rho0 (1 - alpha (T - 273))
    gT += a.arho[e] * (-p.mat.rho0[0] * p.mat.alpha[0]);
#pragma unroll
    for (int i = 0; i < 4; ++i) a.slot1[(size_t)i * ne + e] = gT / 4;
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) a.as[cc * ne + e] = gs[cc];
    a.apls[e] += gpls_props;
    a.avol[e] = gvol;
    a.avolo[e] = gvolo;
    gpar[DES_EF_LOG10_VISC] += glv;
    gpar[DES_EF_SHEAR_MODULUS] += gG;
#pragma unroll
    for (int k = 0; k < DES_EF_COUNT; ++k)
        if (gpar[k] != 0) a.g[(size_t)k * ne + e] += gpar[k];
}

// nodes: adjoint of the updated temperature (state + the stress kernel's
// T' terms), nodal dvoldt (ntmp = sum_e tr(edot) vol / volume_n, edvoldt =
// mean of ntmp), and the temperature update with its Dirichlet BCs
// (fields.cxx:151-162): T' = T - tdot dt / tmass
template <bool STAGED>
__global__ void __launch_bounds__(192) k_adj_nodes_heat(KP p, AdjBufs a, TapeStep t, TapeStep t1, double dt)
{
    const size_t ne = p.ne;
    double sum[2];   // adjoints of the updated temperature and of dvoldt
    const int n = node_sums<SumF64, 2, 3, STAGED>(
        p.sup_off, 0, p.nn, 2,
        [&](int q, double *s) {
            const int ent = p.sup_ent[q];
            const int e = ent >> 2, k = ent & 3;
            s[0] = a.slot1[(size_t)k * ne + e];
            s[1] = a.aedv[e] / 4;
        },
        [&](int c, int m) { return c == 0 ? a.aT[m] : 0.0; }, sum);
    if (n < 0) return;
    const double gTp = sum[0], gnt = sum[1];
    const double ivn = 1 / t.voln[n];
    a.antmp[n] = gnt * ivn;
    a.avn[n] -= gnt * t.ntmp[n] * ivn;
    double gT = gTp, gtd = 0;
    if (p.prm.has_thermal_diffusion) {
        const unsigned flag = p.bcflag[n];
        if ((flag & BOUNDZ1) || ((flag & BOUNDZ0) && !p.prm.has_fixed_bottom_temperature)) {
            gT = 0;
        } else {
            gtd = -gTp * dt * (1 / t.tmass[n]);
            a.atm[n] -= gtd * t.tdot[n] * (1 / t.tmass[n]);
        }
    }
    a.aT[n] = gT;
    a.atdot[n] = gtd;
}

// elements: dvoldt terms, the heat stencil (fields.cxx:99-146) and the
// strain rate (fields.cxx:166-232), reversed, at the start of the step.
// Out: ashp, avol (+=), slot3 = velocity contributions, slot1 = temperature
// contributions, g[therm_cond].
__global__ void __launch_bounds__(TPB_A) k_adj_kinematics(KP p, AdjBufs a, TapeStep t)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= p.ne) return;
    const size_t ne = p.ne, nn = p.nn;
    int nodes[4];
    double sh[3][4], gsh[3][4], v[4][3];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        nodes[i] = conn_at(p, i, e);
        tload3(t.v, nn, nodes[i], v[i]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            sh[k][i] = tshp(t, ne, k, i, e);
            gsh[k][i] = a.ashp[((size_t)k * 4 + i) * ne + e];
        }
    }
    const double vol = t.vol[e];
    double gvol = a.avol[e];
    double g[6];
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) g[cc] = a.aedot[cc * ne + e];
    // dvoldt: sum_e tr(edot) vol
    {
        double sant = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) sant += a.antmp[nodes[i]];
        const double tr = t.edot[e] + t.edot[ne + e] + t.edot[2 * ne + e];
#pragma unroll
        for (int i = 0; i < 3; ++i) g[i] += vol * sant;
        gvol += tr * sant;
    }
    double gTn[4] = {0, 0, 0, 0};
    if (p.prm.has_thermal_diffusion) {
        // tdot_i = kv g_i . G - rh with the temperature gradient G = sum_j g_j
        // (T_j - T_0) (the gradients sum to zero): with U = sum_i gtd_i g_i,
        // the adjoints are U . G of kv, kv g_j . U of T_j and kv (gtd_m G +
        // (T_m - T_0) U) of g_m (a common change of the g_m does not occur)
        double Td[4], gtd[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            Td[i] = t.T[nodes[i]];
            gtd[i] = a.atdot[nodes[i]];
        }
        const double T0 = Td[0];
#pragma unroll
        for (int i = 0; i < 4; ++i) Td[i] -= T0;
        const double k = m_k(p, e), kv = k * vol, hrcp = p.mat.hr_over_cp;
        double gkv = 0;
        const double grh = -((gtd[0] + gtd[1]) + (gtd[2] + gtd[3]));
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double G = sh[c][1] * Td[1] + sh[c][2] * Td[2] + sh[c][3] * Td[3];
            const double U = sh[c][0] * gtd[0] + sh[c][1] * gtd[1] + sh[c][2] * gtd[2] + sh[c][3] * gtd[3];
            gkv += U * G;
            const double kG = kv * G, kU = kv * U;
            gsh[c][0] += gtd[0] * kG;
#pragma unroll
            for (int m = 1; m < 4; ++m) gsh[c][m] += gtd[m] * kG + Td[m] * kU;
#pragma unroll
            for (int m = 0; m < 4; ++m) gTn[m] += sh[c][m] * kU;
        }
        a.g[(size_t)DES_EF_THERM_COND * ne + e] += gkv * vol;
        gvol += gkv * k + grh * hrcp;
    }
    // strain rate
    const double h3 = 0.5 * g[3], h4 = 0.5 * g[4], h5 = 0.5 * g[5];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double sx = sh[0][i], sy = sh[1][i], sz = sh[2][i];
        const double gv0 = g[0] * sx + h3 * sy + h4 * sz;
        const double gv1 = g[1] * sy + h3 * sx + h5 * sz;
        const double gv2 = g[2] * sz + h4 * sx + h5 * sy;
        gsh[0][i] += g[0] * v[i][0] + h3 * v[i][1] + h4 * v[i][2];
        gsh[1][i] += g[1] * v[i][1] + h3 * v[i][0] + h5 * v[i][2];
        gsh[2][i] += g[2] * v[i][2] + h4 * v[i][0] + h5 * v[i][1];
        a.slot3[((size_t)0 * 4 + i) * ne + e] = gv0;
        a.slot3[((size_t)1 * 4 + i) * ne + e] = gv1;
        a.slot3[((size_t)2 * 4 + i) * ne + e] = gv2;
        a.slot1[(size_t)i * ne + e] = gTn[i];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) a.ashp[((size_t)k * 4 + i) * ne + e] = gsh[k][i];
    a.avol[e] = gvol;
}

// a vector slot array and slot1 summed onto out [3][nn] and aT
template <bool STAGED>
__device__ __forceinline__ void gather_slots(const KP &p, const AdjBufs &a, const double *slot, double *out)
{
    const size_t ne = p.ne, nn = p.nn;
    double sum[4];
    const int n = node_sums<SumF64, 4, 3, STAGED>(
        p.sup_off, 0, p.nn, 4,
        [&](int q, double *s) {
            const int ent = p.sup_ent[q];
            const int e = ent >> 2, k = ent & 3;
#pragma unroll
            for (int d = 0; d < 3; ++d) s[d] = slot[((size_t)d * 4 + k) * ne + e];
            s[3] = a.slot1[(size_t)k * ne + e];
        },
        FromZero<SumF64>(), sum);
    if (n < 0) return;
#pragma unroll
    for (int d = 0; d < 3; ++d) out[d * nn + n] += sum[d];
    a.aT[n] += sum[3];
}

// nodes: add the element contributions to the velocity and temperature adjoints
template <bool STAGED>
__global__ void __launch_bounds__(192) k_adj_gather_vT(KP p, AdjBufs a)
{
    gather_slots<STAGED>(p, a, a.slot3, a.av);
}

// window start: adjoints of the derived fields (volume, shape functions,
// mass, tmass, volume_n) -> coordinates and temperature (tmass through
// rho(T) of the start temperature)
__global__ void __launch_bounds__(TPB_A) k_adj_start_geometry(KP p, AdjBufs a, TapeStep t)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= p.ne) return;
    const size_t ne = p.ne;
    int nodes[4];
    double sh[3][4], Tsum = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        nodes[i] = conn_at(p, i, e);
        Tsum += t.T[nodes[i]];
    }
    const double rho_e = m_rho_T(p, e, Tsum / 4);
    double gvol = a.avol[e];
    double gm[4], gtm[4], gvn[4], gs[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        gm[i] = a.am[nodes[i]];
        gtm[i] = a.atm[nodes[i]];
        gvn[i] = a.avn[nodes[i]];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            sh[k][i] = tshp(t, ne, k, i, e);
            gs[k][i] = a.ashp[((size_t)k * 4 + i) * ne + e];
        }
    }
    const double grho = mass_reverse(p, e, gm, gtm, gvn, t.vol[e], rho_e, gvol);
    const double gT = grho * (-p.mat.rho0[0] * p.mat.alpha[0]);
    double gc[4][3];
    geom_reverse(sh, t.vol[e], gs, gvol, gc);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int d = 0; d < 3; ++d) a.slotx[((size_t)d * 4 + i) * ne + e] = gc[i][d];
        a.slot1[(size_t)i * ne + e] = gT / 4;
    }
}

template <bool STAGED>
__global__ void __launch_bounds__(192) k_adj_gather_xT(KP p, AdjBufs a)
{
    gather_slots<STAGED>(p, a, a.slotx, a.ax);
}

// several arrays in one launch, each by its share of the blocks
__global__ void __launch_bounds__(256) k_copy_arrays(const __grid_constant__ CopyTable t)
{
    int k = 0;
    while (k + 1 < t.count && blockIdx.x >= t.first[k + 1]) ++k;
    const size_t stride = (size_t)(t.first[k + 1] - t.first[k]) * blockDim.x, n = t.n[k];
    const double *__restrict__ src = t.src[k];
    double *__restrict__ dst = t.dst[k];
    for (size_t i = (size_t)(blockIdx.x - t.first[k]) * blockDim.x + threadIdx.x; i < n; i += stride) dst[i] = src[i];
}

int launch_copy_arrays(CopyTable &t, cudaStream_t s)
{
    if (t.count == 0) return 0;
    // four values a thread, at most about eight blocks per SM in all
    size_t total = 0;
    for (int k = 0; k < t.count; ++k) total += t.n[k];
    const size_t per_block = std::max<size_t>(1024, (total + 152 * 8 - 1) / (152 * 8));
    unsigned b = 0;
    for (int k = 0; k < t.count; ++k) {
        t.first[k] = b;
        b += (unsigned)std::max<size_t>(1, (t.n[k] + per_block - 1) / per_block);
    }
    t.first[t.count] = b;
    k_copy_arrays<<<b, 256, 0, s>>>(t);
    return 1;
}

int launch_adj_stress(const KP &p, const AdjBufs &a, const TapeStep &t, const TapeStep &t1, double dt,
                      cudaStream_t s)
{
    DES_LAUNCH_W(k_adj_stress, p.ne, s, p, a, t, t1, dt);
    return 1;
}

int launch_adj_nodes_heat(const KP &p, const AdjBufs &a, const TapeStep &t, const TapeStep &t1, double dt,
                          cudaStream_t s)
{
    DES_NODES(k_adj_nodes_heat<STAGED>, p.nn, s, p, a, t, t1, dt);
    return 1;
}

int launch_adj_kinematics(const KP &p, const AdjBufs &a, const TapeStep &t, cudaStream_t s)
{
    DES_LAUNCH_W(k_adj_kinematics, p.ne, s, p, a, t);
    return 1;
}

int launch_adj_gather_vT(const KP &p, const AdjBufs &a, cudaStream_t s)
{
    DES_NODES(k_adj_gather_vT<STAGED>, p.nn, s, p, a);
    return 1;
}

int launch_adj_start_geometry(const KP &p, const AdjBufs &a, const TapeStep &t, cudaStream_t s)
{
    DES_LAUNCH(k_adj_start_geometry, p.ne, s, p, a, t);
    return 1;
}

int launch_adj_gather_xT(const KP &p, const AdjBufs &a, cudaStream_t s)
{
    DES_NODES(k_adj_gather_xT<STAGED>, p.nn, s, p, a);
    return 1;
}

}  // namespace des
