// assembly.cu -- element-per-thread global assembly and Gauss-point flux.
//
// One thread per element.  The element loop of CRFProcess::GlobalAssembly
// (FEM/rf_pcs.cpp:5738-5757) with CFiniteElementStd::Assembly
// (FEM/fem_ele_std.cpp:9367) becomes one launch: each thread gathers its
// node coordinates and primary variable, forms the local matrices in
// registers, combines them into the LHS and RHS exactly as
// AssembleParabolicEquation (fem_ele_std.cpp:7702-8126) or
// AssembleMixedHyperbolicParabolicEquation (:8504-8735) does, and scatters
// with FP64 atomics through the precomputed CSR slot map (no colouring).
//
// Two element paths:
//  * general -- per Gauss point Jacobian, inverse and global gradients,
//    CElement::computeJacobian / ComputeGradShapefct (FEM/fem_ele.cpp:585,
//    1128), then CalcMass / CalcLaplace / CalcAdvection / CalcStorage in
//    the reference's summation order;
//  * affine  -- elements with a constant Jacobian (every tet, parallelogram
//    quads, parallelepiped hexes): Laplace_ij = |J| sum_ab C_ab Q_abij and
//    Mass_ij = c |J| M0_ij with reference tensors Q, M0 summed once over
//    the Gauss points.  Mathematically identical, ~25x fewer FP64 FMAs on
//    hexes, which matters on a part with 1.2 TFLOP/s of FP64.
// Tables (N, dN/dxi, weights; Q, M0) are staged in shared memory per block.
#include <cfloat>
#include <cstdio>

#include "common.cuh"

namespace ogs {

template <int ET> struct ElemTraits;
template <> struct ElemTraits<OGS_ELEM_QUAD4> { static constexpr int NN = 4, DIM = 2; };
template <> struct ElemTraits<OGS_ELEM_HEX8> { static constexpr int NN = 8, DIM = 3; };
template <> struct ElemTraits<OGS_ELEM_TET4> { static constexpr int NN = 4, DIM = 3; };

// Jacobian (row = local direction), |det| and the inverse, as
// CElement::computeJacobian.  Returns false on |det| < DBL_EPSILON.
template <int NN, int DIM>
__device__ __forceinline__ bool jacobian(const double* X, const double* Y,
                                         const double* Z, const double* dN,
                                         double* iJ, double& det)
{
    double J[DIM * DIM];
#pragma unroll
    for (int k = 0; k < DIM * DIM; k++) J[k] = 0.0;
    if (DIM == 2)
    {
#pragma unroll
        for (int i = 0; i < NN; i++)
        {
            J[0] += X[i] * dN[i];
            J[1] += Y[i] * dN[i];
            J[2] += X[i] * dN[NN + i];
            J[3] += Y[i] * dN[NN + i];
        }
        det = J[0] * J[3] - J[1] * J[2];
        if (fabs(det) < DBL_EPSILON) return false;
        // one FP64 division (the cofactors times 1/det; the reference divides
        // each, the results differ by rounding only)
        const double id = 1.0 / det;
        iJ[0] = J[3] * id;
        iJ[1] = -J[1] * id;
        iJ[2] = -J[2] * id;
        iJ[3] = J[0] * id;
    }
    else
    {
#pragma unroll
        for (int i = 0; i < NN; i++)
        {
            J[0] += X[i] * dN[i];
            J[1] += Y[i] * dN[i];
            J[2] += Z[i] * dN[i];
            J[3] += X[i] * dN[NN + i];
            J[4] += Y[i] * dN[NN + i];
            J[5] += Z[i] * dN[NN + i];
            J[6] += X[i] * dN[2 * NN + i];
            J[7] += Y[i] * dN[2 * NN + i];
            J[8] += Z[i] * dN[2 * NN + i];
        }
        det = J[0] * (J[4] * J[8] - J[7] * J[5]) + J[6] * (J[1] * J[5] - J[4] * J[2]) +
              J[3] * (J[2] * J[7] - J[8] * J[1]);
        if (fabs(det) < DBL_EPSILON) return false;
        const double id = 1.0 / det;
        iJ[0] = (J[4] * J[8] - J[7] * J[5]) * id;
        iJ[1] = (J[2] * J[7] - J[1] * J[8]) * id;
        iJ[2] = (J[1] * J[5] - J[2] * J[4]) * id;
        iJ[3] = (J[5] * J[6] - J[8] * J[3]) * id;
        iJ[4] = (J[0] * J[8] - J[6] * J[2]) * id;
        iJ[5] = (J[2] * J[3] - J[5] * J[0]) * id;
        iJ[6] = (J[3] * J[7] - J[6] * J[4]) * id;
        iJ[7] = (J[1] * J[6] - J[7] * J[0]) * id;
        iJ[8] = (J[0] * J[4] - J[3] * J[1]) * id;
    }
    det = fabs(det);
    return true;
}

// global gradients dNg[j*NN+i] = sum_k iJ[j*DIM+k] dN[k*NN+i]
template <int NN, int DIM>
__device__ __forceinline__ void grad_global(const double* iJ, const double* dN, double* dNg)
{
#pragma unroll
    for (int i = 0; i < NN; i++)
#pragma unroll
        for (int j = 0; j < DIM; j++)
        {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < DIM; k++) s += iJ[j * DIM + k] * dN[k * NN + i];
            dNg[j * NN + i] = s;
        }
}

// MassDispersionTensorNew (FEM/rf_mmp_new.cpp:3090-3328), isotropic
// tortuosity: D = n S Daq tau I + alpha_T |q| I + (alpha_L - alpha_T) q q^T / |q|
template <int DIM>
__device__ __forceinline__ void dispersion_raw(const ogs_assembly_params& p, const double* v,
                                               double* D)
{
    const double dm = p.diffusion * p.porosity * p.saturation;
    const double vg = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
#pragma unroll
    for (int i = 0; i < DIM * DIM; i++) D[i] = 0.0;
    if (fabs(vg) > DBL_EPSILON)
    {
        // one division per point: (alpha_L - alpha_T) / |q| times q_i q_j
        // (the reference divides each entry; the results differ by rounding
        // only), the symmetric entries formed once
        const double al = p.alpha_l, at = p.alpha_t;
        const double c = (al - at) / vg;
#pragma unroll
        for (int i = 0; i < DIM; i++)
#pragma unroll
            for (int j = 0; j < i; j++) D[i * DIM + j] = D[j * DIM + i] = c * (v[i] * v[j]);
#pragma unroll
        for (int i = 0; i < DIM; i++) D[i * DIM + i] = (at * vg) + c * (v[i] * v[i]) + dm;
    }
    else
    {
#pragma unroll
        for (int i = 0; i < DIM; i++) D[i * DIM + i] = dm;
    }
}

template <int DIM>
__device__ __forceinline__ void dispersion(const ogs_assembly_params& p, const double* v, double* D)
{
    dispersion_raw<DIM>(p, v, D);
#pragma unroll
    for (int i = 0; i < DIM * DIM; i++) D[i] = D[i] * 1.0 * p.time_unit_factor;
}

// MLangevin (FEM/mathlib.cpp:3009-3021): coth(v) - 1/v, its series below 0.01
__device__ __forceinline__ double langevin(double v)
{
    double s = 0.0;
    if (v < 0.01)
        s = v * (1.0 / 3.0 + v * v * (-1.0 / 45.0 + 18.0 / 8505.0 * v * v));
    else if (0.01 <= v && v < 20)
        s = (exp(v) + exp(-v)) / (exp(v) - exp(-v)) - 1 / v;
    else if (20 <= v)
        s = 1.0;
    return s;
}

// CalcSUPGEffectiveElemenetLength (fem_ele_std.cpp:4034-4095) over the edges
// of CElem::GetLocalIndicesOfEdgeNodes (MSH/msh_elem.cpp:984-1052)
template <int ET>
__device__ __forceinline__ double supg_length(const double* X, const double* Y, const double* Z, int method)
{
    constexpr int NE = ET == OGS_ELEM_HEX8 ? 12 : ET == OGS_ELEM_QUAD4 ? 4 : 6;
    double len[NE];
#pragma unroll
    for (int e = 0; e < NE; e++)
    {
        int a, b;
        if (ET == OGS_ELEM_QUAD4) { a = e; b = (e + 1) % 4; }
        else if (ET == OGS_ELEM_HEX8)
        {
            if (e < 8) { a = e; b = (e + 1) % 4 + 4 * (e / 4); }
            else { a = e % 4; b = e % 4 + 4; }
        }
        else if (e < 3) { a = e; b = (e + 1) % 3; }
        else { a = 3; b = (e + 1) % 3; }
        const double dx = X[b] - X[a], dy = Y[b] - Y[a], dz = Z[b] - Z[a];
        len[e] = sqrt(dx * dx + dy * dy + dz * dz);
    }
    double L = 0.0;
    if (method == 1)
    {
        double mn = len[0];
#pragma unroll
        for (int e = 1; e < NE; e++) { L = len[e]; if (L < mn) mn = L; }
        L = mn;
    }
    else if (method == 2)
    {
        double t = 0.0;
#pragma unroll
        for (int e = 1; e < NE; e++) t += len[e];  // the reference starts at edge 1
        L = t / NE;
    }
    else
    {
        double mx = len[0];
#pragma unroll
        for (int e = 1; e < NE; e++) { L = len[e]; if (L > mx) mx = L; }
        L = mx;
    }
    return L;
}

// CalcSUPGCoefficient (fem_ele_std.cpp:3908-3995), MASS_TRANSPORT; D is the
// raw MassDispersionTensorNew of the Gauss point
template <int DIM>
__device__ __forceinline__ double supg_tau(const ogs_assembly_params& p, const double* vel, const double* D, double L)
{
    const double v_mag = sqrt(vel[0] * vel[0] + vel[1] * vel[1] + vel[2] * vel[2]);
    if (v_mag == 0.0) return 0.0;
    double diff;
    if (p.supg_diffusivity == 1)
    {
        diff = D[0];
#pragma unroll
        for (int i = 1; i < DIM * DIM; i++)
            if (D[i] < diff) diff = D[i];
    }
    else if (p.supg_diffusivity == 2)
    {
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < DIM; i++) t = D[i + i * DIM] * D[i + i * DIM];  // the reference assigns
        diff = sqrt(t);
    }
    else
    {
        diff = D[0];
#pragma unroll
        for (int i = 1; i < DIM * DIM; i++)
            if (D[i] > diff) diff = D[i];
    }
    double tau = 0.0;
    if (p.supg_method == 1)
    {
        const double alpha = 0.5 * v_mag * L / diff;
        tau = 0.5 * L / v_mag * langevin(alpha);
    }
    else if (p.supg_method == 2)
        tau = 1.0 / sqrt((2.0 / p.dt) * (2.0 / p.dt) + (2.0 * v_mag / L) * (2.0 * v_mag / L) +
                         (4.0 * diff / (L * L)) * (4.0 * diff / (L * L)));
    return tau;
}

// flow coefficient of the Laplace term: CalCoefLaplace GWF (:2308-2384,
// mat = K * time_unit_factor * k_rel) or LIQUID_FLOW (:2232-2306,
// mat = time_unit_factor * k / mu, mu -> 1 in the HEAD form)
__device__ __forceinline__ double flow_mat(const ogs_assembly_params& p, double k)
{
    if (p.pcs_type == OGS_PCS_LIQUID_FLOW)
    {
        double mat_fac = p.viscosity;
        if (p.gravity < DBL_EPSILON) mat_fac = 1.0;
        return p.time_unit_factor * k / mat_fac * 1.0 * 1.0;
    }
    return k * p.time_unit_factor * 1.0;
}

// CElem::calcVolume (MSH/msh_elem.cpp:1511-1576) with ComputeDetTri /
// ComputeDetTex (FEM/mathlib.cpp:2911-2955): quads as two triangles,
// hexahedra as six tetrahedra in the mesh's node order
__device__ __forceinline__ double vol_tri(const double* X, const double* Y, const double* Z, int a, int b, int c)
{
    const double u0 = X[c] - X[a], u1 = Y[c] - Y[a], u2 = Z[c] - Z[a];
    const double v0 = X[b] - X[a], v1 = Y[b] - Y[a], v2 = Z[b] - Z[a];
    const double z0 = u1 * v2 - u2 * v1, z1 = u2 * v0 - u0 * v2, z2 = u0 * v1 - u1 * v0;
    return 0.5 * sqrt(z0 * z0 + z1 * z1 + z2 * z2);
}

__device__ __forceinline__ double vol_tet(const double* X, const double* Y, const double* Z, int a, int b, int c,
                                          int d)
{
    const double ax = X[a] - X[d], ay = Y[a] - Y[d], az = Z[a] - Z[d];
    const double bx = X[b] - X[d], by = Y[b] - Y[d], bz = Z[b] - Z[d];
    const double cx = X[c] - X[d], cy = Y[c] - Y[d], cz = Z[c] - Z[d];
    return fabs(ax * (by * cz - bz * cy) - ay * (bx * cz - bz * cx) + az * (bx * cy - by * cx)) / 6.0;
}

template <int ET>
__device__ __forceinline__ double element_volume(const double* X, const double* Y, const double* Z)
{
    if (ET == OGS_ELEM_QUAD4) return vol_tri(X, Y, Z, 0, 1, 2) + vol_tri(X, Y, Z, 2, 3, 0);
    if (ET == OGS_ELEM_TET4) return vol_tet(X, Y, Z, 0, 1, 2, 3);
    double v = vol_tet(X, Y, Z, 4, 7, 5, 0);
    v += vol_tet(X, Y, Z, 5, 3, 1, 0);
    v += vol_tet(X, Y, Z, 5, 7, 3, 0);
    v += vol_tet(X, Y, Z, 5, 7, 6, 2);
    v += vol_tet(X, Y, Z, 1, 3, 5, 2);
    v += vol_tet(X, Y, Z, 3, 7, 5, 2);
    return v;
}

// CalcLumpedMass (fem_ele_std.cpp:4598-4660), selected by
// m_num->ele_mass_lumping: the packed lower-triangle mass becomes
// diag(CalCoefMass * ElementVolumeMultiplyer (1) * volume / nnodes)
template <int ET, int NN>
__device__ __forceinline__ void lump_mass(const double* X, const double* Y, const double* Z, double cm, double* Ml)
{
    double f = cm;
    f *= 1.0;
    f *= element_volume<ET>(X, Y, Z) / (double)NN;
#pragma unroll
    for (int i = 0; i < NN; i++)
#pragma unroll
        for (int j = 0; j <= i; j++) Ml[i * (i + 1) / 2 + j] = i == j ? f : 0.0;
}

// CalCoefMass for GWF (StorageFunction) and LIQUID_FLOW (Ss + n drho/dp).
// AssembleParabolicEquation (fem_ele_std.cpp:7702-8126) has no steady branch:
// a STEADY flow process keeps M/dt, so p.steady is not read here.
__device__ __forceinline__ double flow_mass_coef(const ogs_assembly_params& p)
{
    if (p.pcs_type == OGS_PCS_LIQUID_FLOW) return p.storage + p.porosity * p.drho_dp;
    return p.storage;
}

__device__ __forceinline__ void flag_bad(int* bad, int64_t e)
{
    atomicMin(bad, (int)(e + 1));
}

// stage a table block into shared memory
__device__ __forceinline__ void stage(double* dst, const double* src, int n)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}

template <int NN>
__device__ __forceinline__ void gather(const AsmArgs& a, int64_t e, int* nd, double* X,
                                       double* Y, double* Z, double* U)
{
    const int64_t E = a.E;
#pragma unroll
    for (int i = 0; i < NN; i++)
    {
        nd[i] = __ldg(a.conn_t + (int64_t)i * E + e);
        if (!OGS_IN(nd[i], a.nrows, kOobAsmNode)) nd[i] = 0;
    }
#pragma unroll
    for (int i = 0; i < NN; i++)
    {
        X[i] = __ldg(a.x + nd[i]);
        Y[i] = __ldg(a.y + nd[i]);
        Z[i] = __ldg(a.z + nd[i]);
        U[i] = a.u0 ? __ldg(a.u0 + nd[i]) : 0.0;
    }
}

template <int NN>
__device__ __forceinline__ void scatter(const AsmArgs& a, int64_t e, const int* nd,
                                        const double* S, const double* r)
{
    const int64_t E = a.E;
#pragma unroll
    for (int i = 0; i < NN; i++)
    {
#pragma unroll
        for (int j = 0; j < NN; j++)
        {
            const int32_t k = __ldg(a.slot_t + (int64_t)(i * NN + j) * E + e);
            if (OGS_IN(k, a.nslots, kOobAsmSlot)) atomicAdd(a.val + k, S[i * NN + j]);
        }
        atomicAdd(a.b + nd[i], r[i]);
    }
}

__device__ __forceinline__ void scatter_entry(const AsmArgs& a, int64_t e, int k, double* val, double v)
{
    const int32_t slot = __ldg(a.slot_t + (int64_t)k * a.E + e);
    if (OGS_IN(slot, a.nslots, kOobAsmSlot)) atomicAdd(val + slot, v);
}

// The gradient of a linear or trilinear field through the cofactors of the
// Jacobian: grad_i = (1 / det) sum_k cof[3 i + k] d_k, d the derivatives in
// local coordinates.  Cofactors and det as jacobian<>; false when singular.
__device__ __forceinline__ bool cofactors(const double (&J)[9], double (&C)[9], double& det)
{
    C[0] = J[4] * J[8] - J[7] * J[5];
    C[1] = J[2] * J[7] - J[1] * J[8];
    C[2] = J[1] * J[5] - J[2] * J[4];
    C[3] = J[5] * J[6] - J[8] * J[3];
    C[4] = J[0] * J[8] - J[6] * J[2];
    C[5] = J[2] * J[3] - J[5] * J[0];
    C[6] = J[3] * J[7] - J[6] * J[4];
    C[7] = J[1] * J[6] - J[7] * J[0];
    C[8] = J[0] * J[4] - J[3] * J[1];
    det = J[0] * C[0] + J[6] * C[2] + J[3] * C[1];
    return !(fabs(det) < DBL_EPSILON);
}

// ------------------------------------------------------------------
// Tensor-product forms on hexahedra
// ------------------------------------------------------------------
// Node of the local corner with signs (x, y, z), bit set: -1
__host__ __device__ constexpr int hex_node(int px, int py, int pz)
{
    return pz * 4 + (py ? (px ? 2 : 3) : (px ? 1 : 0));
}
// 1-D Gauss points and weights (MXPGaussPkt / MXPGaussFkt, FEM/mathlib.cpp:1112,1174)
__host__ __device__ constexpr double gauss_x(int ng, int g)
{
    return ng == 1 ? 0.0 : ng == 2 ? (g ? -0.577350269189626 : 0.577350269189626)
                                   : g == 0 ? 0.774596669241483 : g == 1 ? 0.0 : -0.774596669241483;
}
__host__ __device__ constexpr double gauss_w(int ng, int g)
{
    return ng == 1 ? 2.0 : ng == 2 ? 1.0 : g == 1 ? 0.888888888888889 : 0.555555555555556;
}
// 1-D shape function of the node with sign + (p 0) or - (p 1)
__host__ __device__ constexpr double shape1(int ng, int g, int p)
{
    return 0.5 * (p ? 1.0 - gauss_x(ng, g) : 1.0 + gauss_x(ng, g));
}

// Half differences of a field along axis AX of the hex's four edges in that
// direction, e[p + 2 q] with p, q the signs on the other two axes in
// ascending order
template <int AX>
__device__ __forceinline__ void edge_diff(const double* F, double (&e)[4])
{
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
        for (int p = 0; p < 2; p++)
        {
            const int a = AX == 0 ? hex_node(0, p, q) : AX == 1 ? hex_node(p, 0, q) : hex_node(p, q, 0);
            const int b = AX == 0 ? hex_node(1, p, q) : AX == 1 ? hex_node(p, 1, q) : hex_node(p, q, 1);
            e[p + 2 * q] = 0.5 * (F[a] - F[b]);
        }
}

// Local derivatives (r, s, t) of a trilinear field at the Gauss points of
// the slice r = point gr: a derivative along an axis does not depend on the
// coordinate along it, so d/dr is one bilinear form of (s, t) and d/ds,
// d/dt are linear in t and s.  h: the 1-D shape value N_+ at gr.
template <int NG>
struct HexSlice
{
    double dr[NG][NG], ds[NG], dt[NG];  // [s][t], [t], [s]
    __device__ __forceinline__ void set(const double* F, double h)
    {
        double e[4];
        edge_diff<0>(F, e);  // (s, t)
#pragma unroll
        for (int g = 0; g < NG; g++)
        {
            const double u0 = shape1(NG, g, 0) * e[0] + shape1(NG, g, 1) * e[1];  // at s, t = +
            const double u1 = shape1(NG, g, 0) * e[2] + shape1(NG, g, 1) * e[3];
#pragma unroll
            for (int t = 0; t < NG; t++) dr[g][t] = shape1(NG, t, 0) * u0 + shape1(NG, t, 1) * u1;
        }
        edge_diff<1>(F, e);  // (r, t)
        double v0 = h * e[0] + (1.0 - h) * e[1], v1 = h * e[2] + (1.0 - h) * e[3];
#pragma unroll
        for (int t = 0; t < NG; t++) ds[t] = shape1(NG, t, 0) * v0 + shape1(NG, t, 1) * v1;
        edge_diff<2>(F, e);  // (r, s)
        v0 = h * e[0] + (1.0 - h) * e[1];
        v1 = h * e[2] + (1.0 - h) * e[3];
#pragma unroll
        for (int g = 0; g < NG; g++) dt[g] = shape1(NG, g, 0) * v0 + shape1(NG, g, 1) * v1;
    }
};

// Element matrices of a hex by sum factorisation.  A trilinear shape
// function is a product of 1-D ones, and its derivative along an axis is
// +-1/2 times the other two factors.  An integral over the Gauss points of
// coefficient x (shape or derivative of i) x (the same of j) therefore only
// depends on the signs of the two corners, and is contracted an axis at a
// time: along t for the points of a row (r, s), along s for the rows of a
// slice, along r for the slices.  The pair N_p N_q of an axis has three
// forms, k = p + q.  For 27 points this is about 1,000 FP64 operations for
// the full-tensor Laplace form, 600 for the advection and 240 for the mass,
// where the direct sums over points and entry pairs take 4,000, 2,400 and
// 1,900: the element kernels are bound by GB300's FP64 pipe (a warp's FP64
// instruction occupies it for 16 cycles or more), so shared memory traffic,
// low occupancy and integer work are hidden behind it.
//
// The sums over slices are kept in shared memory, one column of kHexThreads
// doubles per sum; those of the current slice in registers.
constexpr int kHexThreads = 128;

__host__ __device__ constexpr double pair1(int ng, int g, int k)
{
    return shape1(ng, g, k == 2 ? 1 : 0) * shape1(ng, g, k == 0 ? 0 : 1);
}
__host__ __device__ constexpr int hex_px(int i) { return (i & 3) == 1 || (i & 3) == 2 ? 1 : 0; }
__host__ __device__ constexpr int hex_py(int i) { return (i & 3) >= 2 ? 1 : 0; }
__host__ __device__ constexpr int hex_pz(int i) { return i >= 4 ? 1 : 0; }
__device__ __forceinline__ double signed_sum(double v, int p) { return p ? -v : v; }

template <int NG, bool LAP, bool ADV, bool MASS>
struct HexSums
{
    // columns of the shared sums
    static constexpr int kRR = 0, kSS = kRR + 3 * NG, kTT = kSS + 9, kRS = kTT + 9, kRT = kRS + 12, kST = kRT + 12;
    static constexpr int kAR = LAP ? kST + 12 : 0, kAS = kAR + 18, kAT = kAS + 18;
    static constexpr int kMM = ADV ? kAT + 18 : kAR, kCols = kMM + (MASS ? 27 : 0);

    double* col;  // this thread's first column
    // the current slice
    double ss[3], tt[3], rs[2][3], rt[3][2], st[2][2], ar[3][3], as_[2][3], at[3][2], mm[3][3];

    __device__ __forceinline__ double& at_col(int k) { return col[k * kHexThreads]; }

    __device__ __forceinline__ void start(double* sm)
    {
        col = sm + threadIdx.x;
#pragma unroll 1
        for (int k = 0; k < kCols; k++) at_col(k) = 0.0;
    }
    __device__ __forceinline__ void start_slice()
    {
#pragma unroll
        for (int k = 0; k < 3; k++)
        {
            ss[k] = tt[k] = 0.0;
            rs[0][k] = rs[1][k] = rt[k][0] = rt[k][1] = as_[0][k] = as_[1][k] = at[k][0] = at[k][1] = 0.0;
#pragma unroll
            for (int q = 0; q < 3; q++) ar[k][q] = mm[k][q] = 0.0;
        }
        st[0][0] = st[0][1] = st[1][0] = st[1][1] = 0.0;
    }
    // sums over t of a row's values: the three pairs, or the two shapes
    static __device__ __forceinline__ void pairs_t(const double (&c)[NG], double (&o)[3])
    {
#pragma unroll
        for (int k = 0; k < 3; k++)
        {
            o[k] = pair1(NG, 0, k) * c[0];
#pragma unroll
            for (int t = 1; t < NG; t++) o[k] += pair1(NG, t, k) * c[t];
        }
    }
    static __device__ __forceinline__ void shapes_t(const double (&c)[NG], double (&o)[2])
    {
#pragma unroll
        for (int p = 0; p < 2; p++)
        {
            o[p] = shape1(NG, 0, p) * c[0];
#pragma unroll
            for (int t = 1; t < NG; t++) o[p] += shape1(NG, t, p) * c[t];
        }
    }
    // the row s of the current slice.  L: the six entries rr, ss, tt, rs,
    // rt, st of the Laplace tensor in local coordinates, A: the three of the
    // flux, each [value][t] and times the quadrature weight and |J|.  DIAG:
    // the entries rs, rt, st are zero
    template <bool DIAG>
    __device__ __forceinline__ void add_lap(int s, const double (&L)[6][NG])
    {
        double o[3], q[2];
        pairs_t(L[0], o);
#pragma unroll
        for (int k = 0; k < 3; k++) at_col(kRR + 3 * s + k) += o[k];
        pairs_t(L[1], o);
#pragma unroll
        for (int k = 0; k < 3; k++) ss[k] += o[k];
        double sum = L[2][0];
#pragma unroll
        for (int t = 1; t < NG; t++) sum += L[2][t];
#pragma unroll
        for (int k = 0; k < 3; k++) tt[k] += pair1(NG, s, k) * sum;
        if (DIAG) return;
        pairs_t(L[3], o);
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int k = 0; k < 3; k++) rs[p][k] += shape1(NG, s, p) * o[k];
        shapes_t(L[4], q);
#pragma unroll
        for (int k = 0; k < 3; k++)
#pragma unroll
            for (int p = 0; p < 2; p++) rt[k][p] += pair1(NG, s, k) * q[p];
        shapes_t(L[5], q);
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int y = 0; y < 2; y++) st[p][y] += shape1(NG, s, y) * q[p];
    }
    __device__ __forceinline__ void add_adv(int s, const double (&A)[3][NG])
    {
        double o[3], q[2];
        pairs_t(A[0], o);
#pragma unroll
        for (int y = 0; y < 3; y++)
#pragma unroll
            for (int k = 0; k < 3; k++) ar[y][k] += pair1(NG, s, y) * o[k];
        pairs_t(A[1], o);
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int k = 0; k < 3; k++) as_[p][k] += shape1(NG, s, p) * o[k];
        shapes_t(A[2], q);
#pragma unroll
        for (int y = 0; y < 3; y++)
#pragma unroll
            for (int p = 0; p < 2; p++) at[y][p] += pair1(NG, s, y) * q[p];
    }
    __device__ __forceinline__ void add_mass(int s, const double (&m)[NG])
    {
        double o[3];
        pairs_t(m, o);
#pragma unroll
        for (int y = 0; y < 3; y++)
#pragma unroll
            for (int k = 0; k < 3; k++) mm[y][k] += pair1(NG, s, y) * o[k];
    }
    // the finished slice into the sums; h: N_+ at its point on the r axis
    __device__ __forceinline__ void end_slice(double h)
    {
        const double w1[2] = {h, 1.0 - h}, w2[3] = {h * h, h * (1.0 - h), (1.0 - h) * (1.0 - h)};
        if (LAP)
        {
#pragma unroll
            for (int x = 0; x < 3; x++)
#pragma unroll
                for (int k = 0; k < 3; k++)
                {
                    at_col(kSS + 3 * x + k) += w2[x] * ss[k];
                    at_col(kTT + 3 * x + k) += w2[x] * tt[k];
                }
#pragma unroll
            for (int x = 0; x < 2; x++)
#pragma unroll
                for (int p = 0; p < 2; p++)
#pragma unroll
                    for (int k = 0; k < 3; k++)
                    {
                        at_col(kRS + 6 * x + 3 * p + k) += w1[x] * rs[p][k];
                        at_col(kRT + 6 * x + 2 * k + p) += w1[x] * rt[k][p];
                    }
#pragma unroll
            for (int x = 0; x < 3; x++)
#pragma unroll
                for (int p = 0; p < 2; p++)
#pragma unroll
                    for (int y = 0; y < 2; y++) at_col(kST + 4 * x + 2 * p + y) += w2[x] * st[p][y];
        }
        if (ADV)
#pragma unroll
            for (int x = 0; x < 3; x++)
#pragma unroll
                for (int y = 0; y < 3; y++)
#pragma unroll
                    for (int p = 0; p < 2; p++)
                    {
                        at_col(kAR + 9 * p + 3 * x + y) += w1[p] * ar[x][y];  // [px][ky][kz]
                        at_col(kAS + 6 * x + 3 * p + y) += w2[x] * as_[p][y];
                        at_col(kAT + 6 * x + 2 * y + p) += w2[x] * at[y][p];
                    }
        if (MASS)
#pragma unroll
            for (int x = 0; x < 3; x++)
#pragma unroll
                for (int y = 0; y < 3; y++)
#pragma unroll
                    for (int k = 0; k < 3; k++) at_col(kMM + 9 * x + 3 * y + k) += w2[x] * mm[y][k];
    }
    // after the last slice: the rr sums contracted along s
    __device__ __forceinline__ void finish(double (&rr)[3][3])
    {
#pragma unroll
        for (int y = 0; y < 3; y++)
#pragma unroll
            for (int k = 0; k < 3; k++)
            {
                rr[y][k] = pair1(NG, 0, y) * at_col(kRR + k);
#pragma unroll
                for (int s = 1; s < NG; s++) rr[y][k] += pair1(NG, s, y) * at_col(kRR + 3 * s + k);
            }
    }
    // entries (i, j) of the forms (the factors 1/4 and 1/2 of the
    // derivatives are in the values added)
    __device__ __forceinline__ double lap(const double (&rr)[3][3], int i, int j)
    {
        const int px = hex_px(i), py = hex_py(i), pz = hex_pz(i), qx = hex_px(j), qy = hex_py(j), qz = hex_pz(j);
        const int x = px + qx, y = py + qy, z = pz + qz;
        double v = signed_sum(rr[y][z], px ^ qx);
        v += signed_sum(at_col(kSS + 3 * x + z), py ^ qy);
        v += signed_sum(at_col(kTT + 3 * x + y), pz ^ qz);
        v += signed_sum(at_col(kRS + 6 * qx + 3 * py + z), px ^ qy);
        v += signed_sum(at_col(kRS + 6 * px + 3 * qy + z), qx ^ py);
        v += signed_sum(at_col(kRT + 6 * qx + 2 * y + pz), px ^ qz);
        v += signed_sum(at_col(kRT + 6 * px + 2 * y + qz), qx ^ pz);
        v += signed_sum(at_col(kST + 4 * x + 2 * pz + qy), py ^ qz);
        v += signed_sum(at_col(kST + 4 * x + 2 * qz + py), qy ^ pz);
        return v;
    }
    __device__ __forceinline__ double adv(int i, int j)
    {
        const int px = hex_px(i), py = hex_py(i), pz = hex_pz(i), qx = hex_px(j), qy = hex_py(j), qz = hex_pz(j);
        const int x = px + qx, y = py + qy, z = pz + qz;
        double v = signed_sum(at_col(kAR + 9 * px + 3 * y + z), qx);
        v += signed_sum(at_col(kAS + 6 * x + 3 * py + z), qy);
        v += signed_sum(at_col(kAT + 6 * x + 2 * y + pz), qz);
        return v;
    }
    __device__ __forceinline__ double mass(int i, int j)
    {
        return at_col(kMM + 9 * (hex_px(i) + hex_px(j)) + 3 * (hex_py(i) + hex_py(j)) + hex_pz(i) + hex_pz(j));
    }
};

// ------------------------------------------------------------------
// flow: GROUNDWATER_FLOW / LIQUID_FLOW
// ------------------------------------------------------------------
template <int NN>
__device__ __forceinline__ void flow_combine(const AsmArgs& a, int64_t e, const int* nd,
                                             const double* U, const double* Ml,
                                             const double* Ll, const double* grav)
{
    // AssembleParabolicEquation: fac1 = 1/dt, fac2 = relax0; RHS with relax1
    const double dt_inverse = 1.0 / a.p.dt;
    double relax0 = a.p.nls_relaxation;
    if (relax0 < DBL_MIN) relax0 = 1.0;
    const double relax1 = 1.0 - relax0;
    // the element matrices are symmetric: each distinct entry of the LHS
    // and of the RHS operator is formed once (the same expressions as per
    // (i, j), so the values are the same bit for bit)
    constexpr int NL = NN * (NN + 1) / 2;
    double Sl[NL], Tl[NL];
#pragma unroll
    for (int l = 0; l < NL; l++)
    {
        const double m = Ml[l], lp = Ll[l];
        Sl[l] = m * dt_inverse + lp * relax0;
        Tl[l] = m * dt_inverse - lp * relax1;
    }
    double S[NN * NN], r[NN];
#pragma unroll
    for (int i = 0; i < NN; i++) r[i] = 0.0;
#pragma unroll
    for (int i = 0; i < NN; i++)
#pragma unroll
        for (int j = 0; j < NN; j++)
        {
            const int l = i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
            S[i * NN + j] = Sl[l];
            r[i] += Tl[l] * U[j];
        }
    if ((a.p.pcs_type == OGS_PCS_LIQUID_FLOW || a.p.pcs_type == OGS_PCS_RICHARDS_FLOW) && a.p.gravity_on)
#pragma unroll
        for (int i = 0; i < NN; i++) r[i] += grav[i];
    scatter<NN>(a, e, nd, S, r);
}

// quads and tets (hexes that are not affine: k_flow_hex)
template <int ET, int NGP>
__global__ void __launch_bounds__(128) k_flow_general(AsmArgs a)
{
    constexpr int NN = ElemTraits<ET>::NN, DIM = ElemTraits<ET>::DIM;
    __shared__ double sN[NGP * NN], sdN[NGP * NN * DIM], sw[NGP * 3];
    stage(sN, a.tab, NGP * NN);
    stage(sdN, a.tab + NGP * NN, NGP * NN * DIM);
    stage(sw, a.tab + NGP * NN + NGP * NN * DIM, NGP * 3);
    __syncthreads();
    const double cm = flow_mass_coef(a.p);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < a.E;
         e += (int64_t)gridDim.x * blockDim.x)
    {
        int nd[NN];
        double X[NN], Y[NN], Z[NN], U[NN];
        gather<NN>(a, e, nd, X, Y, Z, U);
        const double mat = flow_mat(a.p, __ldg(a.elem_k + e));
        double Ml[NN * (NN + 1) / 2], Ll[NN * (NN + 1) / 2], grav[NN];
#pragma unroll
        for (int l = 0; l < NN * (NN + 1) / 2; l++) Ml[l] = Ll[l] = 0.0;
#pragma unroll
        for (int i = 0; i < NN; i++) grav[i] = 0.0;
        bool ok = true;
#pragma unroll 1
        for (int gp = 0; gp < NGP; gp++)
        {
            double iJ[DIM * DIM], det, dNg[DIM * NN];
            if (!jacobian<NN, DIM>(X, Y, Z, sdN + gp * NN * DIM, iJ, det)) { ok = false; break; }
            grad_global<NN, DIM>(iJ, sdN + gp * NN * DIM, dNg);
            const double* w = sw + gp * 3;
            const double fkt = ET == OGS_ELEM_QUAD4 ? det * w[0] * w[1] : det * w[0];
            const double* sf = sN + gp * NN;
            const double mf = cm * fkt * 1.0;
            const double cl = fkt * mat;  // the Gauss-point factors hoisted
#pragma unroll
            for (int i = 0; i < NN; i++)
            {
                const double mi = mf * sf[i];
#pragma unroll
                for (int j = 0; j <= i; j++)
                {
                    const int l = i * (i + 1) / 2 + j;
                    Ml[l] += mi * sf[j];
                    double g = 0.0;
#pragma unroll
                    for (int k = 0; k < DIM; k++) g += dNg[k * NN + i] * dNg[k * NN + j];
                    Ll[l] += cl * g;
                }
            }
            if (a.p.pcs_type == OGS_PCS_LIQUID_FLOW && a.p.gravity_on)
            {
                const double rho = a.p.gravity < DBL_EPSILON ? 1.0 : a.p.density * a.p.gravity;
                const double fg = fkt * rho;
#pragma unroll
                for (int i = 0; i < NN; i++) grav[i] -= fg * dNg[(DIM - 1) * NN + i] * mat;
            }
        }
        if (!ok) { flag_bad(a.bad_elem, e); continue; }
        if (a.p.mass_lumping) lump_mass<ET, NN>(X, Y, Z, cm, Ml);
        flow_combine<NN>(a, e, nd, U, Ml, Ll, grav);
    }
}

// affine flow: C = mat * iJ^T iJ (isotropic), Laplace = |J| sum_ab C_ab Q_ab
template <int ET>
__global__ void __launch_bounds__(128) k_flow_affine(AsmArgs a)
{
    constexpr int NN = ElemTraits<ET>::NN, DIM = ElemTraits<ET>::DIM;
    constexpr int NQ = DIM * DIM * NN * NN;
    __shared__ double sQ[NQ], sM0[NN * NN], sdNc[DIM * NN];
    stage(sQ, a.aff, NQ);
    stage(sM0, a.aff + NQ, NN * NN);
    stage(sdNc, a.aff + NQ + NN * NN, DIM * NN);
    __syncthreads();
    const double cm = flow_mass_coef(a.p);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < a.E;
         e += (int64_t)gridDim.x * blockDim.x)
    {
        int nd[NN];
        double X[NN], Y[NN], Z[NN], U[NN];
        gather<NN>(a, e, nd, X, Y, Z, U);
        const double mat = flow_mat(a.p, __ldg(a.elem_k + e));
        double iJ[DIM * DIM], det;
        if (!jacobian<NN, DIM>(X, Y, Z, sdNc, iJ, det)) { flag_bad(a.bad_elem, e); continue; }
        // axis-aligned boxes: the off-diagonal entries of J^-1, hence of C,
        // are exactly 0, and the sums over the DIM diagonal terms equal the
        // full sums bit for bit (the other terms add +-0)
        bool box = true;
#pragma unroll
        for (int p = 0; p < DIM; p++)
#pragma unroll
            for (int q = 0; q < DIM; q++)
                if (p != q && iJ[p * DIM + q] != 0.0) box = false;
        double C[DIM * DIM];
#pragma unroll
        for (int p = 0; p < DIM; p++)
#pragma unroll
            for (int q = 0; q < DIM; q++)
            {
                if (box && p != q)
                {
                    C[p * DIM + q] = 0.0;
                    continue;
                }
                double s = 0.0;
#pragma unroll
                for (int k = 0; k < DIM; k++) s += iJ[k * DIM + p] * iJ[k * DIM + q];
                C[p * DIM + q] = det * mat * s;
            }
        double Ml[NN * (NN + 1) / 2], Ll[NN * (NN + 1) / 2], grav[NN];
        const double md = cm * det;
        if (box)
        {
#pragma unroll
            for (int i = 0; i < NN; i++)
#pragma unroll
                for (int j = 0; j <= i; j++)
                {
                    const int l = i * (i + 1) / 2 + j;
                    double s = 0.0;
#pragma unroll
                    for (int p = 0; p < DIM; p++) s += C[p * DIM + p] * sQ[((p * DIM + p) * NN + i) * NN + j];
                    Ll[l] = s;
                    Ml[l] = md * sM0[i * NN + j];
                }
        }
        else
        {
#pragma unroll
            for (int i = 0; i < NN; i++)
#pragma unroll
                for (int j = 0; j <= i; j++)
                {
                    const int l = i * (i + 1) / 2 + j;
                    double s = 0.0;
#pragma unroll
                    for (int pq = 0; pq < DIM * DIM; pq++) s += C[pq] * sQ[(pq * NN + i) * NN + j];
                    Ll[l] = s;
                    Ml[l] = md * sM0[i * NN + j];
                }
        }
        if (a.p.mass_lumping) lump_mass<ET, NN>(X, Y, Z, cm, Ml);
#pragma unroll
        for (int i = 0; i < NN; i++) grav[i] = 0.0;
        if (a.p.pcs_type == OGS_PCS_LIQUID_FLOW && a.p.gravity_on)
        {
            // -rho g |J| sum_gp w dNg_last,i = -rho g |J| sum_k iJ[last][k] sum_gp w dN_k,i;
            // sum_gp w dN_k,i is Q-independent: recompute from the centre
            // gradient (constant for affine tets) via the weight sum
            const double rho = a.p.gravity < DBL_EPSILON ? 1.0 : a.p.density * a.p.gravity;
            // sum_gp w_gp dN(gp) for affine maps equals vol_ref * dN(centre)
            const double vol_ref = ET == OGS_ELEM_HEX8 ? 8.0 : ET == OGS_ELEM_QUAD4 ? 4.0 : 1.0 / 6.0;
#pragma unroll
            for (int i = 0; i < NN; i++)
            {
                double g = 0.0;
#pragma unroll
                for (int k = 0; k < DIM; k++) g += iJ[(DIM - 1) * DIM + k] * sdNc[k * NN + i];
                grav[i] = -(det * rho * vol_ref) * g * mat;
            }
        }
        flow_combine<NN>(a, e, nd, U, Ml, Ll, grav);
    }
}

// ------------------------------------------------------------------
// flow on a regular lattice of axis-aligned boxes, one thread per row
// ------------------------------------------------------------------
// Every cell of the lattice has the same Jacobian, so its element matrices
// are mat_c L_box + M_box with L_box, M_box common to all cells, and on a
// box an entry L_box[a][b] depends only on which coordinates of corners a
// and b agree (the pattern: bit 0 x, 1 y, 2 z).  Row i of the assembled
// system, at the column j = i + (dx, dy, dz), is therefore
//   A_ij = cnt_ij M_pat / dt + relax0 L_pat S_ij,  S_ij = sum of mat_c
// over the cells holding both nodes, and b_i = sum_j (cnt_ij M_pat / dt -
// relax1 L_pat S_ij) u0_j (+ the gravity term of LIQUID_FLOW): the same
// element matrices as k_flow_affine (whose per-element Gauss sums, FP64
// atomics and scatter this replaces), added in another order.  The tables
// come from element 0 through the element kernel's own formulas.
struct LatticeArgs
{
    const int32_t* slice_ptr;
    int nx, ny, nz;
    int64_t n;
};

__host__ __device__ constexpr int kCornerX(int k) { return (k == 1 || k == 2 || k == 5 || k == 6) ? 1 : 0; }
__host__ __device__ constexpr int kCornerY(int k) { return (k == 2 || k == 3 || k == 6 || k == 7) ? 1 : 0; }
__host__ __device__ constexpr int kCornerZ(int k) { return k >= 4 ? 1 : 0; }

// PLAIN: relax0 = 1 (no NLS relaxation), so b takes the mass term only
template <bool PLAIN>
__global__ void __launch_bounds__(256, 2) k_flow_lattice(AsmArgs a, LatticeArgs g)
{
    // sL: L_pat; sMC[pat][c] = c M_pat / dt for c shared cells (the product
    // formed once here, looked up per entry); sG: gravity per corner
    __shared__ double sL[8], sMC[8][9], sG[8];
    __shared__ double s_geo[8];  // c[3], det, the last row of J^-1, volume / 8
    __shared__ int s_ok;
    const double* Q = a.aff;
    const double* M0 = a.aff + 9 * 64;
    const double* dNc = a.aff + 9 * 64 + 64;
    if (threadIdx.x == 0)
    {
        int nd[8];
        double X[8], Y[8], Z[8], U[8];
        gather<8>(a, 0, nd, X, Y, Z, U);
        double iJ[9], det;
        const bool ok = jacobian<8, 3>(X, Y, Z, dNc, iJ, det);
        s_ok = ok ? 1 : 0;
        if (!ok)
            flag_bad(a.bad_elem, 0);  // every cell has this Jacobian: element 0 is the first singular one
        else
        {
            for (int q = 0; q < 3; q++)
            {
                double t = 0.0;
                for (int k = 0; k < 3; k++) t += iJ[k * 3 + q] * iJ[k * 3 + q];
                s_geo[q] = det * t;
                s_geo[4 + q] = iJ[2 * 3 + q];
            }
            s_geo[3] = det;
            s_geo[7] = a.p.mass_lumping ? element_volume<OGS_ELEM_HEX8>(X, Y, Z) / 8.0 : 0.0;
        }
    }
    __syncthreads();
    // the tables, a thread each: their FP64 chains beside each other
    if (s_ok && threadIdx.x < 16)
    {
        const double det = s_geo[3];
        const int pat = threadIdx.x & 7;
        if (threadIdx.x < 8)
        {
            const double cm = flow_mass_coef(a.p), dt_inverse = 1.0 / a.p.dt;
            // corner b with this pattern against corner 0 = (0, 0, 0)
            int b = 0;
            for (int k = 0; k < 8; k++)
                if ((kCornerX(k) == 0) == ((pat & 1) != 0) && (kCornerY(k) == 0) == ((pat & 2) != 0) &&
                    (kCornerZ(k) == 0) == ((pat & 4) != 0))
                    b = k;
            double l = 0.0;
            for (int q = 0; q < 3; q++) l += s_geo[q] * Q[((q * 3 + q) * 8 + 0) * 8 + b];
            sL[pat] = l;
            const double m = a.p.mass_lumping ? (pat == 7 ? cm * 1.0 * s_geo[7] : 0.0) : cm * det * M0[b];
            const double mdt = m * dt_inverse;
            for (int n = 0; n <= 8; n++) sMC[pat][n] = (double)n * mdt;
        }
        else
        {
            const bool grav = a.p.pcs_type == OGS_PCS_LIQUID_FLOW && a.p.gravity_on;
            const double rho = a.p.gravity < DBL_EPSILON ? 1.0 : a.p.density * a.p.gravity;
            double t = 0.0;
            for (int q = 0; q < 3; q++) t += s_geo[4 + q] * dNc[q * 8 + pat];
            sG[pat] = grav ? -(det * rho * 8.0) * t : 0.0;
        }
    }
    __syncthreads();
    if (!s_ok) return;
    double relax0 = a.p.nls_relaxation;
    if (relax0 < DBL_MIN) relax0 = 1.0;
    const double relax1 = 1.0 - relax0;
    const bool grav = a.p.pcs_type == OGS_PCS_LIQUID_FLOW && a.p.gravity_on;
    // GROUNDWATER_FLOW with time_unit_factor 1: mat = k * 1.0 * 1.0 = k
    const bool unit_mat = a.p.pcs_type == OGS_PCS_GROUNDWATER_FLOW && a.p.time_unit_factor == 1.0;
    const int nx = g.nx, ny = g.ny, nz = g.nz, ncx = nx - 1, ncy = ny - 1, ncz = nz - 1;
    const int64_t nxy = (int64_t)nx * ny;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < g.n; i += (int64_t)gridDim.x * blockDim.x)
    {
        const int iz = (int)(i / nxy), rem = (int)(i - iz * nxy), iy = rem / nx, ix = rem - iy * nx;
        // the eight cells around the node, (ix - 1 + ex, iy - 1 + ey, iz - 1 + ez)
        double mc[2][2][2];
        int pc[2][2][2];
        double gb = 0.0;
#pragma unroll
        for (int ez = 0; ez < 2; ez++)
#pragma unroll
            for (int ey = 0; ey < 2; ey++)
#pragma unroll
                for (int ex = 0; ex < 2; ex++)
                {
                    const int cx = ix - 1 + ex, cy = iy - 1 + ey, cz = iz - 1 + ez;
                    const bool in = cx >= 0 && cx < ncx && cy >= 0 && cy < ncy && cz >= 0 && cz < ncz;
                    const double k = in ? __ldg(a.elem_k + cx + (int64_t)ncx * (cy + (int64_t)ncy * cz)) : 0.0;
                    const double m = unit_mat ? k : flow_mat(a.p, k);
                    mc[ez][ey][ex] = m;
                    pc[ez][ey][ex] = in ? 1 : 0;
                    // the node is the cell's corner (1 - ex, 1 - ey, 1 - ez)
                    if (grav) gb += m * sG[(1 - ez) * 4 + ((1 - ey) ? ((1 - ex) ? 2 : 3) : ((1 - ex) ? 1 : 0))];
                }
        // sums over the cells shared with the neighbour at offset d: per axis
        // index 0 (d = -1: the lower cell), 1 (d = 0: both), 2 (d = +1)
        double sx[2][2][3], sy[2][3][3], S[3][3][3];
        int cx_[2][2][3], cy_[2][3][3], C[3][3][3];
#pragma unroll
        for (int ez = 0; ez < 2; ez++)
#pragma unroll
            for (int ey = 0; ey < 2; ey++)
            {
                sx[ez][ey][0] = mc[ez][ey][0];
                sx[ez][ey][2] = mc[ez][ey][1];
                sx[ez][ey][1] = mc[ez][ey][0] + mc[ez][ey][1];
                cx_[ez][ey][0] = pc[ez][ey][0];
                cx_[ez][ey][2] = pc[ez][ey][1];
                cx_[ez][ey][1] = pc[ez][ey][0] + pc[ez][ey][1];
            }
#pragma unroll
        for (int ez = 0; ez < 2; ez++)
#pragma unroll
            for (int kx = 0; kx < 3; kx++)
            {
                sy[ez][0][kx] = sx[ez][0][kx];
                sy[ez][2][kx] = sx[ez][1][kx];
                sy[ez][1][kx] = sx[ez][0][kx] + sx[ez][1][kx];
                cy_[ez][0][kx] = cx_[ez][0][kx];
                cy_[ez][2][kx] = cx_[ez][1][kx];
                cy_[ez][1][kx] = cx_[ez][0][kx] + cx_[ez][1][kx];
            }
#pragma unroll
        for (int ky = 0; ky < 3; ky++)
#pragma unroll
            for (int kx = 0; kx < 3; kx++)
            {
                S[0][ky][kx] = sy[0][ky][kx];
                S[2][ky][kx] = sy[1][ky][kx];
                S[1][ky][kx] = sy[0][ky][kx] + sy[1][ky][kx];
                C[0][ky][kx] = cy_[0][ky][kx];
                C[2][ky][kx] = cy_[1][ky][kx];
                C[1][ky][kx] = cy_[0][ky][kx] + cy_[1][ky][kx];
            }
        // the row's stored entries in column order: (dz, dy, dx) lexicographic
        const int64_t s0 = __ldg(g.slice_ptr + (i >> 5)) + (i & 31);
        double* __restrict__ v = a.val + s0;
        double bi = gb;
        int rank = 0;
#pragma unroll
        for (int dz = -1; dz <= 1; dz++)
#pragma unroll
            for (int dy = -1; dy <= 1; dy++)
#pragma unroll
                for (int dx = -1; dx <= 1; dx++)
                {
                    const int jx = ix + dx, jy = iy + dy, jz = iz + dz;
                    if (jx < 0 || jx >= nx || jy < 0 || jy >= ny || jz < 0 || jz >= nz) continue;
                    const int pat = (dx == 0 ? 1 : 0) | (dy == 0 ? 2 : 0) | (dz == 0 ? 4 : 0);
                    const double mt = sMC[pat][C[dz + 1][dy + 1][dx + 1]];
                    const double lt = sL[pat] * S[dz + 1][dy + 1][dx + 1];
                    const int64_t j = i + dx + nx * (dy + (int64_t)ny * dz);
                    const double u = a.u0 && OGS_IN(j, g.n, kOobLatNode) ? __ldg(a.u0 + j) : 0.0;
                    const double e = PLAIN ? mt + lt : mt + lt * relax0;
                    if (OGS_IN(s0 + (int64_t)rank * kSlice, a.nslots, kOobLatSlot))
                    {
                        if (a.val_store)
                            v[(int64_t)rank * kSlice] = e;
                        else
                            v[(int64_t)rank * kSlice] += e;
                    }
                    if constexpr (PLAIN)
                        bi += mt * u;
                    else
                        bi += (mt - lt * relax1) * u;
                    rank++;
                }
        a.b[i] += bi;
    }
}

// The same on a plane lattice of equal rectangles (quads): nine entries a
// row from the four cells around the node.  Without atomics the system is
// the same bit for bit in every assembly; the element kernel's sums move in
// the last place with the order in which its atomics land, and an FP32-inner
// solve to 1e-7 then moves by up to 5e-10.
// 702,000 rows: 170 us with the element kernel, 83 to 96 us here.
template <bool PLAIN>
__global__ void __launch_bounds__(256) k_flow_lattice_quad(AsmArgs a, LatticeArgs g)
{
    // bit 0 of a pattern: same x, bit 1: same y
    __shared__ double sL[4], sMC[4][5], sG[4];
    __shared__ double s_geo[8];  // c[2], det, the last row of J^-1, volume / 4; mass coefficient, 1 / dt
    __shared__ int s_ok;
    const double* Q = a.aff;
    const double* M0 = a.aff + 4 * 16;
    const double* dNc = a.aff + 4 * 16 + 16;
    if (threadIdx.x == 0)
    {
        int nd[4];
        double X[4], Y[4], Z[4], U[4];
        gather<4>(a, 0, nd, X, Y, Z, U);
        double iJ[4], det;
        const bool ok = jacobian<4, 2>(X, Y, Z, dNc, iJ, det);
        s_ok = ok ? 1 : 0;
        if (!ok)
            flag_bad(a.bad_elem, 0);
        else
        {
            for (int q = 0; q < 2; q++) s_geo[q] = det * (iJ[q] * iJ[q] + iJ[2 + q] * iJ[2 + q]);
            s_geo[2] = det;
            s_geo[3] = iJ[2];
            s_geo[4] = iJ[3];
            s_geo[5] = a.p.mass_lumping ? element_volume<OGS_ELEM_QUAD4>(X, Y, Z) / 4.0 : 0.0;
        }
    }
    else if (threadIdx.x == 32)
    {
        s_geo[6] = flow_mass_coef(a.p);
        s_geo[7] = 1.0 / a.p.dt;
    }
    __syncthreads();
    if (!s_ok) return;
    // the tables, a thread each (a call with gravity on 702,000 rows 193 us when
    // thread 0 formed them one after the other, 147 so; on 3,000 rows 35.5 and 34.2)
    if (threadIdx.x < 4)
    {
        // corner b with this pattern against corner 0
        const int pat = threadIdx.x, b = pat == 3 ? 0 : pat == 2 ? 1 : pat == 0 ? 2 : 3;
        sL[pat] = s_geo[0] * Q[b] + s_geo[1] * Q[3 * 16 + b];
        const double m = a.p.mass_lumping ? (pat == 3 ? s_geo[6] * 1.0 * s_geo[5] : 0.0) : s_geo[6] * s_geo[2] * M0[b];
        for (int n = 0; n <= 4; n++) sMC[pat][n] = (double)n * (m * s_geo[7]);
    }
    else if (threadIdx.x < 8)
    {
        const int k = threadIdx.x - 4;
        const bool on = a.p.pcs_type == OGS_PCS_LIQUID_FLOW && a.p.gravity_on;
        const double rho = a.p.gravity < DBL_EPSILON ? 1.0 : a.p.density * a.p.gravity;
        sG[k] = on ? -(s_geo[2] * rho * 4.0) * (s_geo[3] * dNc[k] + s_geo[4] * dNc[4 + k]) : 0.0;
    }
    __syncthreads();
    double relax0 = a.p.nls_relaxation;
    if (relax0 < DBL_MIN) relax0 = 1.0;
    const double relax1 = 1.0 - relax0;
    const bool grav = a.p.pcs_type == OGS_PCS_LIQUID_FLOW && a.p.gravity_on;
    const bool unit_mat = a.p.pcs_type == OGS_PCS_GROUNDWATER_FLOW && a.p.time_unit_factor == 1.0;
    const int nx = g.nx, ny = g.ny;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < g.n; i += (int64_t)gridDim.x * blockDim.x)
    {
        const int iy = (int)(i / nx), ix = (int)(i - (int64_t)iy * nx);
        // the cells (ix - 1 + ex, iy - 1 + ey); the node is their corner (1 - ex, 1 - ey)
        double s[2][3], S[3][3], gb = 0.0;
        int n[2][3];
#pragma unroll
        for (int ey = 0; ey < 2; ey++)
        {
            double mc[2];
            int pc[2];
#pragma unroll
            for (int ex = 0; ex < 2; ex++)
            {
                const int cx = ix - 1 + ex, cy = iy - 1 + ey;
                const bool in = cx >= 0 && cx < nx - 1 && cy >= 0 && cy < ny - 1;
                const double k = in ? __ldg(a.elem_k + cx + (int64_t)(nx - 1) * cy) : 0.0;
                mc[ex] = unit_mat ? k : flow_mat(a.p, k);
                pc[ex] = in ? 1 : 0;
                if (grav) gb += mc[ex] * sG[ey ? (ex ? 0 : 1) : (ex ? 3 : 2)];
            }
            s[ey][0] = mc[0];
            s[ey][2] = mc[1];
            s[ey][1] = mc[0] + mc[1];
            n[ey][0] = pc[0];
            n[ey][2] = pc[1];
            n[ey][1] = pc[0] + pc[1];
        }
#pragma unroll
        for (int k = 0; k < 3; k++)
        {
            S[0][k] = s[0][k];
            S[2][k] = s[1][k];
            S[1][k] = s[0][k] + s[1][k];
        }
        const int64_t s0 = __ldg(g.slice_ptr + (i >> 5)) + (i & 31);
        double bi = gb;
        int rank = 0;
#pragma unroll
        for (int dy = -1; dy <= 1; dy++)
#pragma unroll
            for (int dx = -1; dx <= 1; dx++)
            {
                if (ix + dx < 0 || ix + dx >= nx || iy + dy < 0 || iy + dy >= ny) continue;
                const int pat = (dx == 0 ? 1 : 0) | (dy == 0 ? 2 : 0);
                const int cells = dy == 0 ? n[0][dx + 1] + n[1][dx + 1] : n[dy < 0 ? 0 : 1][dx + 1];
                const double mt = sMC[pat][cells], lt = sL[pat] * S[dy + 1][dx + 1];
                const int64_t j = i + dx + (int64_t)nx * dy;
                const double u = a.u0 && OGS_IN(j, g.n, kOobLatNode) ? __ldg(a.u0 + j) : 0.0;
                const double e = PLAIN ? mt + lt : mt + lt * relax0;
                if (OGS_IN(s0 + (int64_t)rank * kSlice, a.nslots, kOobLatSlot))
                {
                    double* v = a.val + s0 + (int64_t)rank * kSlice;
                    *v = a.val_store ? e : *v + e;
                }
                bi += PLAIN ? mt * u : (mt - lt * relax1) * u;
                rank++;
            }
        a.b[i] += bi;
    }
}

// ------------------------------------------------------------------
// MASS_TRANSPORT
// ------------------------------------------------------------------
// STORE: the kernel may be the one that fills the stored operators (the SUPG
// instantiation, whose extra terms vanish with supg_method 0)
template <int NN, bool STORE = false>
__device__ __forceinline__ void mt_combine(const AsmArgs& a, int64_t e, const int* nd,
                                           const double* U, const double* Ml,
                                           const double* L, const double* A,
                                           const double* St, const double* Mx = nullptr)
{
    // Mx: the non-symmetric SUPG mass term (full NN x NN), added to the mass
    // AssembleMixedHyperbolicParabolicEquation (fem_ele_std.cpp:8592-8692)
    if (STORE && a.val2)
    {
        // the operators stored for memory_type > 0 (EleMat->SetMass_notsym,
        // SetLaplace, SetAdvection, SetStorage; fem_ele_std.cpp:8565-8573),
        // scattered: their time weights are applied per assembly
#pragma unroll
        for (int i = 0; i < NN; i++)
#pragma unroll
            for (int j = 0; j < NN; j++)
            {
                const int l = i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
                const int k = i * NN + j;
                const int32_t slot = __ldg(a.slot_t + (int64_t)k * a.E + e);
                atomicAdd(a.val + slot, Mx ? Ml[l] + Mx[k] : Ml[l]);
                atomicAdd(a.val2 + slot, L[k] + A[k] + St[l]);
            }
        return;
    }
    const double dt_inverse = 1.0 / a.p.dt;
    const double th = a.p.theta;
    double S[NN * NN], r[NN];
#pragma unroll
    for (int i = 0; i < NN; i++) r[i] = 0.0;
#pragma unroll
    for (int i = 0; i < NN; i++)
#pragma unroll
        for (int j = 0; j < NN; j++)
        {
            const int l = i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
            const int k = i * NN + j;
            const double mij = Mx ? Ml[l] + Mx[k] : Ml[l];
            double s = mij * dt_inverse;
            s += L[k] * th;
            s += A[k] * th;
            s += St[l] * th;
            S[k] = s;
            double q = mij * dt_inverse;
            q += L[k] * (-(1.0 - th));
            q += A[k] * (-(1.0 - th));
            q += St[l] * (-(1.0 - th));
            r[i] += q * U[j];
        }
    scatter<NN>(a, e, nd, S, r);
}

// SUPG: with the streamline-upwind terms of ele_supg_method > 0
template <int ET, int NGP, bool SUPG>
__global__ void __launch_bounds__(128) k_mt_general(AsmArgs a)
{
    constexpr int NN = ElemTraits<ET>::NN, DIM = ElemTraits<ET>::DIM;
    __shared__ double sN[NGP * NN], sdN[NGP * NN * DIM], sw[NGP * 3];
    stage(sN, a.tab, NGP * NN);
    stage(sdN, a.tab + NGP * NN, NGP * NN * DIM);
    stage(sw, a.tab + NGP * NN + NGP * NN * DIM, NGP * 3);
    __syncthreads();
    const ogs_assembly_params& p = a.p;
    const double cm = p.steady ? 0.0 : p.porosity * p.saturation * p.retardation;
    const double cs = p.porosity * p.saturation * p.decay * p.retardation;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < a.E;
         e += (int64_t)gridDim.x * blockDim.x)
    {
        int nd[NN];
        double X[NN], Y[NN], Z[NN], U[NN];
        gather<NN>(a, e, nd, X, Y, Z, U);
        // Ls: the symmetric dispersion term, lower triangle (expanded for
        // the combine)
        double Ml[NN * (NN + 1) / 2], St[NN * (NN + 1) / 2], Ls[NN * (NN + 1) / 2], A[NN * NN];
        double Mx[SUPG ? NN * NN : 1];
#pragma unroll
        for (int l = 0; l < NN * (NN + 1) / 2; l++) Ml[l] = St[l] = Ls[l] = 0.0;
#pragma unroll
        for (int k = 0; k < NN * NN; k++) A[k] = 0.0;
#pragma unroll
        for (int k = 0; k < (SUPG ? NN * NN : 1); k++) Mx[k] = 0.0;
        const double Lsupg = SUPG ? supg_length<ET>(X, Y, Z, p.supg_length) : 0.0;
        bool ok = true;
        const double* ve = a.gpv + e * NGP * 3;
#pragma unroll 1
        for (int gp = 0; gp < NGP; gp++)
        {
            double iJ[DIM * DIM], det, dNg[DIM * NN];
            if (!jacobian<NN, DIM>(X, Y, Z, sdN + gp * NN * DIM, iJ, det)) { ok = false; break; }
            grad_global<NN, DIM>(iJ, sdN + gp * NN * DIM, dNg);
            const double* w = sw + gp * 3;
            const double fkt = ET == OGS_ELEM_HEX8 ? det * w[0] * w[1] * w[2]
                             : ET == OGS_ELEM_QUAD4 ? det * w[0] * w[1] : det * w[0];
            const double* sf = sN + gp * NN;
            const double v[3] = {__ldg(ve + gp * 3), __ldg(ve + gp * 3 + 1), __ldg(ve + gp * 3 + 2)};
            double D[DIM * DIM];
            dispersion<DIM>(p, v, D);
            const double mf = cm * fkt * 1.0;
            const double fs = fkt * cs;
            const double vt[3] = {1.0 * p.time_unit_factor * v[0], 1.0 * p.time_unit_factor * v[1],
                                  1.0 * p.time_unit_factor * v[2]};
            // the Gauss-point sums with their factors hoisted: T = D grad N
            // once, the symmetric dispersion term over distinct pairs,
            // vd_j = v . grad N_j once (rounding-level differences from the
            // per-entry products)
            double T[DIM * NN], vd[NN];
#pragma unroll
            for (int j = 0; j < NN; j++)
            {
                double q = 0.0;
#pragma unroll
                for (int k = 0; k < DIM; k++)
                {
                    double t = 0.0;
#pragma unroll
                    for (int l2 = 0; l2 < DIM; l2++) t += D[DIM * k + l2] * dNg[l2 * NN + j];
                    T[k * NN + j] = t;
                    q += vt[k] * dNg[k * NN + j];
                }
                vd[j] = q;
            }
#pragma unroll
            for (int i = 0; i < NN; i++)
            {
                const double mi = mf * sf[i], si = fs * sf[i], ai = fkt * sf[i];
#pragma unroll
                for (int j = 0; j <= i; j++)
                {
                    const int l = i * (i + 1) / 2 + j;
                    Ml[l] += mi * sf[j];
                    St[l] += si * sf[j];
                    double g = 0.0;
#pragma unroll
                    for (int k = 0; k < DIM; k++) g += dNg[k * NN + i] * T[k * NN + j];
                    Ls[l] += fkt * g;
                }
#pragma unroll
                for (int j = 0; j < NN; j++) A[i * NN + j] += ai * vd[j];
            }
            if constexpr (SUPG)
            {
                // CalcSUPGWeightingFunction (fem_ele_std.cpp:4004-4025): w_i =
                // v . grad N_i with the raw flux; SUPG mass (CalcMass :3856-3879)
                // and advection (CalcAdvection :5467-5490) terms
                double Dr[DIM * DIM], wf[NN];
                dispersion_raw<DIM>(p, v, Dr);
                const double tau = supg_tau<DIM>(p, v, Dr, Lsupg);
#pragma unroll
                for (int i = 0; i < NN; i++)
                {
                    wf[i] = 0.0;
#pragma unroll
                    for (int k = 0; k < DIM; k++) wf[i] += dNg[k * NN + i] * v[k];
                }
#pragma unroll
                for (int i = 0; i < NN; i++)
#pragma unroll
                    for (int j = 0; j < NN; j++)
                    {
                        Mx[i * NN + j] += mf * tau * wf[i] * sf[j];
                        A[i * NN + j] += fkt * (1.0 * p.time_unit_factor) * tau * wf[i] * wf[j];
                    }
            }
        }
        if (!ok) { flag_bad(a.bad_elem, e); continue; }
        double L[NN * NN];
#pragma unroll
        for (int i = 0; i < NN; i++)
#pragma unroll
            for (int j = 0; j < NN; j++) L[i * NN + j] = Ls[i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i];
        if (p.mass_lumping)
        {
            // CalcLumpedMass has no SUPG term
            lump_mass<ET, NN>(X, Y, Z, cm, Ml);
            mt_combine<NN, SUPG>(a, e, nd, U, Ml, L, A, St);
        }
        else
            mt_combine<NN, SUPG>(a, e, nd, U, Ml, L, A, St, SUPG ? Mx : nullptr);
    }
}

// affine MASS_TRANSPORT on tets.  The FP64 pipe bounds the kernel (18 cycles
// a warp instruction on an SM), so what counts is the number of operations:
//  * The gradients are C_k / det, C_k the cofactors of the edges from corner 0
//    and C_0 = -(C_1 + C_2 + C_3).  |det| grad N needs no division, and the
//    Laplace C_k . D C_j / |det| one.
//  * |det| int N_i v . grad N_j = s W_i (v . C_j), s the sign of det and W_i =
//    sum_gp w N_i, when all five Gauss points hold the same flux bit for bit
//    (a linear head on an affine tet: Cal_Velocity gives one flux); then also
//    D = d I + c v v^T and C_k . D C_j = d C_k . C_j + c (v . C_k)(v . C_j),
//    whose last factors the advection has.  Else the points' tensors and the
//    vectors sum_gp w N_i v are summed first.
//  * Rows of the Laplace add to zero: corner 0's entries are sums of the
//    others.
//  * M and the decay term have two values a tet, added to the Laplace's six;
//    applied to u0 they take one sum.  For theta = 1 that is all of the
//    right-hand side.
// 6.29 million tets: 5.83 ms when each entry was built from the four stored
// element matrices (8.59 with five different fluxes a tet), 1.83 (4.73) so.
struct MtTetConst
{
    // per |det|, diagonal and off it: mass / dt + theta decay (matrix), mass /
    // dt - (1 - theta) decay (right-hand side)
    double ms_d, ms_o, mr_d, mr_o;
    double dm, al_at, at, tf, sw, th;
    double W[4], wN[5][4], w[5];
};

__global__ void __launch_bounds__(128) k_mt_tet_affine(AsmArgs a)
{
    constexpr int NN = 4, DIM = 3, NGP = 5;
    __shared__ MtTetConst s_c;
    if (threadIdx.x == 0)
    {
        const ogs_assembly_params& p = a.p;
        const double* N = a.tab;
        const double* w = a.tab + NGP * NN + NGP * NN * DIM;
        const double* M0 = a.aff + DIM * DIM * NN * NN;
        const double cm = p.steady ? 0.0 : p.porosity * p.saturation * p.retardation;
        const double cs = p.porosity * p.saturation * p.decay * p.retardation;
        const double dt_inverse = 1.0 / p.dt;
        // CalcLumpedMass: cm times volume / 4
        const double md = (p.mass_lumping ? cm * (1.0 / 24.0) : cm * M0[0]) * dt_inverse;
        const double mo = (p.mass_lumping ? 0.0 : cm * M0[1]) * dt_inverse;
        s_c.ms_d = md + p.theta * (cs * M0[0]);
        s_c.ms_o = mo + p.theta * (cs * M0[1]);
        s_c.mr_d = md - (1.0 - p.theta) * (cs * M0[0]);
        s_c.mr_o = mo - (1.0 - p.theta) * (cs * M0[1]);
        s_c.dm = p.diffusion * p.porosity * p.saturation;
        s_c.al_at = p.alpha_l - p.alpha_t;
        s_c.at = p.alpha_t;
        s_c.tf = p.time_unit_factor;
        s_c.th = p.theta;
        s_c.sw = 0.0;
        for (int i = 0; i < NN; i++) s_c.W[i] = 0.0;
        for (int gp = 0; gp < NGP; gp++)
        {
            s_c.w[gp] = w[gp * 3];
            s_c.sw += w[gp * 3];
            for (int i = 0; i < NN; i++)
            {
                s_c.wN[gp][i] = w[gp * 3] * N[gp * NN + i];
                s_c.W[i] += s_c.wN[gp][i];
            }
        }
    }
    __syncthreads();
    const MtTetConst& c = s_c;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < a.E;
         e += (int64_t)gridDim.x * blockDim.x)
    {
        int nd[NN];
        double C[3][4], U[NN], det;  // C: cofactor vectors of the corners
        {
            double X[NN], Y[NN], Z[NN];
            gather<NN>(a, e, nd, X, Y, Z, U);
            double d[3][3];
#pragma unroll
            for (int k = 0; k < 3; k++)
            {
                d[k][0] = X[k + 1] - X[0];
                d[k][1] = Y[k + 1] - Y[0];
                d[k][2] = Z[k + 1] - Z[0];
            }
#pragma unroll
            for (int k = 0; k < 3; k++)
#pragma unroll
                for (int q = 0; q < 3; q++)
                {
                    const int k1 = (k + 1) % 3, k2 = (k + 2) % 3, q1 = (q + 1) % 3, q2 = (q + 2) % 3;
                    C[q][k + 1] = d[k1][q1] * d[k2][q2] - d[k1][q2] * d[k2][q1];
                }
            det = d[0][0] * C[0][1] + d[0][1] * C[1][1] + d[0][2] * C[2][1];
        }
        if (fabs(det) < DBL_EPSILON) { flag_bad(a.bad_elem, e); continue; }
        const double* ve = a.gpv + e * NGP * 3;
        double v[3];
        bool same = true;
#pragma unroll
        for (int k = 0; k < 3; k++) v[k] = __ldg(ve + k);
#pragma unroll
        for (int gp = 1; gp < NGP; gp++)
#pragma unroll
            for (int k = 0; k < 3; k++)
                same = same && __double_as_longlong(__ldg(ve + gp * 3 + k)) == __double_as_longlong(v[k]);
        const double ad = fabs(det), id = c.tf / ad, sf = det < 0.0 ? -c.tf : c.tf, th = c.th;
        // the system from the Laplace entries of the corners 1..3 (11, 21, 22,
        // 31, 32, 33) and the advection adv(i, j)
        auto finish = [&](const double (&L)[6], auto adv) {
            const double l01 = -(L[0] + L[1] + L[3]), l02 = -(L[1] + L[2] + L[4]), l03 = -(L[3] + L[4] + L[5]);
            const double lap[10] = {-(l01 + l02 + l03), l01, L[0], l02, L[1], L[2], l03, L[3], L[4], L[5]};
            const double sd = ad * c.ms_d, so = ad * c.ms_o, rd = ad * c.mr_d, ro = ad * c.mr_o;
            const double ru = ro * (U[0] + U[1] + U[2] + U[3]);
            double r[NN];
#pragma unroll
            for (int i = 0; i < NN; i++) r[i] = ru + (rd - ro) * U[i];
            if (th == 1.0)
            {
#pragma unroll
                for (int i = 0; i < NN; i++)
#pragma unroll
                    for (int j = 0; j < NN; j++)
                    {
                        const int l = i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
                        scatter_entry(a, e, i * NN + j, a.val, adv(i, j) + (lap[l] + (i == j ? sd : so)));
                    }
            }
            else
            {
                const double th1 = 1.0 - th;
#pragma unroll
                for (int i = 0; i < NN; i++)
                {
                    double ku = 0.0;
#pragma unroll
                    for (int j = 0; j < NN; j++)
                    {
                        const int l = i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
                        const double k = adv(i, j) + lap[l];
                        scatter_entry(a, e, i * NN + j, a.val, (i == j ? sd : so) + k * th);
                        ku += k * U[j];
                    }
                    r[i] -= th1 * ku;
                }
            }
#pragma unroll
            for (int i = 0; i < NN; i++) atomicAdd(a.b + nd[i], r[i]);
        };
        double L[6];
        if (same)
        {
            const double v2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
            double dd = c.dm, dc = 0.0;
            if (v2 > DBL_EPSILON * DBL_EPSILON)
            {
                const double iv = rsqrt(v2);
                dd += c.at * (v2 * iv);
                dc = c.al_at * iv;
            }
            const double f = id * c.sw;
            dd *= f;
            dc *= f;
            double vc[4];
#pragma unroll
            for (int k = 1; k < 4; k++) vc[k] = v[0] * C[0][k] + v[1] * C[1][k] + v[2] * C[2][k];
#pragma unroll
            for (int k = 1; k < 4; k++)
#pragma unroll
                for (int l = 1; l <= k; l++)
                    L[k * (k - 1) / 2 + l - 1] =
                        dd * (C[0][k] * C[0][l] + C[1][k] * C[1][l] + C[2][k] * C[2][l]) + (dc * vc[k]) * vc[l];
#pragma unroll
            for (int k = 1; k < 4; k++) vc[k] *= sf;
            vc[0] = -(vc[1] + vc[2] + vc[3]);
            finish(L, [&](int i, int j) { return c.W[i] * vc[j]; });
        }
        else
        {
            double D[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, av[NN][3];
#pragma unroll
            for (int i = 0; i < NN; i++) av[i][0] = av[i][1] = av[i][2] = 0.0;
#pragma unroll 1
            for (int gp = 0; gp < NGP; gp++)
            {
                double x[3];
#pragma unroll
                for (int k = 0; k < 3; k++) x[k] = __ldg(ve + gp * 3 + k);
                const double v2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2], w = c.w[gp];
                double dd = c.dm, dc = 0.0;
                if (v2 > DBL_EPSILON * DBL_EPSILON)
                {
                    const double iv = rsqrt(v2);
                    dd += c.at * (v2 * iv);
                    dc = c.al_at * iv * w;
                }
                dd *= w;
#pragma unroll
                for (int k = 0; k < 3; k++)
#pragma unroll
                    for (int l = 0; l <= k; l++)
                        D[k * (k + 1) / 2 + l] += k == l ? dd + dc * (x[k] * x[k]) : dc * (x[k] * x[l]);
#pragma unroll
                for (int i = 0; i < NN; i++)
#pragma unroll
                    for (int k = 0; k < 3; k++) av[i][k] += c.wN[gp][i] * x[k];
            }
#pragma unroll
            for (int l = 1; l < 4; l++)
            {
                const double t0 = id * (D[0] * C[0][l] + D[1] * C[1][l] + D[3] * C[2][l]);
                const double t1 = id * (D[1] * C[0][l] + D[2] * C[1][l] + D[4] * C[2][l]);
                const double t2 = id * (D[3] * C[0][l] + D[4] * C[1][l] + D[5] * C[2][l]);
#pragma unroll
                for (int k = l; k < 4; k++) L[k * (k - 1) / 2 + l - 1] = C[0][k] * t0 + C[1][k] * t1 + C[2][k] * t2;
            }
            double A[NN][NN];
#pragma unroll
            for (int i = 0; i < NN; i++)
            {
#pragma unroll
                for (int j = 1; j < 4; j++) A[i][j] = sf * (av[i][0] * C[0][j] + av[i][1] * C[1][j] + av[i][2] * C[2][j]);
                A[i][0] = -(A[i][1] + A[i][2] + A[i][3]);
            }
            finish(L, [&](int i, int j) { return A[i][j]; });
        }
    }
}

// ------------------------------------------------------------------
// Gauss-point Darcy flux (Cal_Velocity scalar branch, fem_ele_std.cpp:6627-6870)
// ------------------------------------------------------------------
// q = -mat grad u / time_unit_factor (mat grad u + rho g on the last axis
// for LIQUID_FLOW with gravity)
template <int DIM>
__device__ __forceinline__ void darcy_flux(const ogs_assembly_params& p, double mat, double* vel, double* q)
{
    if (p.pcs_type == OGS_PCS_LIQUID_FLOW && p.gravity_on && p.gravity >= DBL_EPSILON)
        vel[DIM - 1] += p.gravity * p.density;
    q[0] = q[1] = q[2] = 0.0;
    // x / 1.0 is x: the division only where a factor is set
    const bool unit = p.time_unit_factor == 1.0;
#pragma unroll
    for (int i = 0; i < DIM; i++) q[i] -= unit ? mat * vel[i] : mat * vel[i] / p.time_unit_factor;
}

// One warp's staged fluxes (`per` doubles per lane, from sm) to the
// consecutive elements e0 .. : consecutive lanes write consecutive doubles.
// Element e's doubles start at out + e * stride; `rep` copies per element.
template <int PER, int REP>
__device__ __forceinline__ void write_staged(const double* sm, double* out, int64_t e0, int64_t E, int64_t stride)
{
    __syncwarp();
    const int n = (int)min((int64_t)32, E - e0);
    for (int f = threadIdx.x & 31; f < n * PER * REP; f += 32)
    {
        const int el = f / (PER * REP), k = f - el * (PER * REP);
        out[(e0 + el) * stride + k] = sm[el * PER + k % PER];
    }
    __syncwarp();
}

// quads: per Gauss point Jacobian and gradients
template <int NGP>
__global__ void __launch_bounds__(128) k_gp_velocity_quad(AsmArgs a)
{
    constexpr int NN = 4, DIM = 2;
    __shared__ double sdN[NGP * NN * DIM];
    stage(sdN, a.tab + NGP * NN, NGP * NN * DIM);
    __syncthreads();
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < a.E;
         e += (int64_t)gridDim.x * blockDim.x)
    {
        int nd[NN];
        double X[NN], Y[NN], Z[NN], U[NN];
        gather<NN>(a, e, nd, X, Y, Z, U);
        const double mat = flow_mat(a.p, __ldg(a.elem_k + e));
        double* qo = a.q_out + e * NGP * 3;
#pragma unroll 1
        for (int gp = 0; gp < NGP; gp++)
        {
            double iJ[DIM * DIM], det, dNg[DIM * NN], vel[3] = {0.0, 0.0, 0.0}, q[3];
            if (!jacobian<NN, DIM>(X, Y, Z, sdN + gp * NN * DIM, iJ, det)) { flag_bad(a.bad_elem, e); break; }
            grad_global<NN, DIM>(iJ, sdN + gp * NN * DIM, dNg);
#pragma unroll
            for (int i = 0; i < DIM; i++)
            {
                double s = 0.0;
#pragma unroll
                for (int j = 0; j < NN; j++) s += U[j] * dNg[i * NN + j];
                vel[i] = s;
            }
            darcy_flux<DIM>(a.p, mat, vel, q);
            qo[gp * 3 + 0] = q[0];
            qo[gp * 3 + 1] = q[1];
            qo[gp * 3 + 2] = q[2];
        }
    }
}

// Tets: the gradient is constant, so one flux serves the five Gauss points.
// Bound by the FP64 pipe (about 60 operations a tet: edge differences, the
// cofactors, one division) and the 120 B written per tet; the points' own
// Jacobians, inverses and divisions had made it about 840 operations, and
// the 15 stores a thread, 120 B apart, four times the sectors.  6.29M tets:
// 8365 us before, 680 us now (1.3 TB/s).
__global__ void __launch_bounds__(128) k_gp_velocity_tet(AsmArgs a)
{
    __shared__ double sq[4][32 * 3];
    double* sm = sq[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    for (int64_t e0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) - lane; e0 < a.E;
         e0 += (int64_t)gridDim.x * blockDim.x)
    {
        const int64_t e = e0 + lane;
        if (e < a.E)
        {
            int nd[4];
            double X[4], Y[4], Z[4], U[4];
            gather<4>(a, e, nd, X, Y, Z, U);
            const double mat = flow_mat(a.p, __ldg(a.elem_k + e));
            const double J[9] = {X[1] - X[0], Y[1] - Y[0], Z[1] - Z[0], X[2] - X[0], Y[2] - Y[0],
                                 Z[2] - Z[0], X[3] - X[0], Y[3] - Y[0], Z[3] - Z[0]};
            double C[9], det, q[3] = {0.0, 0.0, 0.0};
            if (!cofactors(J, C, det))
                flag_bad(a.bad_elem, e);
            else
            {
                const double id = 1.0 / det, d[3] = {U[1] - U[0], U[2] - U[0], U[3] - U[0]};
                double vel[3];
#pragma unroll
                for (int i = 0; i < 3; i++)
                    vel[i] = (C[3 * i] * d[0] + C[3 * i + 1] * d[1] + C[3 * i + 2] * d[2]) * id;
                darcy_flux<3>(a.p, mat, vel, q);
            }
#pragma unroll
            for (int k = 0; k < 3; k++) sm[lane * 3 + k] = q[k];
        }
        write_staged<3, 5>(sm, a.q_out, e0, a.E, 15);
    }
}

// Hexes, a slice of NG x NG Gauss points at a time: local derivatives of the
// heads (and, where the Jacobian varies, of the coordinates) by tensor
// products -- about 100 operations an element per field instead of 24 a
// Gauss point -- and the slice's fluxes staged per warp so that its stores
// are consecutive.  AFFINE: one Jacobian per element (its centre's).
// 250,047 boxes: 2729 us before, 264 us now; bound by the FP64 pipe.
template <int NG, bool AFFINE>
__global__ void __launch_bounds__(128) k_gp_velocity_hex(AsmArgs a)
{
    constexpr int PER = NG * NG * 3;
    __shared__ double sq[4][32 * PER];
    double* sm = sq[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    for (int64_t e0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) - lane; e0 < a.E;
         e0 += (int64_t)gridDim.x * blockDim.x)
    {
        const int64_t e = e0 + lane;
        const bool in = e < a.E;
        int nd[8];
        double X[8], Y[8], Z[8], U[8], mat = 0.0, G[9];
        bool ok = in;
        if (in)
        {
            gather<8>(a, e, nd, X, Y, Z, U);
            mat = flow_mat(a.p, __ldg(a.elem_k + e));
            if (AFFINE)
            {
                HexSlice<1> x, y, z;
                x.set(X, 0.5);
                y.set(Y, 0.5);
                z.set(Z, 0.5);
                const double J[9] = {x.dr[0][0], y.dr[0][0], z.dr[0][0], x.ds[0], y.ds[0],
                                     z.ds[0],    x.dt[0],    y.dt[0],    z.dt[0]};
                double det;
                ok = cofactors(J, G, det);
                const double id = 1.0 / det;
#pragma unroll
                for (int k = 0; k < 9; k++) G[k] *= id;
            }
        }
#pragma unroll 1
        for (int gr = 0; gr < NG; gr++)
        {
            const double h = gr == 0 ? shape1(NG, 0, 0) : gr == 1 ? shape1(NG, 1 % NG, 0) : shape1(NG, 2 % NG, 0);
            if (ok)
            {
                HexSlice<NG> u, x, y, z;
                u.set(U, h);
                if (!AFFINE)
                {
                    x.set(X, h);
                    y.set(Y, h);
                    z.set(Z, h);
                }
#pragma unroll
                for (int gs = 0; gs < NG; gs++)
#pragma unroll
                    for (int gt = 0; gt < NG; gt++)
                    {
                        double f = 1.0, vel[3], q[3];
                        if (!AFFINE)
                        {
                            const double J[9] = {x.dr[gs][gt], y.dr[gs][gt], z.dr[gs][gt], x.ds[gt], y.ds[gt],
                                                 z.ds[gt],     x.dt[gs],     y.dt[gs],     z.dt[gs]};
                            double det;
                            if (!cofactors(J, G, det)) ok = false;
                            f = 1.0 / det;
                        }
#pragma unroll
                        for (int i = 0; i < 3; i++)
                        {
                            vel[i] = G[3 * i] * u.dr[gs][gt] + G[3 * i + 1] * u.ds[gt] + G[3 * i + 2] * u.dt[gs];
                            if (!AFFINE) vel[i] *= f;
                        }
                        darcy_flux<3>(a.p, mat, vel, q);
#pragma unroll
                        for (int k = 0; k < 3; k++) sm[lane * PER + (gs * NG + gt) * 3 + k] = q[k];
                    }
            }
            write_staged<PER, 1>(sm, a.q_out + gr * PER, e0, a.E, (int64_t)NG * PER);
        }
        if (in && !ok) flag_bad(a.bad_elem, e);
    }
}

// ------------------------------------------------------------------
// RICHARDS_FLOW (fem_ele_std.cpp:9470-9481): AssembleParabolicEquation and
// Assemble_Gravity with the storage and conductivity of the Picard iterate
// at each Gauss point
// ------------------------------------------------------------------
__host__ __device__ __forceinline__ double mrange(double a, double b, double c)
{
    return b < a ? a : b > c ? c : b;  // MRange (FEM/mathlib.cpp:447)
}

// CMediumProperties::SaturationCapillaryPressureFunction, models 4 (van
// Genuchten) and 6 (Brooks-Corey) (rf_mmp_new.cpp:5243-5328)
// x^y for x >= 0 as exp(y log x): the curves' bases are never negative, and
// 0^y (0 for y > 0, inf for y < 0) comes out of log(0) = -inf.  Cheaper than
// pow on GB300's FP64 unit; the result is within |y log x| ulps of pow's
// (<= ~1e-14 relative on the curves' range)
__host__ __device__ __forceinline__ double powp(double x, double y) { return exp(y * log(x)); }

__host__ __device__ __forceinline__ double rich_saturation(const ogs_richards_params& r, double pc)
{
    // divisions by parameters as products with their reciprocals (loop
    // invariants of the Gauss-point loop; rounding-level differences)
    const double ipb = 1.0 / r.pb;
    double se;
    if (r.capillary_model == 4)
    {
        if (pc < 0.0) pc = 0.0;
        se = powp(pc * ipb, 1.0 / (1.0 - r.m)) + 1.0;
        se = powp(se, -r.m);
    }
    else
    {
        if (pc < r.pb) pc = r.pb;
        se = powp(pc * ipb, -r.m);
    }
    const double sl = se * (r.slm - r.slr) + r.slr;
    return mrange(r.slr + DBL_EPSILON, sl, r.slm - DBL_EPSILON);
}

// PressureSaturationDependency(Sw, invert = true): dSw/dpc (<= 0), bounded
// below by -1/DBL_EPSILON (rf_mmp_new.cpp:5425-5520)
__device__ __forceinline__ double rich_dsdpc(const ogs_richards_params& r, double sl)
{
    // dS/dpc = 1 / (dpc/dS) formed as one quotient; divisions by
    // parameters as products with their reciprocals
    const double isr = 1.0 / (r.slm - r.slr);
    double dsdp;
    if (r.capillary_model == 4)
    {
        sl = mrange(r.slr + DBL_EPSILON, sl, r.slm - DBL_EPSILON);
        const double v1 = powp((sl - r.slr) * isr, -1.0 / r.m);
        const double v2 = powp(v1 - 1.0, -r.m);
        dsdp = (r.m * (sl - r.slr)) / (r.pb * (r.m - 1.0) * v1 * v2);
    }
    else
    {
        sl = mrange(r.slr + DBL_EPSILON, sl, r.slm);
        const double v1 = powp((sl - r.slr) * isr, -1.0 / r.m);
        dsdp = (r.m * (r.slr - sl)) / (r.pb * v1);
    }
    const double lim = (-1.0) / DBL_EPSILON;
    if (dsdp < lim) dsdp = lim;
    return dsdp;
}

// PermeabilitySaturationFunction(Sw, 0), models 4 (van Genuchten-Mualem)
// and 6 (Brooks-Corey) (rf_mmp_new.cpp:2576-2635)
__host__ __device__ __forceinline__ double rich_krel(const ogs_richards_params& r, double sl)
{
    sl = mrange(r.kr_slr, sl, r.kr_slm);
    const double se = (sl - r.kr_slr) * (1.0 / (r.kr_slm - r.kr_slr));
    double kr;
    if (r.permeability_model == 4)
    {
        const double b = 1.0 - powp(1.0 - powp(se, 1.0 / r.kr_m), r.kr_m);
        kr = sqrt(se) * (b * b);
    }
    else
        kr = powp(se, 3.0 + 2.0 / r.kr_m);
    if (kr < r.kr_min) kr = r.kr_min;
    return kr;
}

// CalCoefMass, EPT_RICHARDS_FLOW (fem_ele_std.cpp:1721-1770), isothermal,
// constant drho_dp
__device__ __forceinline__ double rich_mass_coef(const ogs_assembly_params& p, const ogs_richards_params& r,
                                                 double PG)
{
    double Sw = 1.0, dSdp = 0.0;
    if (PG < 0.0)
    {
        Sw = rich_saturation(r, -PG);
        dSdp = -rich_dsdpc(r, Sw);
    }
    double val = p.storage * Sw;
    if (p.density > 0.0) val += p.porosity * Sw * p.drho_dp;
    if (PG < 0.0) val += p.porosity * dSdp;
    return val;
}

// CalCoefLaplace (fem_ele_std.cpp:2614-2640): K * (time_unit_factor *
// kr(Sw) / mu) * fac_perm (1), and CalCoefMass (:1721-1770), which reuses
// S(-PG), the same call, when unsaturated
//
// Three ways, by the point.  Saturated points (-PG <= 0, where the curves are
// constant) take the values formed once a launch, on the host.  Van Genuchten
// curves with the same m and limits for both curves: with
// t = (pc / pb)^(1 / (1 - m)),
//   Se = (1 + t)^-m, 1 - Se^(1/m) = t / (1 + t), dSe/dpc ~ y / (1 + t),
//   y = (t / (1 + t))^m, kr = Se^(1/2) (1 - y)^2,
// so the three curves share two logarithms and three exponentials instead of
// six powers (five of them of Se, which undo the first).  Against 80-bit
// arithmetic its errors are below those of the powers from t = 1e-6 to 1e6 and
// for m = 0.05 to 0.99 (Se 2e-16 to 4e-15, kr to 4e-15, ds/dpc to 1e-11 at t =
// 1e-6, m = 0.9, where the powers have 3e-10: their 1 - y and v1 - 1 cancel).
// t < 1e-6 and Se < 1e-3, where the general form's limits of the saturation
// act and its rounding is no longer small, keep the general form.  A warp that
// has such a point takes it for all of its unsaturated points: both forms one
// after the other made the few warps at a water table, and with them a mesh of
// one wave of blocks, slower than the powers alone.
// us of a call, with the powers / both forms a warp from t = 1e-3 on / here: 3,000
// quads 165 / 213 / 142, 196,608 boxes with the water table at mid-depth 5218 /
// 1702 / 1678, 600,000 hexes with node pressures in random order 17081 / 22884 / 7750.
static void rich_curves(const ogs_assembly_params& p, const ogs_richards_params& r, RichCurves& c)
{
    c.ivis = 1.0 / p.viscosity;
    c.sat = r.capillary_model == 4 || r.pb > 0.0;
    c.kr_sat = rich_krel(r, rich_saturation(r, 0.0));
    c.vg = r.capillary_model == 4 && r.permeability_model == 4 && r.kr_m == r.m && r.kr_slr == r.slr &&
           r.kr_slm == r.slm && r.pb > 0.0 && r.m >= 0.05 && r.m <= 0.99 && r.slm - r.slr >= 1e-3 && r.slr >= 0.0 &&
           r.slm <= 1.0 && r.m / (r.pb * (1.0 - r.m)) < 1e12;  // far from the limit on ds/dpc
    c.ipb = 1.0 / r.pb;
    c.m = r.m;
    c.n = 1.0 / (1.0 - r.m);
    c.slr = r.slr;
    c.dsl = r.slm - r.slr;
    c.cds = -(r.m * c.n) * c.ipb * c.dsl;
    c.lo = r.pb * pow(1e-6, 1.0 - r.m);
    c.hi = r.pb * pow(pow(1e3, 1.0 / r.m) - 1.0, 1.0 - r.m);
}

__device__ __forceinline__ void rich_coefficients(const ogs_assembly_params& p, const ogs_richards_params& r,
                                                  const RichCurves& c, double ke, double PG, double& mat, double& mc)
{
    double Sw = 1.0, kr = c.kr_sat, ds = 0.0;
    const bool sat = PG >= 0.0 && c.sat;
    bool general = !sat && !(c.vg && -PG >= c.lo && -PG <= c.hi);
    if (c.vg) general = __any_sync(__activemask(), general);
    if (!sat && general)
    {
        Sw = rich_saturation(r, -PG);
        kr = rich_krel(r, Sw);
        ds = PG < 0.0 ? rich_dsdpc(r, Sw) : 0.0;
    }
    else if (!sat)
    {
        // q = min(t, 1 / t): log(1 + t) and log((1 + t) / t) without a difference
        const double nl = c.n * log(-PG * c.ipb), q = exp(-fabs(nl)), w = log1p(q);
        const double h = exp(-0.5 * c.m * (w + fmax(nl, 0.0))), se = h * h;
        const double b = expm1(-c.m * (w + fmax(-nl, 0.0)));  // y - 1
        Sw = se * c.dsl + c.slr;
        kr = h * (b * b);
        if (kr < r.kr_min) kr = r.kr_min;
        ds = c.cds * ((1.0 + b) * ((nl > 0.0 ? q : 1.0) / (1.0 + q)));
    }
    mat = ke * (p.time_unit_factor * kr * c.ivis) * 1.0;
    const double Sm = PG < 0.0 ? Sw : 1.0;
    mc = p.storage * Sm;
    if (p.density > 0.0) mc += p.porosity * Sm * p.drho_dp;
    if (PG < 0.0) mc += p.porosity * -ds;
}

// element geometry constant over the Gauss points (see k_richards)
template <int ET>
__device__ __forceinline__ bool const_geometry(const double* X, const double* Y, const double* Z)
{
    if (ET == OGS_ELEM_TET4) return true;
    // r along x, s along y: J^-1 is then diagonal, as its users take it
    const bool rect = X[0] == X[3] && X[1] == X[2] && Y[0] == Y[1] && Y[2] == Y[3];
    if (ET == OGS_ELEM_QUAD4) return rect;
    bool box = rect && Z[0] == Z[1] && Z[0] == Z[2] && Z[0] == Z[3] && Z[4] == Z[5] && Z[4] == Z[6] && Z[4] == Z[7];
#pragma unroll
    for (int k = 0; k < 4; k++) box = box && X[k + 4] == X[k] && Y[k + 4] == Y[k];
    return box;
}

// quads and tets (hexes: k_flow_hex)
template <int ET, int NGP>
__global__ void __launch_bounds__(128) k_richards(AsmArgs a)
{
    constexpr int NN = ElemTraits<ET>::NN, DIM = ElemTraits<ET>::DIM;
    __shared__ double sN[NGP * NN], sdN[NGP * NN * DIM], sw[NGP * 3];
    stage(sN, a.tab, NGP * NN);
    stage(sdN, a.tab + NGP * NN, NGP * NN * DIM);
    stage(sw, a.tab + NGP * NN + NGP * NN * DIM, NGP * 3);
    __syncthreads();
    const ogs_assembly_params& p = a.p;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < a.E;
         e += (int64_t)gridDim.x * blockDim.x)
    {
        int nd[NN];
        double X[NN], Y[NN], Z[NN], U[NN], U1[NN];
        gather<NN>(a, e, nd, X, Y, Z, U);
#pragma unroll
        for (int i = 0; i < NN; i++) U1[i] = __ldg(a.u1 + nd[i]);
        const double ke = __ldg(a.elem_k + e);
        double Ml[NN * (NN + 1) / 2], Ll[NN * (NN + 1) / 2], grav[NN];
#pragma unroll
        for (int l = 0; l < NN * (NN + 1) / 2; l++) Ml[l] = Ll[l] = 0.0;
#pragma unroll
        for (int i = 0; i < NN; i++) grav[i] = 0.0;
        // geometry constant over the Gauss points: linear tets (constant shape
        // gradients), and quads that are axis-aligned rectangles (exact
        // coordinate equalities; J is then diagonal, its off-diagonal sums
        // cancel exactly): J^-1 and |J| from the first Gauss point
        const bool cgeo = const_geometry<ET>(X, Y, Z);
        double iJ[DIM * DIM], det = 0.0, dNg[DIM * NN];
        bool ok = !cgeo || jacobian<NN, DIM>(X, Y, Z, sdN, iJ, det);
        if (ok && cgeo && ET == OGS_ELEM_TET4) grad_global<NN, DIM>(iJ, sdN, dNg);
#pragma unroll 1
        for (int gp = 0; gp < NGP && ok; gp++)
        {
            const double* dNr = sdN + gp * NN * DIM;
            if (!cgeo)
            {
                if (!jacobian<NN, DIM>(X, Y, Z, dNr, iJ, det)) { ok = false; break; }
                grad_global<NN, DIM>(iJ, dNr, dNg);
            }
            else if (ET != OGS_ELEM_TET4)
            {
#pragma unroll
                for (int k = 0; k < DIM; k++)
#pragma unroll
                    for (int i = 0; i < NN; i++) dNg[k * NN + i] = iJ[k * DIM + k] * dNr[k * NN + i];
            }
            const double* w = sw + gp * 3;
            const double fkt = ET == OGS_ELEM_QUAD4 ? det * w[0] * w[1] : det * w[0];
            const double* sf = sN + gp * NN;
            double PG = 0.0;  // interpolate(NodalVal1)
#pragma unroll
            for (int i = 0; i < NN; i++) PG += U1[i] * sf[i];
            double mat, mc;
            rich_coefficients(p, a.r, a.rc, ke, PG, mat, mc);
            const double mf = mc * fkt * 1.0;
            const double cl = fkt * mat;
#pragma unroll
            for (int i = 0; i < NN; i++)
            {
                const double mi = mf * sf[i];
#pragma unroll
                for (int j = 0; j <= i; j++)
                {
                    const int l = i * (i + 1) / 2 + j;
                    Ml[l] += mi * sf[j];
                    double g = 0.0;
#pragma unroll
                    for (int k = 0; k < DIM; k++) g += dNg[k * NN + i] * dNg[k * NN + j];
                    Ll[l] += cl * g;
                }
            }
            if (p.gravity_on)
            {
                // Assemble_Gravity (:5859-6000): rho g, or 1 in the head form
                const double rho = p.gravity < DBL_EPSILON ? 1.0 : p.density * p.gravity;
                const double fg = fkt * rho;
#pragma unroll
                for (int i = 0; i < NN; i++) grav[i] -= fg * dNg[(DIM - 1) * NN + i] * mat;
            }
        }
        if (!ok) { flag_bad(a.bad_elem, e); continue; }
        if (p.mass_lumping)
        {
            // CalcLumpedMass: CalCoefMass at the element centre (equal shape
            // function values 1/NN there)
            double PG = 0.0;
#pragma unroll
            for (int i = 0; i < NN; i++) PG += U1[i] * (1.0 / NN);
            lump_mass<ET, NN>(X, Y, Z, rich_mass_coef(p, a.r, PG), Ml);
        }
        flow_combine<NN>(a, e, nd, U, Ml, Ll, grav);
    }
}

// ------------------------------------------------------------------
// Hexahedra with varying coefficients or Jacobians (see HexSums)
// ------------------------------------------------------------------
// N_+ and weight of point g on the r axis (a run-time index: the slices are
// one loop body)
template <int NG>
__device__ __forceinline__ void slice_point(int g, double& h, double& w)
{
    h = shape1(NG, 0, 0);
    w = gauss_w(NG, 0);
    if (NG > 1 && g == 1) { h = shape1(NG, 1 % NG, 0); w = gauss_w(NG, 1 % NG); }
    if (NG > 2 && g == 2) { h = shape1(NG, 2 % NG, 0); w = gauss_w(NG, 2 % NG); }
}

// C_ab = f sum_i cof[3 i + a] cof[3 i + b]: rr, ss, tt, rs, rt, st
__device__ __forceinline__ void metric(const double (&C)[9], double f, double (&G)[6])
{
#pragma unroll
    for (int k = 0; k < 6; k++)
    {
        const int a = k < 3 ? k : k == 5 ? 1 : 0, b = k < 3 ? k : k == 3 ? 1 : 2;
        G[k] = f * (C[a] * C[b] + C[3 + a] * C[3 + b] + C[6 + a] * C[6 + b]);
    }
}

// GROUNDWATER_FLOW / LIQUID_FLOW on hexes that are not affine, and
// RICHARDS_FLOW (RICH) on all hexes.  The gravity vector of element i,
// -rho g sum_gp w |J| mat dN_i/dz, is the Laplace form applied to the z
// coordinate (the isoparametric map reproduces it exactly), taken relative
// to corner 0.  Two blocks of 128 threads per SM (their sums fill the
// shared memory).
// 151,951 distorted hexes: 2896 us as direct sums, 978 us now; Richards on
// 196,608 boxes: 5370 us before, 1680 us now, with the curves of
// rich_coefficients.
template <int NG, bool RICH>
__global__ void __launch_bounds__(kHexThreads, 2) k_flow_hex(AsmArgs a)
{
    extern __shared__ double sums[];
    const ogs_assembly_params& p = a.p;
    const double cm = flow_mass_coef(p), dt_inverse = 1.0 / p.dt;
    double relax0 = p.nls_relaxation;
    if (relax0 < DBL_MIN) relax0 = 1.0;
    const double relax1 = 1.0 - relax0;
    const bool grav = (RICH || p.pcs_type == OGS_PCS_LIQUID_FLOW) && p.gravity_on;
    const double rho = p.gravity < DBL_EPSILON ? 1.0 : p.density * p.gravity;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < a.E; e += (int64_t)gridDim.x * blockDim.x)
    {
        int nd[8];
        double X[8], Y[8], Z[8], U[8], V[8];
        gather<8>(a, e, nd, X, Y, Z, U);
        if (RICH)
#pragma unroll
            for (int i = 0; i < 8; i++) V[i] = __ldg(a.u1 + nd[i]);
        const double ke = __ldg(a.elem_k + e), mat = RICH ? ke : flow_mat(p, ke);
        HexSums<NG, true, false, true> H;
        H.start(sums);
        // boxes along the axes: one diagonal Jacobian
        const bool box = RICH && const_geometry<OGS_ELEM_HEX8>(X, Y, Z);
        double det = 0.0, G[6];
        bool ok = true;
        if (box)
        {
            const double J0 = 0.5 * (X[0] - X[1]), J4 = 0.5 * (Y[0] - Y[3]), J8 = 0.5 * (Z[0] - Z[4]);
            det = fabs(J0 * J4 * J8);
            ok = !(det < DBL_EPSILON);
            G[0] = 0.25 * det / (J0 * J0);
            G[1] = 0.25 * det / (J4 * J4);
            G[2] = 0.25 * det / (J8 * J8);
        }
#pragma unroll 1
        for (int gr = 0; gr < NG && ok; gr++)
        {
            double h, wr;
            slice_point<NG>(gr, h, wr);
            HexSlice<NG> x, y, z;
            if (!box)
            {
                x.set(X, h);
                y.set(Y, h);
                z.set(Z, h);
            }
            double pc[4];  // the iterate at the slice's corners p + 2 q of (s, t)
            if (RICH)
#pragma unroll
                for (int c = 0; c < 4; c++)
                    pc[c] = h * V[hex_node(0, c & 1, c >> 1)] + (1.0 - h) * V[hex_node(1, c & 1, c >> 1)];
            H.start_slice();
#pragma unroll
            for (int gs = 0; gs < NG; gs++)
            {
                double L[6][NG], m[NG], f[NG], ds[NG];
                const double p0 = RICH ? shape1(NG, gs, 0) * pc[0] + shape1(NG, gs, 1) * pc[1] : 0.0;
                const double p1 = RICH ? shape1(NG, gs, 0) * pc[2] + shape1(NG, gs, 1) * pc[3] : 0.0;
#pragma unroll
                for (int gt = 0; gt < NG; gt++)
                {
                    const double w = (gauss_w(NG, gs) * gauss_w(NG, gt)) * wr;
                    double cl = mat, cc = cm;
                    if (RICH)
                    {
                        const double PG = shape1(NG, gt, 0) * p0 + shape1(NG, gt, 1) * p1;
                        rich_coefficients(p, a.r, a.rc, ke, PG, cl, cc);
                    }
                    if (box)
                    {
                        const double wc = w * cl;
                        m[gt] = w * det * cc;
#pragma unroll
                        for (int k = 0; k < 3; k++)
                        {
                            L[k][gt] = wc * G[k];
                            L[3 + k][gt] = 0.0;
                        }
                    }
                    else
                    {
                        const double J[9] = {x.dr[gs][gt], y.dr[gs][gt], z.dr[gs][gt], x.ds[gt], y.ds[gt],
                                             z.ds[gt],     x.dt[gs],     y.dt[gs],     z.dt[gs]};
                        double C[9], d;
                        ok = cofactors(J, C, d) && ok;
                        ds[gt] = d = fabs(d);
                        m[gt] = w * d * cc;
                        metric(C, 1.0, G);
                        f[gt] = 0.25 * w * cl;
#pragma unroll
                        for (int k = 0; k < 6; k++) L[k][gt] = G[k];
                    }
                }
                if (!box)
                {
                    // one division for the row's points: 1 / d_t = (1 / prod d)
                    // times the other d
                    double prod = ds[0], other[NG];
#pragma unroll
                    for (int t = 1; t < NG; t++) prod *= ds[t];
                    const double inv = 1.0 / prod;
#pragma unroll
                    for (int t = 0; t < NG; t++)
                    {
                        other[t] = 1.0;
#pragma unroll
                        for (int q = 0; q < NG; q++)
                            if (q != t) other[t] *= ds[q];
                        f[t] *= other[t] * inv;
#pragma unroll
                        for (int k = 0; k < 6; k++) L[k][t] *= f[t];
                    }
                }
                if (box)
                    H.template add_lap<true>(gs, L);
                else
                    H.template add_lap<false>(gs, L);
                H.add_mass(gs, m);
            }
            H.end_slice(h);
        }
        if (!ok) { flag_bad(a.bad_elem, e); continue; }
        double fl = 0.0;
        if (p.mass_lumping)
        {
            // CalcLumpedMass; Richards: CalCoefMass at the element centre
            double cc = cm;
            if (RICH)
            {
                double PG = 0.0;
#pragma unroll
                for (int i = 0; i < 8; i++) PG += V[i] * (1.0 / 8);
                cc = rich_mass_coef(p, a.r, PG);
            }
            fl = cc * (element_volume<OGS_ELEM_HEX8>(X, Y, Z) / 8.0);
        }
        double rr[3][3], r[8];
        H.finish(rr);
#pragma unroll
        for (int i = 0; i < 8; i++) r[i] = 0.0;
        // AssembleParabolicEquation: M / dt + relax0 L, (M / dt - relax1 L) u0
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j <= i; j++)
            {
                const double l = H.lap(rr, i, j);
                const double m = (p.mass_lumping ? (i == j ? fl : 0.0) : H.mass(i, j)) * dt_inverse;
                const double S = m + l * relax0, T = m - l * relax1;
                scatter_entry(a, e, i * 8 + j, a.val, S);
                r[i] += T * U[j];
                if (grav) r[i] -= rho * (l * (Z[j] - Z[0]));
                if (i != j)
                {
                    scatter_entry(a, e, j * 8 + i, a.val, S);
                    r[j] += T * U[i];
                    if (grav) r[j] -= rho * (l * (Z[i] - Z[0]));
                }
            }
#pragma unroll
        for (int i = 0; i < 8; i++) atomicAdd(a.b + nd[i], r[i]);
    }
}

// MASS_TRANSPORT on hexes, without SUPG.  In local coordinates the
// dispersion form needs w |J| (s J^-1 J^-T + c v' v'^T), v' = J^-1 v, with
// D = s I + c v v^T (MassDispersionTensorNew): 1 / |v| comes from one
// reciprocal square root.  AFFINE: one Jacobian an element (its centre's)
// and the mass from the reference tensor M0.  One block of 128 threads per
// SM (120 to 147 KB of sums).
// 250,047 boxes: 7746 us as direct sums, 2172 us now.
template <int NG, bool AFFINE>
__global__ void __launch_bounds__(kHexThreads, 1) k_mt_hex(AsmArgs a)
{
    extern __shared__ double sums[];
    const ogs_assembly_params& p = a.p;
    const double cm = p.steady ? 0.0 : p.porosity * p.saturation * p.retardation;
    const double cs = p.porosity * p.saturation * p.decay * p.retardation;
    const double dm = p.diffusion * p.porosity * p.saturation, al_at = p.alpha_l - p.alpha_t, tf = p.time_unit_factor;
    const double dt_inverse = 1.0 / p.dt, th = p.theta, th1 = 1.0 - p.theta;
    const double* M0 = a.aff + 9 * 64;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < a.E; e += (int64_t)gridDim.x * blockDim.x)
    {
        int nd[8];
        double X[8], Y[8], Z[8], U[8];
        gather<8>(a, e, nd, X, Y, Z, U);
        HexSums<NG, true, true, !AFFINE> H;
        H.start(sums);
        double C[9], G0[6], det = 0.0, qd = 0.0, hs = 0.5;  // 1 / (4 |det|), sign of det / 2
        bool ok = true;
        if (AFFINE)
        {
            HexSlice<1> x, y, z;
            x.set(X, 0.5);
            y.set(Y, 0.5);
            z.set(Z, 0.5);
            const double J[9] = {x.dr[0][0], y.dr[0][0], z.dr[0][0], x.ds[0], y.ds[0],
                                 z.ds[0],    x.dt[0],    y.dt[0],    z.dt[0]};
            ok = cofactors(J, C, det);
            metric(C, 1.0, G0);
            qd = 0.25 / fabs(det);
            hs = det < 0.0 ? -0.5 : 0.5;
        }
        const double* ve = a.gpv + e * (NG * NG * NG * 3);
#pragma unroll 1
        for (int gr = 0; gr < NG && ok; gr++)
        {
            double h, wr;
            slice_point<NG>(gr, h, wr);
            const double wrt = wr * tf;
            HexSlice<NG> x, y, z;
            if (!AFFINE)
            {
                x.set(X, h);
                y.set(Y, h);
                z.set(Z, h);
            }
            H.start_slice();
#pragma unroll
            for (int gs = 0; gs < NG; gs++)
            {
                double L[6][NG], A[3][NG], m[NG];
#pragma unroll
                for (int gt = 0; gt < NG; gt++)
                {
                    const double g = gauss_w(NG, gs) * gauss_w(NG, gt), wt = g * wrt;
                    const double* vp = ve + ((gr * NG + gs) * NG + gt) * 3;
                    const double v[3] = {__ldg(vp), __ldg(vp + 1), __ldg(vp + 2)};
                    double G[6];
                    if (!AFFINE)
                    {
                        const double J[9] = {x.dr[gs][gt], y.dr[gs][gt], z.dr[gs][gt], x.ds[gt], y.ds[gt],
                                             z.ds[gt],     x.dt[gs],     y.dt[gs],     z.dt[gs]};
                        ok = cofactors(J, C, det) && ok;
                        metric(C, 1.0, G);
                        m[gt] = (g * wr) * fabs(det);
                        qd = 0.25 / fabs(det);
                        hs = det < 0.0 ? -0.5 : 0.5;
                    }
                    const double id = wt * qd, wa = wt * hs;
                    double cv[3];
#pragma unroll
                    for (int k = 0; k < 3; k++) cv[k] = v[0] * C[k] + v[1] * C[3 + k] + v[2] * C[6 + k];
                    const double vv = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
                    double sd = dm, cd = 0.0;
                    if (vv > DBL_EPSILON * DBL_EPSILON)
                    {
                        const double iv = rsqrt(vv);
                        sd = p.alpha_t * (vv * iv) + dm;
                        cd = al_at * iv;
                    }
                    sd *= id;
                    cd *= id;
                    const double cx = cd * cv[0], cy = cd * cv[1], cz = cd * cv[2];
                    const double q[6] = {cx * cv[0], cy * cv[1], cz * cv[2], cx * cv[1], cx * cv[2], cy * cv[2]};
#pragma unroll
                    for (int k = 0; k < 6; k++) L[k][gt] = sd * (AFFINE ? G0[k] : G[k]) + q[k];
#pragma unroll
                    for (int k = 0; k < 3; k++) A[k][gt] = wa * cv[k];
                }
                H.template add_lap<false>(gs, L);
                H.add_adv(gs, A);
                if (!AFFINE) H.add_mass(gs, m);
            }
            H.end_slice(h);
        }
        if (!ok) { flag_bad(a.bad_elem, e); continue; }
        const double fl = p.mass_lumping ? cm * (element_volume<OGS_ELEM_HEX8>(X, Y, Z) / 8.0) : 0.0;
        double rr[3][3], r[8];
        H.finish(rr);
        det = fabs(det);
#pragma unroll
        for (int i = 0; i < 8; i++) r[i] = 0.0;
        // AssembleMixedHyperbolicParabolicEquation (fem_ele_std.cpp:8592-8692),
        // or (a.val2) the mass and the operator stored for memory_type > 0
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j <= i; j++)
            {
                const double mij = AFFINE ? det * __ldg(M0 + i * 8 + j) : H.mass(i, j);
                const double m = p.mass_lumping ? (i == j ? fl : 0.0) : cm * mij;
                const double ls = H.lap(rr, i, j) + cs * mij;
#pragma unroll
                for (int q = 0; q < 2; q++)
                {
                    if (q && i == j) continue;
                    const int s = q ? j : i, t = q ? i : j;
                    const double k = ls + H.adv(s, t);
                    if (a.val2)
                    {
                        scatter_entry(a, e, s * 8 + t, a.val, m);
                        scatter_entry(a, e, s * 8 + t, a.val2, k);
                        continue;
                    }
                    const double md = m * dt_inverse;
                    scatter_entry(a, e, s * 8 + t, a.val, md + k * th);
                    r[s] += (md - k * th1) * U[t];
                }
            }
        if (a.val2) continue;
#pragma unroll
        for (int i = 0; i < 8; i++) atomicAdd(a.b + nd[i], r[i]);
    }
}

static int grid_for(int64_t E, int threads, int per_sm = 16)
{
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t need = (E + threads - 1) / threads;
    const int64_t cap = (int64_t)sms * per_sm;
    return (int)std::max<int64_t>(1, std::min(need, cap));
}

constexpr int gauss_axis(int ngp) { return ngp == 27 ? 3 : ngp == 8 ? 2 : 1; }

// a sum-factorised hex kernel with `cols` shared sums per thread
static void launch_hex(void (*kernel)(AsmArgs), int cols, const AsmArgs& a, cudaStream_t s)
{
    const int bytes = cols * kHexThreads * (int)sizeof(double);
    cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    kernel<<<grid_for(a.E, kHexThreads), kHexThreads, bytes, s>>>(a);
}

template <int ET, int NGP>
static void launch_flow(const AsmArgs& a, bool affine, cudaStream_t s)
{
    const int g = grid_for(a.E, 128);
    if (affine)
        k_flow_affine<ET><<<g, 128, 0, s>>>(a);
    else if constexpr (ET == OGS_ELEM_HEX8)
    {
        constexpr int NG = gauss_axis(NGP);
        launch_hex(k_flow_hex<NG, false>, HexSums<NG, true, false, true>::kCols, a, s);
    }
    else
        k_flow_general<ET, NGP><<<g, 128, 0, s>>>(a);
}

template <int ET, int NGP>
static void launch_mt(const AsmArgs& a, bool affine, cudaStream_t s)
{
    const int g = grid_for(a.E, 128);
    // the affine tet kernel folds the Gauss points away; SUPG needs them.
    // Filling the stored operators (a.val2) goes through the SUPG kernel,
    // exact for supg_method 0 too (tau = 0 adds zeros), but on hexes.
    if constexpr (ET == OGS_ELEM_HEX8)
    {
        constexpr int NG = gauss_axis(NGP);
        if (a.p.supg_method > 0)
            k_mt_general<ET, NGP, true><<<g, 128, 0, s>>>(a);
        else if (affine)
            launch_hex(k_mt_hex<NG, true>, HexSums<NG, true, true, false>::kCols, a, s);
        else
            launch_hex(k_mt_hex<NG, false>, HexSums<NG, true, true, true>::kCols, a, s);
    }
    else if (a.val2 || a.p.supg_method > 0)
        k_mt_general<ET, NGP, true><<<g, 128, 0, s>>>(a);
    else if (ET == OGS_ELEM_TET4 && affine)
        k_mt_tet_affine<<<g, 128, 0, s>>>(a);
    else
        k_mt_general<ET, NGP, false><<<g, 128, 0, s>>>(a);
}

template <int ET, int NGP>
static void launch_richards(AsmArgs a, cudaStream_t s)
{
    rich_curves(a.p, a.r, a.rc);
    if constexpr (ET == OGS_ELEM_HEX8)
    {
        constexpr int NG = gauss_axis(NGP);
        launch_hex(k_flow_hex<NG, true>, HexSums<NG, true, false, true>::kCols, a, s);
    }
    else
        k_richards<ET, NGP><<<grid_for(a.E, 128), 128, 0, s>>>(a);
}

template <int ET, int NGP>
static void launch_vel(const AsmArgs& a, bool affine, cudaStream_t s)
{
    const int g = grid_for(a.E, 128);
    if constexpr (ET == OGS_ELEM_TET4)
        k_gp_velocity_tet<<<g, 128, 0, s>>>(a);
    else if constexpr (ET == OGS_ELEM_QUAD4)
        k_gp_velocity_quad<NGP><<<g, 128, 0, s>>>(a);
    else
    {
        constexpr int NG = gauss_axis(NGP);
        if (affine)
            k_gp_velocity_hex<NG, true><<<g, 128, 0, s>>>(a);
        else
            k_gp_velocity_hex<NG, false><<<g, 128, 0, s>>>(a);
    }
}

// Cell coefficients of the flow operator on a regular hex lattice.  Without
// mass lumping the left-hand side flow_combine scatters is
// sum_c (alpha_c L_box + beta M_box) with alpha_c = relax0 * mat(K_c) and
// beta = CalCoefMass / dt, L_box and M_box the Laplace and mass matrices of
// the unit-coefficient box; the FP32 inner CG applies the operator from
// these (summed over the assemblies since Initialize).  beta sits at
// coef[E].
__global__ void k_flow_cell_coef(ogs_assembly_params p, const double* __restrict__ elem_k, int64_t E,
                                 double* coef)
{
    double relax0 = p.nls_relaxation;
    if (relax0 < DBL_MIN) relax0 = 1.0;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x)
        coef[e] += relax0 * flow_mat(p, __ldg(elem_k + e));
    if (blockIdx.x == 0 && threadIdx.x == 0) coef[E] += flow_mass_coef(p) * (1.0 / p.dt);
}

void launch_flow_cell_coef(const AsmArgs& a, double* coef, cudaStream_t s)
{
    k_flow_cell_coef<<<grid_for(a.E, 256), 256, 0, s>>>(a.p, a.elem_k, a.E, coef);
}

// dispatch on (element type, Gauss points); returns false for an
// unsupported combination.  Flow on a regular hex or quad lattice takes the
// row kernel (not for the split assembly of memory_type, which needs the terms
// apart)
bool launch_assembly(const ogs_mesh* m, const AsmArgs& a, bool affine, int kind,
                     cudaStream_t s)
{
    const int et = m->elem_type, ngp = m->ngp;
    if (kind == 0 && (m->grid || m->grid2d) && affine && !a.val2 &&
        (a.p.pcs_type == OGS_PCS_GROUNDWATER_FLOW || a.p.pcs_type == OGS_PCS_LIQUID_FLOW))
    {
        LatticeArgs g;
        g.slice_ptr = m->slice_ptr;
        g.nx = m->gx; g.ny = m->gy; g.nz = m->gz;
        g.n = m->n_nodes;
        double relax0 = a.p.nls_relaxation;
        if (relax0 < DBL_MIN) relax0 = 1.0;
        // as many blocks as are resident: each forms the tables once (a chain
        // of FP64 operations of about 10 us in one thread, 8 blocks after each
        // other on an SM: 410 us for 1.08 million hex rows, 283 so with the
        // tables by 16 threads; 20,900 rows 28 and 18)
        if (m->grid2d)
        {
            if (relax0 == 1.0)
                k_flow_lattice_quad<true><<<grid_for(g.n, 256, 4), 256, 0, s>>>(a, g);
            else
                k_flow_lattice_quad<false><<<grid_for(g.n, 256, 4), 256, 0, s>>>(a, g);
        }
        else if (relax0 == 1.0)
            k_flow_lattice<true><<<grid_for(g.n, 256, 2), 256, 0, s>>>(a, g);
        else
            k_flow_lattice<false><<<grid_for(g.n, 256, 2), 256, 0, s>>>(a, g);
        return true;
    }
#define OGS_DISPATCH(ET_, NGP_)                                      \
    if (et == ET_ && ngp == NGP_)                                    \
    {                                                                \
        if (kind == 0) launch_flow<ET_, NGP_>(a, affine, s);         \
        else if (kind == 1) launch_mt<ET_, NGP_>(a, affine, s);      \
        else if (kind == 3) launch_richards<ET_, NGP_>(a, s);        \
        else launch_vel<ET_, NGP_>(a, affine, s);                            \
        return true;                                                 \
    }
    OGS_DISPATCH(OGS_ELEM_QUAD4, 1)
    OGS_DISPATCH(OGS_ELEM_QUAD4, 4)
    OGS_DISPATCH(OGS_ELEM_QUAD4, 9)
    OGS_DISPATCH(OGS_ELEM_HEX8, 1)
    OGS_DISPATCH(OGS_ELEM_HEX8, 8)
    OGS_DISPATCH(OGS_ELEM_HEX8, 27)
    OGS_DISPATCH(OGS_ELEM_TET4, 5)
#undef OGS_DISPATCH
    return false;
}

}  // namespace ogs

unsigned long long ogs_oob_assembly() { return ogs::oob_take(); }
