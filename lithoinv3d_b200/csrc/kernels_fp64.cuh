// FP64 device kernels of the LithoInv hot path (sm_100a).
//
// Forward (station per thread, facet records staged in shared memory): the
// facet sums of faceNagyContribution / magneticFacet / solidAngle /
// lineIntegralTerm of the reference
// (modules/litho-forward/src/forward/gravity_forward.cpp:13-42,
//  modules/litho-forward/src/forward/magnetic_forward.cpp:312-347,
//  modules/litho-core/src/core/geometry.cpp:10-52).  Close to a facet's edges
// and in its plane every operation is the reference's, in its order, so that
// its branches are taken as it takes them; everywhere else the same sums in the
// symmetric form, by polynomials.  The station-independent facet quantities
// (unit normal, edge lengths, in-plane edge normals, magnetic direction
// products) are computed once per facet by face_consts_fwd, in the reference's
// operation order.
//
// Gradient (objective: a warp per facet, lanes over the stations; Jacobian rows:
// a thread per facet and station): the derivative of every facet term with
// respect to its three vertices, in closed form, contracted with the
// per-station weighted residual in the same pass so the Jacobian is never
// stored.  Derivation (per facet, local frame
// with origin at vertex a, x along a->b, z along the unit normal):
//   d Lambda_e / d p2 = ( e_hat - q W ) / d2,   d Lambda_e / d p1 = (-e_hat - q W) / d1,
//   d Omega / d p1 += (e_hat x r1) W / d1,      d Omega / d p2 += (e_hat x r1) W / d2,
// with r1 = p1 - o, q = r1 - (r1.e_hat) e_hat, W = L / (d1 d2 + r1.r2); the
// station-independent factors (n_z, n_hat, in-plane edge normals, magnetic
// direction products) are differentiated once per facet from accumulated
// station sums.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace litho_b200 {

constexpr double kEps = 1e-15;
constexpr double kPi = 3.14159265358979323846;

// ---------------------------------------------------------------- layouts --
// Forward facet record, AoS [T][NFC], 16-byte aligned (NFC even): a CTA copies
// its facets' records as one contiguous range and a warp reads a record with
// 128-bit broadcast loads.
enum FwdConst {
    FC_AX = 0, FC_AY, FC_AZ, FC_BX, FC_BY, FC_BZ, FC_CX, FC_CY, FC_CZ,
    FC_AREA2,                          // |(b-a) x (c-a)|; -1 for a facet that contributes nothing
    FC_NX, FC_NY, FC_NZ,               // unit normal
    FC_NZ2,                            // 2 n_z
    FC_L0, FC_L1, FC_L2,               // edge lengths
    FC_HL0, FC_HL1, FC_HL2,            // half their squares
    FC_P0X, FC_P0Y, FC_P0Z, FC_P1X, FC_P1Y, FC_P1Z, FC_P2X, FC_P2Y, FC_P2Z,  // in-plane edge normals
    FC_MF2, FC_MT0, FC_MT1, FC_MT2,    // magnetic direction products, doubled
    FC_PAD,
    NFC
};
static_assert(NFC % 2 == 0, "records are copied 16 bytes at a time");

// Gradient facet constants (local frame), SoA [NGC][T].
enum GradConst {
    GC_AX = 0, GC_AY, GC_AZ,           // origin (vertex a)
    GC_XX, GC_XY, GC_XZ,               // local x axis (global components)
    GC_YX, GC_YY, GC_YZ,               // local y axis
    GC_ZX, GC_ZY, GC_ZZ,               // local z axis = unit normal
    GC_L0, GC_CX, GC_CY,               // b = (L0, 0, 0), c = (CX, CY, 0)
    GC_E1X, GC_E1Y, GC_L1,             // edge b->c direction and length
    GC_E2X, GC_E2Y, GC_L2,             // edge c->a direction and length
    GC_GS,                             // gz scale of the facet's group (0: no gravity)
    GC_MS,                             // TMI scale of the facet's group (0: skipped)
    GC_MF, GC_MT0, GC_MT1, GC_MT2,     // magnetic direction products
    GC_FLAGS,                          // bit0 valid facet, bit1 needs gradient
    NGC
};

struct GroupConst {
    double gscale_fwd;  // G * rho * 1e3 * 1e5 (forward association)
    double gscale_jac;  // (G * 1e3 * 1e5) * rho (Jacobian association)
    double mscale;      // magnetization amplitude * 100 / (4 pi)
    double mdir[3];
    int mag_active;     // amplitude >= 1e-15 (the Jacobian skips weaker groups)
};

// ------------------------------------------------------------- utilities --
struct d3 { double x, y, z; };
__device__ __forceinline__ d3 mk3(double x, double y, double z) { return {x, y, z}; }
__device__ __forceinline__ d3 operator-(d3 a, d3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ d3 operator+(d3 a, d3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ d3 operator*(d3 a, double s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ double dot3(d3 a, d3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ d3 cross3(d3 a, d3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ double norm3(d3 a) { return sqrt(dot3(a, a)); }

// lineIntegralTerm branch semantics (geometry.cpp:39-51) given s1, s2, d1, d2.
__device__ __forceinline__ double lambda_from(double s1, double s2, double d1, double d2, bool* live) {
    double num = s2 + d2, den = s1 + d1;
    *live = false;
    if (fabs(den) < kEps) return 0.0;  // covers the "both ~0" branch too
    if (num <= 0.0 || den <= 0.0) return 0.0;
    *live = true;
    return log(num / den);
}

// Lambda in the symmetric form log((d1 + d2 + L) / (d1 + d2 - L)) =
// log1p(2 L / (d1 + d2 - L)), equal to lineIntegralTerm's oriented
// log((s2 + d2) / (s1 + d1)) (d2^2 - d1^2 = s2^2 - s1^2 along the edge's
// line) wherever that is live.  The local-frame FP64 kernels (mixed near
// pairs, the analytic derivatives) use it: it depends only on distances,
// so the rounding of the frame change cannot flip a branch.  Where the
// reference's branch returns 0 although the station lies off the segment
// -- exactly on the edge's line, beyond its end point, which synthetic
// station grids can hit when they share the voxel lattice (s1 + d1 is then
// an exact 0 in the reference's global coordinates) -- this is the
// continuous value log(d1 / d2) instead: the reference's forward is
// discontinuous there and its own finite-difference Jacobian undefined.
// The FP64 forward keeps lambda_from wherever a station may be on an edge's
// line (pair_forward_fp64_branches).  live = the station is not on the segment
// itself (d1 + d2 > L).
__device__ __forceinline__ double lambda_sym(double d1, double d2, double L, bool* live) {
    const double dsum = d1 + d2, den = dsum - L;
    *live = den > 1e-13 * dsum;
    return *live ? log1p(2.0 * L / den) : 0.0;
}

// ------------------------------------------------------------- scatter ----
// LithologyModel::applyParameterVector (lithology_model.cpp:210-248) step 1:
// every global DOF writes the (vertex, axis) slots it controls.
__global__ void k_scatter_dofs(int np, const double* __restrict__ params, const int32_t* __restrict__ dof_off,
                               const int32_t* __restrict__ ref_vertex, const uint8_t* __restrict__ ref_axis,
                               const double* __restrict__ ref_scale, double* __restrict__ pos) {
    int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= np) return;
    double val = params[d];
    for (int r = dof_off[d]; r < dof_off[d + 1]; ++r)
        pos[3 * ref_vertex[r] + ref_axis[r]] = __dmul_rn(val, ref_scale[r]);
}

// Step 2: interpolateFromControlPoints (surface_mesh.cpp:610-623); rows only
// read control-point vertices, which are never rows themselves.
__global__ void k_interpolate(int nrows, const int32_t* __restrict__ rows, const int32_t* __restrict__ interp_off,
                              const int32_t* __restrict__ interp_src, const double* __restrict__ interp_w,
                              double* __restrict__ pos) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nrows) return;
    int v = rows[i];
    double px = 0.0, py = 0.0, pz = 0.0;
    for (int k = interp_off[v]; k < interp_off[v + 1]; ++k) {
        const double* q = pos + 3 * interp_src[k];
        double w = interp_w[k];
        px = __dadd_rn(px, __dmul_rn(q[0], w));
        py = __dadd_rn(py, __dmul_rn(q[1], w));
        pz = __dadd_rn(pz, __dmul_rn(q[2], w));
    }
    pos[3 * v] = px;
    pos[3 * v + 1] = py;
    pos[3 * v + 2] = pz;
}

// Step 3: shared-vertex averaging groups (lithology_model.cpp:235-247).
__global__ void k_sync_shared(int ns, const int32_t* __restrict__ sync_off, const int32_t* __restrict__ sync_vertex,
                              double* __restrict__ pos) {
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= ns) return;
    int b = sync_off[s], e = sync_off[s + 1];
    if (e - b < 2) return;
    double ax = 0.0, ay = 0.0, az = 0.0;
    for (int k = b; k < e; ++k) {
        const double* q = pos + 3 * sync_vertex[k];
        ax = __dadd_rn(ax, q[0]);
        ay = __dadd_rn(ay, q[1]);
        az = __dadd_rn(az, q[2]);
    }
    double n = static_cast<double>(e - b);
    ax = __ddiv_rn(ax, n); ay = __ddiv_rn(ay, n); az = __ddiv_rn(az, n);
    for (int k = b; k < e; ++k) {
        double* q = pos + 3 * sync_vertex[k];
        q[0] = ax; q[1] = ay; q[2] = az;
    }
}

// ------------------------------------------------------- facet constants --
// Exact-order helpers: no FMA contraction, the reference's left-to-right
// evaluation.  Facets collapsed by the control-point interpolation have a
// twice-area of ~1e-12 (above the reference's 1e-15 cutoff), so their unit
// normal is pure rounding; the TMI facet term does not vanish with the area,
// so it is reproduced only when the normal is rounded exactly as on the CPU.
__device__ __forceinline__ d3 sub_rn(d3 a, d3 b) { return {__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y), __dsub_rn(a.z, b.z)}; }
__device__ __forceinline__ double dot_rn(d3 a, d3 b) {
    return __dadd_rn(__dadd_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)), __dmul_rn(a.z, b.z));
}
__device__ __forceinline__ d3 cross_rn(d3 a, d3 b) {
    return {__dsub_rn(__dmul_rn(a.y, b.z), __dmul_rn(a.z, b.y)), __dsub_rn(__dmul_rn(a.z, b.x), __dmul_rn(a.x, b.z)),
            __dsub_rn(__dmul_rn(a.x, b.y), __dmul_rn(a.y, b.x))};
}
__device__ __forceinline__ double norm_rn(d3 a) { return __dsqrt_rn(dot_rn(a, a)); }
__device__ __forceinline__ d3 div_rn(d3 a, double s) { return {__ddiv_rn(a.x, s), __ddiv_rn(a.y, s), __ddiv_rn(a.z, s)}; }

// A facet collapsed onto a line: twice-area below 1e-10 x its longest edge
// squared (control-point interpolation produces them).  Its unit normal is
// rounding noise, and the reference's TMI facet term, which does not vanish
// with the area (magnetic_forward.cpp:312-347), is then a discontinuous
// function of the positions.  The derivative kernels always take such facets
// as contributing zero; the forward does too when the context drops them
// (lf_set_collapsed_facets), so that the objective is the function its
// gradient differentiates.  No reference counterpart.
__device__ __forceinline__ bool facet_collapsed(const d3 (&v)[3], double area2) {
    const double l0 = norm_rn(sub_rn(v[1], v[0])), l1 = norm_rn(sub_rn(v[2], v[1])), l2 = norm_rn(sub_rn(v[0], v[2]));
    const double lm = fmax(l0, fmax(l1, l2));
    return area2 < 1e-10 * lm * lm;
}

// Forward record of one facet (vertices v), its constants in the reference's
// operation order; out[NFC].  drop: collapsed facets contribute nothing.
__device__ __forceinline__ void face_consts_fwd(const d3 (&v)[3], d3 m, d3 fdir, double (&out)[NFC],
                                                bool drop = false) {
    // faceNagyContribution / magneticFacet: n = (b-a) x (c-a), unit_n = n / |n|
    d3 n = cross_rn(sub_rn(v[1], v[0]), sub_rn(v[2], v[0]));
    double area2 = norm_rn(n);
    bool valid = !(area2 < kEps) && !(drop && facet_collapsed(v, area2));
    d3 un = valid ? div_rn(n, area2) : mk3(0, 0, 0);
    out[FC_PAD] = 0.0;
    for (int i = 0; i < 3; ++i) {
        out[FC_AX + 3 * i] = v[i].x; out[FC_AY + 3 * i] = v[i].y; out[FC_AZ + 3 * i] = v[i].z;
    }
    out[FC_AREA2] = valid ? area2 : -1.0;
    out[FC_NX] = un.x; out[FC_NY] = un.y; out[FC_NZ] = un.z;
    out[FC_NZ2] = 2.0 * un.z;
    out[FC_MF2] = 2.0 * __dmul_rn(dot_rn(m, un), dot_rn(fdir, un));  // mn * fn
    for (int i = 0; i < 3; ++i) {
        d3 e = sub_rn(v[(i + 1) % 3], v[i]);
        double L = norm_rn(e);
        d3 eh = (L < kEps) ? mk3(0, 0, 0) : div_rn(e, L);
        d3 perp = cross_rn(un, eh);
        out[FC_L0 + i] = L;
        out[FC_HL0 + i] = 0.5 * (L * L);
        out[FC_P0X + 3 * i] = perp.x; out[FC_P0Y + 3 * i] = perp.y; out[FC_P0Z + 3 * i] = perp.z;
        out[FC_MT0 + i] = 2.0 * __dmul_rn(dot_rn(m, perp), dot_rn(fdir, perp));  // mt * ft
    }
}

// A record to its 16-byte aligned slot.
__device__ __forceinline__ void store_face_fwd(const double (&rec)[NFC], double* __restrict__ slot) {
#pragma unroll
    for (int k = 0; k < NFC / 2; ++k) reinterpret_cast<double2*>(slot)[k] = make_double2(rec[2 * k], rec[2 * k + 1]);
}

__global__ void k_face_prep_fwd(int T, const int32_t* __restrict__ tri, const double* __restrict__ pos,
                                const int16_t* __restrict__ face_group, const GroupConst* __restrict__ groups,
                                d3 fdir, double* __restrict__ fc, int drop_collapsed) {
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= T) return;
    const double* pa = pos + 3 * tri[3 * f];
    const double* pb = pos + 3 * tri[3 * f + 1];
    const double* pc = pos + 3 * tri[3 * f + 2];
    d3 v[3] = {mk3(pa[0], pa[1], pa[2]), mk3(pb[0], pb[1], pb[2]), mk3(pc[0], pc[1], pc[2])};
    double out[NFC];
    const GroupConst& g = groups[face_group[f]];
    face_consts_fwd(v, mk3(g.mdir[0], g.mdir[1], g.mdir[2]), fdir, out, drop_collapsed != 0);
    store_face_fwd(out, fc + (size_t)f * NFC);
}

// Finite-difference-XY gradient mode (no reference counterpart; the
// reference differentiates every axis by per-facet forward differences with
// h = 1e-4 m, faceNagyWithGradient gravity_forward.cpp:48-85): forward
// constants of each listed facet and of its six copies with one vertex moved
// by +h in x or y, variant k = 1 + 2 * corner + axis.  Layout [nf][7][NFC]
// over the list index.
__global__ void k_face_prep_fdxy(int nf, const int32_t* __restrict__ facets, const int32_t* __restrict__ tri,
                                 const double* __restrict__ pos, const int16_t* __restrict__ face_group,
                                 const GroupConst* __restrict__ groups, d3 fdir, double h, double* __restrict__ fcfd) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = blockIdx.y;  // variant
    if (i >= nf) return;
    const int f = facets[i];
    d3 v[3];
    for (int c = 0; c < 3; ++c) {
        const double* p = pos + 3 * tri[3 * f + c];
        v[c] = mk3(p[0], p[1], p[2]);
    }
    if (k > 0) {
        const int c = (k - 1) >> 1;
        if ((k - 1) & 1) v[c].y = __dadd_rn(v[c].y, h);
        else v[c].x = __dadd_rn(v[c].x, h);
    }
    double out[NFC];
    const GroupConst& g = groups[face_group[f]];
    face_consts_fwd(v, mk3(g.mdir[0], g.mdir[1], g.mdir[2]), fdir, out);
    store_face_fwd(out, fcfd + ((size_t)i * 7 + k) * NFC);
}

// FP32 adjoints of the far-field gradient: adjoint x group scale, rounded once
// per (group, station) instead of once per pair.  Layout [groups][ng] gravity,
// then [groups][nm] magnetic (groups = 1 with every station scaled by its own
// body's group when sta_group is given); ng = nm = 0: none wanted.
struct FarAdjoints {
    int groups, ng, nm;
    const int32_t* sta_group;
    const double *gcoef, *mcoef;
    float* out;
    __host__ __device__ long long count() const { return (long long)groups * (ng + nm); }
};

__device__ __forceinline__ void far_adjoint(const FarAdjoints& a, long long i, const GroupConst* __restrict__ groups) {
    if (i >= a.count()) return;
    const long long gravity = (long long)a.groups * a.ng;
    const bool grav = i < gravity;
    const long long k = grav ? i : i - gravity;
    const int n = grav ? a.ng : a.nm, s = (int)(k % n), g = a.sta_group ? a.sta_group[s] : (int)(k / n);
    // the scales of GC_GS and GC_MS
    a.out[i] = grav ? (float)(a.gcoef[s] * groups[g].gscale_jac)
                    : (float)(a.mcoef[s] * (groups[g].mag_active ? -groups[g].mscale : 0.0));
}

// Gradient constants of every facet (blocks 0 .. T / 128), and the far-field
// kernel's adjoints in the blocks after them: as a kernel of their own they
// cost small evaluations a launch (mixed gradient of a 320-facet body under 144
// stations 113 us, 108 without).
constexpr int kGradPrepThreads = 128;
__global__ void __launch_bounds__(kGradPrepThreads)
    k_face_prep_grad(int T, const int32_t* __restrict__ tri, const double* __restrict__ pos,
                     const int16_t* __restrict__ face_group, const GroupConst* __restrict__ groups,
                     const uint8_t* __restrict__ face_needs, int want_grav, int want_mag, d3 fdir,
                     double* __restrict__ gc, FarAdjoints far) {
    const int face_blocks = (T + kGradPrepThreads - 1) / kGradPrepThreads;
    if ((int)blockIdx.x >= face_blocks) {
        far_adjoint(far, (long long)(blockIdx.x - face_blocks) * kGradPrepThreads + threadIdx.x, groups);
        return;
    }
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= T) return;
    const double* pa = pos + 3 * tri[3 * f];
    const double* pb = pos + 3 * tri[3 * f + 1];
    const double* pc = pos + 3 * tri[3 * f + 2];
    d3 a = mk3(pa[0], pa[1], pa[2]), b = mk3(pb[0], pb[1], pb[2]), c = mk3(pc[0], pc[1], pc[2]);
    d3 n = cross3(b - a, c - a);
    double area2 = norm3(n);
    double L0 = norm3(b - a), L1 = norm3(c - b), L2 = norm3(a - c);
    // Facets collapsed onto a line (twice-area below 1e-10 of the longest edge
    // squared, e.g. by control-point interpolation) carry a kink in their
    // facet term: its central difference is zero and so is their derivative
    // contribution here.
    double Lmax = fmax(L0, fmax(L1, L2));
    bool valid = !(area2 < kEps) && !(L0 < kEps) && !(L1 < kEps) && !(L2 < kEps) && !(area2 < 1e-10 * Lmax * Lmax);
    double out[NGC];
    for (int k = 0; k < NGC; ++k) out[k] = 0.0;
    if (valid) {
        d3 zh = n * (1.0 / area2);
        d3 xh = (b - a) * (1.0 / L0);
        d3 yh = cross3(zh, xh);
        d3 ca = c - a;
        double cx = dot3(ca, xh), cy = dot3(ca, yh);
        const GroupConst& g = groups[face_group[f]];
        d3 m = mk3(g.mdir[0], g.mdir[1], g.mdir[2]);
        out[GC_AX] = a.x; out[GC_AY] = a.y; out[GC_AZ] = a.z;
        out[GC_XX] = xh.x; out[GC_XY] = xh.y; out[GC_XZ] = xh.z;
        out[GC_YX] = yh.x; out[GC_YY] = yh.y; out[GC_YZ] = yh.z;
        out[GC_ZX] = zh.x; out[GC_ZY] = zh.y; out[GC_ZZ] = zh.z;
        out[GC_L0] = L0; out[GC_CX] = cx; out[GC_CY] = cy;
        out[GC_E1X] = (cx - L0) / L1; out[GC_E1Y] = cy / L1; out[GC_L1] = L1;
        out[GC_E2X] = -cx / L2; out[GC_E2Y] = -cy / L2; out[GC_L2] = L2;
        out[GC_GS] = want_grav ? g.gscale_jac : 0.0;
        out[GC_MS] = (want_mag && g.mag_active) ? -g.mscale : 0.0;
        // magnetic direction products in the local frame
        d3 ml = mk3(dot3(m, xh), dot3(m, yh), dot3(m, zh));
        d3 fl = mk3(dot3(fdir, xh), dot3(fdir, yh), dot3(fdir, zh));
        out[GC_MF] = ml.z * fl.z;
        double ex[3] = {1.0, out[GC_E1X], out[GC_E2X]}, ey[3] = {0.0, out[GC_E1Y], out[GC_E2Y]};
        for (int i = 0; i < 3; ++i) {
            // in-plane edge normal perp = z x e = (-ey, ex, 0)
            double mp = -ml.x * ey[i] + ml.y * ex[i], fp = -fl.x * ey[i] + fl.y * ex[i];
            out[GC_MT0 + i] = mp * fp;
        }
        out[GC_FLAGS] = 1.0 + (face_needs[f] ? 2.0 : 0.0);
    }
    for (int k = 0; k < NGC; ++k) gc[(size_t)k * T + f] = out[k];
}

// ------------------------------------------------------------- forward ----
// FP64 square root, reciprocal and reciprocal square root for positive normal
// arguments: the hardware's approximations (relative error below 2^-19.9,
// measured over 2^-40..2^40) refined by one third-order step -- Halley's for
// x^(-1/2), y (1 + e/2 + 3 e^2/8) with e = 1 - x y^2; for 1/x, y (1 + e + e^2)
// with e = 1 - x y.  The remaining error is rounding: at most 1 ulp for the
// square root and the reciprocal, 2^-51.7 for the reciprocal square root.  The
// pair kernels evaluate seven of them per pair; the library forms cost 2-4
// times the instructions and a special-case branch each.
__device__ __forceinline__ double sqrt_pos64(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double t = x * y, e = fma(-t, y, 1.0);
    return fma(t * e, fma(0.375, e, 0.5), t);
}
__device__ __forceinline__ double rcp_pos64(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// Square root of x > 0 and its reciprocal from one approximation.
__device__ __forceinline__ double sqrt_inv64(double x, double* inv) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double t = x * y, e = fma(-t, y, 1.0), ep = e * fma(0.375, e, 0.5);
    *inv = fma(y, ep, y);
    return fma(t, ep, t);
}

// atanh(v) for 0 <= v <= 1/2 (atanh_poly64), for v <= 1/4 (atanh_short64), and
// atan(t) for t^2 <= 0.1: polynomials in the square, Chebyshev interpolants of
// atanh(sqrt w) / sqrt w on [0, 1/4] and [0, 1/16] and of atan(sqrt w) /
// sqrt w on [0, 0.1] (60-digit arithmetic; relative errors of the coefficients
// as rounded below 1.9e-16, 1.7e-17 and 1.2e-17 before the evaluation's own
// rounding).
__device__ __forceinline__ double atanh_poly64(double v) {
    const double w = v * v;
    double p = fma(0.2113466728500407, w, -0.11607286571460644);
    p = fma(p, w, 0.12342317349394255);
    p = fma(p, w, 0.030552784701105364);
    p = fma(p, w, 0.06305373925151087);
    p = fma(p, w, 0.06611875378546901);
    p = fma(p, w, 0.07697116199755842);
    p = fma(p, w, 0.09090628331896689);
    p = fma(p, w, 0.11111121577224739);
    p = fma(p, w, 0.14285714054503637);
    p = fma(p, w, 0.20000000002644475);
    p = fma(p, w, 0.33333333333321485);
    return fma(p * w, v, v);
}
__device__ __forceinline__ double atanh_short64(double v) {
    const double w = v * v;
    double p = fma(0.07610224602501783, w, 0.06454071625136103);
    p = fma(p, w, 0.07706064964345138);
    p = fma(p, w, 0.09090395415324985);
    p = fma(p, w, 0.11111122319976208);
    p = fma(p, w, 0.14285714148744663);
    p = fma(p, w, 0.20000000000836662);
    p = fma(p, w, 0.33333333333331366);
    return fma(p * w, v, v);
}
__device__ __forceinline__ double atan_poly64(double t) {
    const double w = t * t;
    double p = fma(-0.03400559203053808, w, 0.055195446424522086);
    p = fma(p, w, -0.0662578202739514);
    p = fma(p, w, 0.0768947276046168);
    p = fma(p, w, -0.0909078630887742);
    p = fma(p, w, 0.11111107856392849);
    p = fma(p, w, -0.1428571423598591);
    p = fma(p, w, 0.19999999999613183);
    p = fma(p, w, -0.33333333333332166);
    return fma(p * w, t, t);
}

// The largest of three edge ratios v = L / (d1 + d2) by their high words.  As
// unsigned numbers the high words of positive doubles keep their order, and a
// NaN of either sign (a station on a vertex: its distance is 0 x inf) exceeds
// every finite value.
__device__ __forceinline__ unsigned max_ratio_hi(double v0, double v1, double v2) {
    return max((unsigned)__double2hiint(v0), max((unsigned)__double2hiint(v1), (unsigned)__double2hiint(v2)));
}

// One pair (station o, facet record F) with every branch of the reference
// (solidAngle, lineIntegralTerm) and the library functions: the gz facet
// factor and the TMI facet factor.  Up to the logarithms and the arctangent
// every operation is rounded as the reference's, so that a station on a
// facet's edge or in its plane takes the branch it takes there.
template <bool GZ, bool TMI>
__device__ __noinline__ double2 pair_forward_fp64_branches(const double* __restrict__ F, d3 o) {
    d3 p[3], r[3];
    double l[3];
    for (int i = 0; i < 3; ++i) {
        p[i] = mk3(F[FC_AX + 3 * i], F[FC_AY + 3 * i], F[FC_AZ + 3 * i]);
        r[i] = sub_rn(p[i], o);
        l[i] = norm_rn(r[i]);
    }
    double omega = 0.0;
    if (!(l[0] < kEps || l[1] < kEps || l[2] < kEps)) {
        const double num = dot_rn(r[0], cross_rn(r[1], r[2]));
        double den = __dmul_rn(__dmul_rn(l[0], l[1]), l[2]);
        den = __dadd_rn(den, __dmul_rn(dot_rn(r[0], r[1]), l[2]));
        den = __dadd_rn(den, __dmul_rn(dot_rn(r[0], r[2]), l[1]));
        den = __dadd_rn(den, __dmul_rn(dot_rn(r[1], r[2]), l[0]));
        omega = 2.0 * atan2(num, den);
    }
    const d3 un = mk3(F[FC_NX], F[FC_NY], F[FC_NZ]);
    const double h = dot_rn(r[0], un);
    double dsum = 0.0, tsum = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int j = (i + 1) % 3;
        const double L = F[FC_L0 + i];
        if (L < kEps) continue;
        const d3 e = sub_rn(p[j], p[i]);
        bool live;
        const double lam =
            lambda_from(__ddiv_rn(dot_rn(r[i], e), L), __ddiv_rn(dot_rn(r[j], e), L), l[i], l[j], &live);
        if (GZ) dsum -= dot_rn(r[i], mk3(F[FC_P0X + 3 * i], F[FC_P0Y + 3 * i], F[FC_P0Z + 3 * i])) * lam;
        if (TMI) tsum += 0.5 * F[FC_MT0 + i] * lam;
    }
    return make_double2(GZ ? un.z * (dsum - h * omega) : 0.0, TMI ? 0.5 * F[FC_MF2] * omega + tsum : 0.0);
}

// The same pair away from the facet, which is nearly every pair: Lambda in
// the symmetric form 2 atanh(v), v = L / (d1 + d2), the solid angle's
// numerator as height x twice-area, its dot products from the distances, and
// the polynomials above.  Taken when every v is below 1/2 (each edge is then
// seen under at most 60 degrees, so the solid angle's denominator is at least
// 2.5 la lb lc and its tangent at most 0.283) and the station lies further
// than 2^-20 la from the facet's plane (so it is on no edge's line, where the
// reference's lineIntegralTerm is 0); every other pair, zero distances and
// NaN among them (max_ratio_hi), takes the branches above.  Both tests compare
// the high words of doubles.
// Bound by the FP64 pipe (73 % busy): 130 FP64 instructions of 227 per pair,
// against more than 500 through the library functions.  Its error against 64-bit sums in
// the symmetric form fell with the cancellation in s + d: 1.7e-13 to 2e-15 on
// a 320-facet body, 1.6e-13 to 3e-15 on a contact model's unit responses.
// The shorter atanh polynomial for v < 1/4 is worth 4 % (304 against 316 us).
template <bool GZ, bool TMI>
__device__ __forceinline__ void pair_forward_fp64(const double* __restrict__ F, d3 o, double* gz, double* tmi) {
    const double2* __restrict__ q = reinterpret_cast<const double2*>(F);
    const double2 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q4 = q[4];
    // contributes nothing (the same for every lane): -1 itself, since the area of
    // a facet that overflows is a NaN with a sign bit and has to reach the sums
    if (__double2hiint(q4.y) == (int)0xbff00000) return;
    const d3 ra = mk3(q0.x - o.x, q0.y - o.y, q1.x - o.z), rb = mk3(q1.y - o.x, q2.x - o.y, q2.y - o.z),
             rc = mk3(q3.x - o.x, q3.y - o.y, q4.x - o.z);
    const double a2 = dot3(ra, ra), b2 = dot3(rb, rb), c2 = dot3(rc, rc);
    const double la = sqrt_pos64(a2), lb = sqrt_pos64(b2), lc = sqrt_pos64(c2);
    const double2 q5 = q[5], q6 = q[6], q7 = q[7], q8 = q[8], q9 = q[9];
    const double h = ra.x * q5.x + ra.y * q5.y + ra.z * q6.x;
    const double v0 = q7.x * rcp_pos64(la + lb), v1 = q7.y * rcp_pos64(lb + lc), v2 = q8.x * rcp_pos64(lc + la);
    const unsigned vmax = max_ratio_hi(v0, v1, v2);
    if (!(vmax < 0x3fe00000u && (__double2hiint(h) & 0x7fffffff) + (20 << 20) > __double2hiint(la))) {
        const double2 r = pair_forward_fp64_branches<GZ, TMI>(F, o);
        if (GZ) *gz += r.x;
        if (TMI) *tmi += r.y;
        return;
    }
    // ra . rb = (a2 + b2) / 2 - L^2 / 2
    const double dab = fma(0.5, a2 + b2, -q8.y), dbc = fma(0.5, b2 + c2, -q9.x), dac = fma(0.5, c2 + a2, -q9.y);
    const double den = fma(la * lb, lc, fma(dab, lc, fma(dac, lb, dbc * la)));
    const double om = atan_poly64(h * q4.y * rcp_pos64(den));
    double l0, l1, l2;
    if (vmax < 0x3fd00000u) {  // every v < 1/4
        l0 = atanh_short64(v0);
        l1 = atanh_short64(v1);
        l2 = atanh_short64(v2);
    } else {
        l0 = atanh_poly64(v0);
        l1 = atanh_poly64(v1);
        l2 = atanh_poly64(v2);
    }
    const double2 q14 = q[14];
    if (GZ) {
        const double2 p0 = q[10], p1 = q[11], p2 = q[12], p3 = q[13];
        const double d0 = ra.x * p0.x + ra.y * p0.y + ra.z * p1.x, d1 = rb.x * p1.y + rb.y * p2.x + rb.z * p2.y,
                     d2 = rc.x * p3.x + rc.y * p3.y + rc.z * q14.x;
        *gz -= q6.y * fma(h, om, fma(d0, l0, fma(d1, l1, d2 * l2)));
    }
    if (TMI) {
        const double2 m = q[15];
        *tmi += fma(q14.y, om, fma(m.x, l0, fma(m.y, l1, F[FC_MT2] * l2)));
    }
}

// Grid: x = station blocks, y = facet chunks (each inside one group).  Writes
// the chunk's unscaled facet sums per station.
// One CTA's work: station s (act = s is a station of the block) against
// facets [fb, fe); out_gz[s] / out_tmi[s] receive the unscaled sums.
// SLICES = 1: one station per thread of the CTA, every thread against every
// facet.  SLICES = 4: the CTA's four warps hold the same 32 stations and take
// every fourth facet each; their sums are added in warp order through shared
// memory.  The second form gives a small launch four times the CTAs for the
// same number of chunk partials.
template <bool GZ, bool TMI, int FT, int SLICES = 1>
__device__ __forceinline__ void forward_fp64_block(double* __restrict__ sm, int s, bool act,
                                                   const double* __restrict__ sta, const double* __restrict__ fc,
                                                   int fb, int fe, double* __restrict__ out_gz,
                                                   double* __restrict__ out_tmi) {
    d3 o = mk3(0, 0, 0);
    if (act) o = mk3(sta[3 * s], sta[3 * s + 1], sta[3 * s + 2]);
    double gz = 0.0, tmi = 0.0;
    for (int f0 = fb; f0 < fe; f0 += FT) {
        int nf = min(FT, fe - f0);
        __syncthreads();
        const double2* __restrict__ src = reinterpret_cast<const double2*>(fc + (size_t)f0 * NFC);
        for (int idx = threadIdx.x; idx < nf * (NFC / 2); idx += blockDim.x)
            reinterpret_cast<double2*>(sm)[idx] = __ldg(src + idx);
        __syncthreads();
        if (act)
            for (int j = SLICES == 1 ? 0 : (int)(threadIdx.x >> 5); j < nf; j += SLICES)
                pair_forward_fp64<GZ, TMI>(sm + j * NFC, o, &gz, &tmi);
    }
    if (SLICES > 1) {
        __syncthreads();  // the records are no longer read
        sm[threadIdx.x] = gz;
        sm[blockDim.x + threadIdx.x] = tmi;
        __syncthreads();
        if (threadIdx.x >= 32) return;
#pragma unroll
        for (int k = 1; k < SLICES; ++k) {
            gz += sm[32 * k + threadIdx.x];
            tmi += sm[blockDim.x + 32 * k + threadIdx.x];
        }
    }
    if (act) {
        if (GZ) out_gz[s] = gz;
        if (TMI) out_tmi[s] = tmi;
    }
}

// 29.4 M pairs (9,904 facets, 2,964 stations, gz and TMI): 993 us with the
// library functions and SoA records in shared memory, 291 us now, 1.0e11
// pairs/s.  Five CTAs per SM: six or seven (84, 72 registers) are 3 and 6 %
// slower, the unbounded 96 registers 2 %.
template <bool GZ, bool TMI, int FT, int SLICES>
__global__ void __launch_bounds__(128, 5) k_forward_fp64(int S, const double* __restrict__ sta,
                                                         const double* __restrict__ fc,
                                                         const int32_t* __restrict__ chunk_begin,
                                                         const int32_t* __restrict__ chunk_end,
                                                         double* __restrict__ part_gz, double* __restrict__ part_tmi) {
    __shared__ __align__(16) double sm[NFC * FT];
    static_assert(NFC * FT >= 2 * 128, "the slices' sums fit where the records were");
    const int s = SLICES == 1 ? (int)(blockIdx.x * blockDim.x + threadIdx.x)
                              : (int)(blockIdx.x * 32 + (threadIdx.x & 31));
    const int chunk = blockIdx.y;
    forward_fp64_block<GZ, TMI, FT, SLICES>(sm, s, s < S, sta, fc, chunk_begin[chunk], chunk_end[chunk],
                                            GZ ? part_gz + (size_t)chunk * S : nullptr,
                                            TMI ? part_tmi + (size_t)chunk * S : nullptr);
}

// Batched bodies: a persistent grid walks a list of (station block, facet
// range) items -- one body's stations against one chunk of that body's
// facets -- in the order given (largest first).  Item out: offset added to
// the global station index to address the item's partial slot.
struct FwdItem {
    int32_t s0, s_end, fb, fe;
    int64_t out;
};

template <bool GZ, bool TMI, int FT>
__global__ void __launch_bounds__(128, 5) k_forward_fp64_items(const FwdItem* __restrict__ items, int nitems,
                                                            const double* __restrict__ sta,
                                                            const double* __restrict__ fc,
                                                            double* __restrict__ part_gz, double* __restrict__ part_tmi) {
    __shared__ __align__(16) double sm[NFC * FT];
    for (int it = blockIdx.x; it < nitems; it += gridDim.x) {
        const FwdItem w = items[it];
        const int s = w.s0 + (int)threadIdx.x;
        forward_fp64_block<GZ, TMI, FT>(sm, s, s < w.s_end, sta, fc, w.fb, w.fe,
                                        GZ ? part_gz + w.out : nullptr, TMI ? part_tmi + w.out : nullptr);
    }
}

// acc + v(c0) + v(c0 + 8) + ... (c < n), added in that order with eight
// loads in flight: the chunk reductions below are bound by the latency of
// their partial loads, not by the additions.
template <class F>
__device__ __forceinline__ double strided_sum8(int c0, int n, double acc, F v) {
    int c = c0;
    for (; c + 56 < n; c += 64) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = v(c + 8 * u);
#pragma unroll
        for (int u = 0; u < 8; ++u) acc += x[u];
    }
    for (; c < n; c += 8) acc += v(c);
    return acc;
}

// Per station of a batch of bodies: sum of its body's chunk partials
// (grp_part_off[g] + c * n_g + local index, c < grp_nch[g]), times the body's
// group scales when `groups` is given (FP64 path; the mixed partials carry
// their scales).  Lane sums over chunks as in k_forward_reduce.
__global__ void __launch_bounds__(256) k_forward_reduce_groups(int S, const int32_t* __restrict__ sta_group,
                                                               const int32_t* __restrict__ grp_sta_off,
                                                               const int64_t* __restrict__ grp_part_off,
                                                               const int32_t* __restrict__ grp_nch,
                                                               const GroupConst* __restrict__ groups,
                                                               const double* __restrict__ part_gz,
                                                               const double* __restrict__ part_tmi,
                                                               double* __restrict__ gz, double* __restrict__ tmi) {
    __shared__ double sg[8][33], st[8][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int s = blockIdx.x * 32 + tx;
    double g = 0.0, t = 0.0;
    int grp = 0;
    if (s < S) {
        grp = sta_group[s];
        const int n = grp_sta_off[grp + 1] - grp_sta_off[grp], loc = s - grp_sta_off[grp];
        const int64_t base = grp_part_off[grp] + loc;
        const int nch = grp_nch[grp];
        if (part_gz) g = strided_sum8(ty, nch, g, [&](int c) { return part_gz[base + (int64_t)c * n]; });
        if (part_tmi) t = strided_sum8(ty, nch, t, [&](int c) { return part_tmi[base + (int64_t)c * n]; });
    }
    sg[ty][tx] = g;
    st[ty][tx] = t;
    __syncthreads();
    if (ty == 0 && s < S) {
        double G = 0.0, Tm = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            G += sg[k][tx];
            Tm += st[k][tx];
        }
        if (groups) {
            G = G * groups[grp].gscale_fwd;
            Tm = -groups[grp].mscale * Tm;
        }
        if (gz) gz[s] = G;
        if (tmi) tmi[s] = Tm;
    }
}

// Per body (group) of a batch: data misfit of its stations, gravity + alpha
// x magnetic, from the residual definition of k_residual.
__global__ void k_group_misfit(int G, const int32_t* __restrict__ grp_sta_off, const double* __restrict__ gpred,
                               const double* __restrict__ gobs, const double* __restrict__ gw,
                               const double* __restrict__ mpred, const double* __restrict__ mobs,
                               const double* __restrict__ mw, double alpha, double* __restrict__ out) {
    __shared__ double red[256];
    const int g = blockIdx.x;
    if (g >= G) return;
    double acc = 0.0;
    for (int s = grp_sta_off[g] + threadIdx.x; s < grp_sta_off[g + 1]; s += blockDim.x) {
        if (gpred) {
            const double r = gw[s] * (gobs[s] - gpred[s]);
            acc += 0.5 * r * r;
        }
        if (mpred) {
            const double r = mw[s] * (mobs[s] - mpred[s]);
            acc += alpha * (0.5 * r * r);
        }
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int k = blockDim.x / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[g] = red[0];
}

// Sums chunk partials with the group scales applied chunk by chunk (a chunk
// lies in one group): gz = sum_c G*rho_g(c)*1e3*1e5 * part (gravityClosedMesh
// :162-178), tmi = sum_c -(amp_g(c)*100/(4 pi)) * part
// (magneticClosedMeshVector :367-386).  Blocks of 32 stations x 8 chunk
// lanes, lane sums added in lane order.
__global__ void __launch_bounds__(256) k_forward_reduce(int S, int nchunks, const int32_t* __restrict__ chunk_group,
                                                        const GroupConst* __restrict__ groups,
                                                        const double* __restrict__ part_gz,
                                                        const double* __restrict__ part_tmi, double* __restrict__ gz,
                                                        double* __restrict__ tmi) {
    __shared__ double sg[8][33], st[8][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int s = blockIdx.x * 32 + tx;
    double g = 0.0, t = 0.0;
    if (s < S) {
        if (part_gz)
            g = strided_sum8(ty, nchunks, g, [&](int c) {
                return part_gz[(size_t)c * S + s] * groups[chunk_group[c]].gscale_fwd;
            });
        if (part_tmi)
            t = strided_sum8(ty, nchunks, t, [&](int c) {
                return -groups[chunk_group[c]].mscale * part_tmi[(size_t)c * S + s];
            });
    }
    sg[ty][tx] = g;
    st[ty][tx] = t;
    __syncthreads();
    if (ty == 0 && s < S) {
        double G = 0.0, Tm = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            G += sg[k][tx];
            Tm += st[k][tx];
        }
        if (gz) gz[s] = G;
        if (tmi) tmi[s] = Tm;
    }
}

// ----------------------------------------------------------- residuals ----
// ObjectiveFunction misfit (objective.cpp:22-31, 83-105): w = 1/std or 1;
// adjoint c = -alpha * w^2 * (obs - pred); per-block partial misfit sums.
__global__ void k_residual(int S, const double* __restrict__ pred, const double* __restrict__ obs,
                           const double* __restrict__ w, double alpha, double* __restrict__ coef,
                           double* __restrict__ block_misfit) {
    __shared__ double red[256];
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    double mis = 0.0;
    if (s < S) {
        double ws = w[s];
        double r = obs[s] - pred[s];
        double res = ws * r;
        mis = 0.5 * res * res;
        if (coef) coef[s] = -alpha * (ws * ws * r);
    }
    red[threadIdx.x] = mis;
    __syncthreads();
    for (int k = blockDim.x / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) block_misfit[blockIdx.x] = red[0];
}

// ------------------------------------------------------------ gradient ----
struct StationTile {
    // per station: x, y, z, gravity adjoint, magnetic adjoint
    double v[5];
};

// Per-facet accumulators over stations (local frame).
struct GradAcc {
    d3 va, vb, vc;      // vertex-direct terms
    double alam[3];     // sum Gs * Lambda_i       (d_perp direct on p1)
    double aom;         // sum Gs * Omega          (h direct on a)
    double ai;          // sum G0 * I              (n_z factor)
    d3 bh;              // sum Gs * Omega * r_a    (h through n_hat; z is not needed)
    d3 bl[3];           // sum Gs * Lambda_i * r1  (d_perp through perp_i; bl[0].y is not needed)
    double amf;         // sum Ts * Omega          (MF)
    double amt[3];      // sum Ts * Lambda_i       (MT_i)
};

// Per-facet finalisation in the local frame: differentiates the facet
// constants (n_z, the unit normal, the in-plane edge normals, the magnetic
// direction products, the edge directions) once, from the station sums, and
// returns d(contracted facet terms)/d(a, b, c) in the global frame.
__device__ inline void grad_finalize(const double* C, const GradAcc& A, const GroupConst& g, d3 fdir, double outv[9]) {
    const double L0 = C[GC_L0], cx = C[GC_CX], cy = C[GC_CY];
    const double area2 = L0 * cy;
    d3 xh = mk3(C[GC_XX], C[GC_XY], C[GC_XZ]), yh = mk3(C[GC_YX], C[GC_YY], C[GC_YZ]),
       zh = mk3(C[GC_ZX], C[GC_ZY], C[GC_ZZ]);
    d3 mg = mk3(g.mdir[0], g.mdir[1], g.mdir[2]);
    d3 ml = mk3(dot3(mg, xh), dot3(mg, yh), dot3(mg, zh));
    d3 fl = mk3(dot3(fdir, xh), dot3(fdir, yh), dot3(fdir, zh));
    d3 nh = mk3(0, 0, 1);
    d3 eh[3] = {mk3(1, 0, 0), mk3(C[GC_E1X], C[GC_E1Y], 0), mk3(C[GC_E2X], C[GC_E2Y], 0)};
    double Ls[3] = {L0, C[GC_L1], C[GC_L2]};
    d3 vbar[3] = {A.va, A.vb, A.vc};
    // n_hat adjoint
    d3 nbar = A.bh * -1.0;
    {
        double mn = ml.z, fn = fl.z;
        nbar = nbar + (ml * fn + fl * mn) * A.amf;
        // n_z = n_hat . e_z(global); e_z in local coordinates
        nbar = nbar + mk3(xh.z, yh.z, zh.z) * A.ai;
    }
    // vertex-direct: h on a, d_perp on p1
    vbar[0] = vbar[0] + nh * (-A.aom);
    for (int i = 0; i < 3; ++i) {
        d3 perp = cross3(nh, eh[i]);
        vbar[i] = vbar[i] + perp * (-A.alam[i]);
        double mp = dot3(ml, perp), fp = dot3(fl, perp);
        d3 pbar = A.bl[i] * -1.0 + (ml * fp + fl * mp) * A.amt[i];
        // perp = n x e: n_bar += e x pbar, e_bar = pbar x n
        nbar = nbar + cross3(eh[i], pbar);
        d3 ebar = cross3(pbar, nh);
        double pe = dot3(ebar, eh[i]);
        d3 eraw = (ebar - eh[i] * pe) * (1.0 / Ls[i]);
        vbar[(i + 1) % 3] = vbar[(i + 1) % 3] + eraw;
        vbar[i] = vbar[i] - eraw;
    }
    // n_hat = n / |n|, n = (b-a) x (c-a)
    double pn = dot3(nbar, nh);
    d3 nraw = (nbar - nh * pn) * (1.0 / area2);
    d3 u = mk3(L0, 0, 0), w = mk3(cx, cy, 0);
    d3 ubar = cross3(w, nraw), wbar = cross3(nraw, u);
    vbar[1] = vbar[1] + ubar;
    vbar[2] = vbar[2] + wbar;
    vbar[0] = vbar[0] - ubar - wbar;
    for (int v = 0; v < 3; ++v) {
        d3 gv = xh * vbar[v].x + yh * vbar[v].y + zh * vbar[v].z;
        outv[3 * v] = gv.x; outv[3 * v + 1] = gv.y; outv[3 * v + 2] = gv.z;
    }
}

__device__ __forceinline__ void grad_acc_zero(GradAcc& A) {
    A.va = A.vb = A.vc = mk3(0, 0, 0);
    A.bh = mk3(0, 0, 0);
    for (int i = 0; i < 3; ++i) { A.alam[i] = 0; A.bl[i] = mk3(0, 0, 0); A.amt[i] = 0; }
    A.aom = A.ai = A.amf = 0.0;
}

// Station tiles: kStationTile consecutive stations (Morton order on the
// device), bounding boxes precomputed per station set (tile_box[t][6]:
// min xyz, max xyz).
constexpr int kStationTile = 64;

// Near/far split of the mixed-precision gradient: a facet is far from a
// station tile when its centroid lies at least tau x its longest edge from
// the tile's bounding box.  Every operation is rounded explicitly, so the
// near-field and far-field kernels, compiled separately, classify every
// (facet, tile) identically and each pair is counted exactly once.
// FarKey: the facet's centroid and squared threshold; th2 < 0 means
// "everything near" (tau >= 1e30, the FP64 mode).
struct FarKey {
    double c0, c1, c2, th2;
};

__device__ __forceinline__ FarKey facet_far_key(const double* C, double tau) {
    FarKey k;
    const double L0 = C[GC_L0], cx = C[GC_CX], cy = C[GC_CY];
    const double px = __ddiv_rn(__dadd_rn(L0, cx), 3.0), py = __ddiv_rn(cy, 3.0);
    k.c0 = __dadd_rn(C[GC_AX], __dadd_rn(__dmul_rn(px, C[GC_XX]), __dmul_rn(py, C[GC_YX])));
    k.c1 = __dadd_rn(C[GC_AY], __dadd_rn(__dmul_rn(px, C[GC_XY]), __dmul_rn(py, C[GC_YY])));
    k.c2 = __dadd_rn(C[GC_AZ], __dadd_rn(__dmul_rn(px, C[GC_XZ]), __dmul_rn(py, C[GC_YZ])));
    const double th = __dmul_rn(tau, fmax(L0, fmax(C[GC_L1], C[GC_L2])));
    k.th2 = tau >= 1e30 ? -1.0 : __dmul_rn(th, th);
    return k;
}

__device__ __forceinline__ bool tile_far(const FarKey& k, const double* __restrict__ bbox) {
    if (k.th2 < 0.0) return false;
    const double d0 = fmax(0.0, fmax(__dadd_rn(bbox[0], -k.c0), __dadd_rn(k.c0, -bbox[3])));
    const double d1 = fmax(0.0, fmax(__dadd_rn(bbox[1], -k.c1), __dadd_rn(k.c1, -bbox[4])));
    const double d2 = fmax(0.0, fmax(__dadd_rn(bbox[2], -k.c2), __dadd_rn(k.c2, -bbox[5])));
    const double dd = __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2));
    return dd >= k.th2;
}

// Omega, the edge integrals, W_i = L_i / (d1 d2 + r1.r2) and which edges are
// live (bit i) for a pair close to its facet, by the library functions; dead:
// the station lies on a vertex, where nothing is differentiable.
struct NearTerms {
    double om, lam[3], W[3];
    int live;
    bool dead;
};
__device__ __forceinline__ NearTerms gradient_near_terms(double x, double y, double z, double L0, double cx, double cy,
                                                      double L1, double L2) {
    NearTerms N;
    const d3 r[3] = {mk3(-x, -y, -z), mk3(L0 - x, -y, -z), mk3(cx - x, cy - y, -z)};
    double l[3];
    N.dead = false;
    N.live = 0;
    for (int i = 0; i < 3; ++i) {
        l[i] = sqrt(dot3(r[i], r[i]));
        N.dead |= l[i] < kEps;
    }
    const double L[3] = {L0, L1, L2};
    double den = l[0] * l[1] * l[2];
    for (int i = 0; i < 3; ++i) {
        const int j = (i + 1) % 3;
        const double dot = dot3(r[i], r[j]), dw = l[i] * l[j] + dot;
        bool lv;
        N.lam[i] = lambda_sym(l[i], l[j], L[i], &lv);
        N.live |= lv ? 1 << i : 0;
        N.W[i] = dw > 1e-300 ? L[i] / dw : 0.0;
        den += dot * l[(i + 2) % 3];
    }
    N.om = 2.0 * atan2(-z * (L0 * cy), den);
    return N;
}

// One (facet, station) pair of the FP64 gradient: adds the station's terms,
// weighted by its adjoints (gco gravity, mco magnetic), to the facet's
// local-frame accumulators.  gsn / ms: the facet group's gz / TMI scales.
// GZ / TMI: which adjoints can be non-zero.
//
// Per edge with direction e, in-plane normal n = (-ey, ex), kl = Gs d_perp +
// Ts MT and kom = -Gs h + Ts MF, the vertex terms are
//   p1 += (-kl e + alpha n + beta z) / d1,  p2 += (kl e + alpha n + beta z) / d2,
//   alpha = W (kom z + kl d_perp),  beta = W (kl z - kom d_perp),
// (q = r1 - (r1.e) e = -d_perp n - z zhat and e x r1 = z n - d_perp zhat in
// the facet's frame), so the terms of a vertex's two edges are added before
// the division by its distance.  Away from the facet (every v = L / (d1 + d2)
// below 1/2, see pair_forward_fp64) W = 2 L / ((d1 + d2)^2 - L^2) and the
// polynomials replace the library's log1p and atan2; other pairs take
// gradient_near_terms.  About 230 FP64 instructions per pair against more than
// 700 through the library functions.  Gravity Jacobian of a 1,280-facet body
// against extended precision: 3.5e-13 through the library functions, 3.4e-13
// here (3.6e-13 without the corrected quotients).
template <bool GZ, bool TMI>
__device__ __forceinline__ void pair_gradient_fp64(const double* C, double gsn, double ms, double ox, double oy,
                                                   double oz, double gco, double mco, GradAcc& A) {
    const double L0 = C[GC_L0], cx = C[GC_CX], cy = C[GC_CY], L1 = C[GC_L1], L2 = C[GC_L2];
    const double G0 = GZ ? gco * gsn : 0.0;      // gravity adjoint x group scale
    const double Gs = GZ ? G0 * C[GC_ZZ] : 0.0;  // ... x n_z
    const double Ts = TMI ? mco * ms : 0.0;      // magnetic adjoint x group TMI scale
    if (G0 == 0.0 && Ts == 0.0) return;
    const d3 dd = mk3(ox - C[GC_AX], oy - C[GC_AY], oz - C[GC_AZ]);
    const double x = dd.x * C[GC_XX] + dd.y * C[GC_XY] + dd.z * C[GC_XZ];
    const double y = dd.x * C[GC_YX] + dd.y * C[GC_YY] + dd.z * C[GC_YZ];
    const double z = dd.x * C[GC_ZX] + dd.y * C[GC_ZY] + dd.z * C[GC_ZZ];
    const double rbx = L0 - x, rcx = cx - x, rcy = cy - y;
    const double z2 = z * z, yz2 = fma(y, y, z2);
    const double a2 = fma(x, x, yz2), b2 = fma(rbx, rbx, yz2), c2 = fma(rcx, rcx, fma(rcy, rcy, z2));
    double ia, ib, ic;
    const double la = sqrt_inv64(a2, &ia), lb = sqrt_inv64(b2, &ib), lc = sqrt_inv64(c2, &ic);
    const double D0 = la + lb, D1 = lb + lc, D2 = lc + la;
    const double m0 = fma(D0, D0, -L0 * L0), m1 = fma(D1, D1, -L1 * L1), m2 = fma(D2, D2, -L2 * L2);
    const double q0 = rcp_pos64(D0), q1 = rcp_pos64(D1), q2 = rcp_pos64(D2);
    double v0 = L0 * q0, v1 = L1 * q1, v2 = L2 * q2;
    if (GZ && !TMI) {  // the gz terms cancel: quotients to half an ulp
        v0 = fma(fma(-v0, D0, L0), q0, v0);
        v1 = fma(fma(-v1, D1, L1), q1, v1);
        v2 = fma(fma(-v2, D2, L2), q2, v2);
    }
    const unsigned vmax = max_ratio_hi(v0, v1, v2);
    double om, l0, l1, l2, W0, W1, W2;
    bool lv0 = true, lv1 = true, lv2 = true;
    if (vmax < 0x3fe00000u) {  // every v < 1/2
        W0 = (L0 + L0) * rcp_pos64(m0);
        W1 = (L1 + L1) * rcp_pos64(m1);
        W2 = (L2 + L2) * rcp_pos64(m2);
        // ra . rb = (a2 + b2 - L^2) / 2
        const double dab = 0.5 * fma(-L0, L0, a2 + b2), dbc = 0.5 * fma(-L1, L1, b2 + c2),
                     dac = 0.5 * fma(-L2, L2, c2 + a2);
        const double den = fma(la * lb, lc, fma(dab, lc, fma(dac, lb, dbc * la)));
        om = 2.0 * atan_poly64(-z * (L0 * cy) * rcp_pos64(den));
        if (vmax < 0x3fd00000u) {  // every v < 1/4
            l0 = 2.0 * atanh_short64(v0);
            l1 = 2.0 * atanh_short64(v1);
            l2 = 2.0 * atanh_short64(v2);
        } else {
            l0 = 2.0 * atanh_poly64(v0);
            l1 = 2.0 * atanh_poly64(v1);
            l2 = 2.0 * atanh_poly64(v2);
        }
    } else {
        const NearTerms N = gradient_near_terms(x, y, z, L0, cx, cy, L1, L2);
        if (N.dead) return;
        om = N.om;
        l0 = N.lam[0]; l1 = N.lam[1]; l2 = N.lam[2];
        W0 = N.W[0]; W1 = N.W[1]; W2 = N.W[2];
        lv0 = N.live & 1; lv1 = N.live & 2; lv2 = N.live & 4;
    }
    // edges: 0 a->b (e = (1, 0)), 1 b->c, 2 c->a
    const double e1x = C[GC_E1X], e1y = C[GC_E1Y], e2x = C[GC_E2X], e2y = C[GC_E2Y];
    const double dp0 = y, dp1 = fma(rbx, e1y, y * e1x), dp2 = fma(rcx, e2y, -rcy * e2x);  // -r1 . n_i
    double kom, k0, k1, k2;
    if (TMI) {
        kom = Ts * C[GC_MF];
        k0 = Ts * C[GC_MT0];
        k1 = Ts * C[GC_MT1];
        k2 = Ts * C[GC_MT2];
    }
    if (GZ) {
        kom = TMI ? fma(Gs, z, kom) : Gs * z;
        k0 = TMI ? fma(Gs, dp0, k0) : Gs * dp0;
        k1 = TMI ? fma(Gs, dp1, k1) : Gs * dp1;
        k2 = TMI ? fma(Gs, dp2, k2) : Gs * dp2;
    }
    if (!lv0) k0 = 0.0;
    if (!lv1) k1 = 0.0;
    if (!lv2) k2 = 0.0;
    const double kz = kom * z;
    const double al0 = W0 * fma(k0, dp0, kz), be0 = W0 * fma(k0, z, -kom * dp0);
    const double al1 = W1 * fma(k1, dp1, kz), be1 = W1 * fma(k1, z, -kom * dp1);
    const double al2 = W2 * fma(k2, dp2, kz), be2 = W2 * fma(k2, z, -kom * dp2);
    A.va.x = fma(ia, fma(-al2, e2y, fma(k2, e2x, -k0)), A.va.x);
    A.va.y = fma(ia, fma(al2, e2x, fma(k2, e2y, al0)), A.va.y);
    A.va.z = fma(ia, be0 + be2, A.va.z);
    A.vb.x = fma(ib, fma(-al1, e1y, fma(-k1, e1x, k0)), A.vb.x);
    A.vb.y = fma(ib, fma(al1, e1x, fma(-k1, e1y, al0)), A.vb.y);
    A.vb.z = fma(ib, be0 + be1, A.vb.z);
    A.vc.x = fma(ic, fma(-al2, e2y, fma(-k2, e2x, fma(-al1, e1y, k1 * e1x))), A.vc.x);
    A.vc.y = fma(ic, fma(al2, e2x, fma(-k2, e2y, fma(al1, e1x, k1 * e1y))), A.vc.y);
    A.vc.z = fma(ic, be1 + be2, A.vc.z);
    if (GZ) {
        const double w0 = Gs * l0, w1 = Gs * l1, w2 = Gs * l2, wo = Gs * om;
        A.ai = fma(G0, fma(dp0, l0, fma(dp1, l1, fma(dp2, l2, z * om))), A.ai);
        A.alam[0] += w0; A.alam[1] += w1; A.alam[2] += w2;
        A.aom += wo;
        A.bh.x = fma(-x, wo, A.bh.x); A.bh.y = fma(-y, wo, A.bh.y);
        A.bl[0].x = fma(-x, w0, A.bl[0].x); A.bl[0].z = fma(-z, w0, A.bl[0].z);
        A.bl[1].x = fma(rbx, w1, A.bl[1].x); A.bl[1].y = fma(-y, w1, A.bl[1].y); A.bl[1].z = fma(-z, w1, A.bl[1].z);
        A.bl[2].x = fma(rcx, w2, A.bl[2].x); A.bl[2].y = fma(rcy, w2, A.bl[2].y); A.bl[2].z = fma(-z, w2, A.bl[2].z);
    }
    if (TMI) {
        A.amf = fma(Ts, om, A.amf);
        A.amt[0] = fma(Ts, l0, A.amt[0]);
        A.amt[1] = fma(Ts, l1, A.amt[1]);
        A.amt[2] = fma(Ts, l2, A.amt[2]);
    }
}

__device__ __forceinline__ bool facet_grad_active(const double* C) {
    int flags = static_cast<int>(C[GC_FLAGS]);
    return (flags & 1) && (flags & 2) && (C[GC_GS] != 0.0 || C[GC_MS] != 0.0);
}

// Per-station facet gradients for dense Jacobian rows of one data type (GZ:
// gravity, else TMI; unit adjoints).  Grid: x = facet warps (one facet per
// thread), y = stations; part layout [station][9][T] (vertex a xyz, b xyz, c
// xyz; global frame).  Stations are warp-uniform loads.
template <bool GZ>
__global__ void __launch_bounds__(32) k_gradient_fp64(int T, const double* __restrict__ gc,
                                                      const double* __restrict__ sta,
                                                      const int16_t* __restrict__ face_group,
                                                      const GroupConst* __restrict__ groups, d3 fdir,
                                                      double* __restrict__ part) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (f >= T) return;
    double C[NGC];
#pragma unroll
    for (int k = 0; k < NGC; ++k) C[k] = gc[(size_t)k * T + f];
    double outv[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (facet_grad_active(C)) {
        GradAcc A;
        grad_acc_zero(A);
        pair_gradient_fp64<GZ, !GZ>(C, C[GC_GS], C[GC_MS], sta[3 * j], sta[3 * j + 1], sta[3 * j + 2], 1.0, 1.0, A);
        grad_finalize(C, A, groups[face_group[f]], fdir, outv);
    }
    for (int k = 0; k < 9; ++k) part[((size_t)j * 9 + k) * T + f] = outv[k];
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// Warp totals of the accumulators, transposed: 28 sums padded to 32 are folded
// in five halving steps (31 exchanges instead of 28 x 5), lane k writes total
// k to row[k] (shared memory, 32 doubles), and every lane reads them back.
__device__ __forceinline__ void grad_acc_warp_sum(GradAcc& A, double* row) {
    const int lane = threadIdx.x & 31;
    double v[32] = {A.va.x, A.va.y, A.va.z, A.vb.x, A.vb.y, A.vb.z, A.vc.x, A.vc.y, A.vc.z,
                    A.bh.x, A.bh.y, A.bl[0].x, A.bl[0].z, A.bl[1].x, A.bl[1].y, A.bl[1].z,
                    A.bl[2].x, A.bl[2].y, A.bl[2].z, A.alam[0], A.alam[1], A.alam[2], A.aom, A.ai,
                    A.amf, A.amt[0], A.amt[1], A.amt[2], 0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
        const bool upper = (lane & step) != 0;
#pragma unroll
        for (int i = 0; i < step; ++i) {
            const double send = upper ? v[i] : v[i + step];
            const double keep = upper ? v[i + step] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, step);
        }
    }
    row[lane] = v[0];
    __syncwarp();
    A.va = mk3(row[0], row[1], row[2]);
    A.vb = mk3(row[3], row[4], row[5]);
    A.vc = mk3(row[6], row[7], row[8]);
    A.bh = mk3(row[9], row[10], 0.0);
    A.bl[0] = mk3(row[11], 0.0, row[12]);
    A.bl[1] = mk3(row[13], row[14], row[15]);
    A.bl[2] = mk3(row[16], row[17], row[18]);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        A.alam[i] = row[19 + i];
        A.amt[i] = row[25 + i];
    }
    A.aom = row[22];
    A.ai = row[23];
    A.amf = row[24];
}

// Objective gradient, FP64: one warp per facet.  The warp visits the
// facet's near station tiles (every tile when tau >= 1e30), lanes taking
// the tile's stations in turn; per-lane sums are reduced across the warp
// once per facet and lane 0 finalises.  The work of a facet is spread over
// 32 lanes, so facets with many near tiles leave no long tail behind.
// GZ / TMI: which adjoints there are (gcoef, mcoef not null).
// Warps run over `facets` (those with a DOF vertex); grid.y splits the
// station tiles into chunks of tiles_per_chunk so that a model with few such
// facets still fills the GPU.  part layout [chunk][9][T].
// FP64 pipe 63 % busy at 12 warps per SM (168 registers, of which 56 hold the
// sums): 24.6 M pairs (8,308 facets, 2,964 stations) took 1,131 us with the
// library functions, 484 us now; a 1,280-facet body under 1,600 stations 115
// and 55 us.  Two CTAs per SM (no spill) 523 us, four (128 registers) 539;
// CTAs of one or two warps no different.
template <bool GZ, bool TMI>
__global__ void __launch_bounds__(128, 3) k_gradient_warp_fp64(int T, const double* __restrict__ gc, int S,
                                                            const double* __restrict__ sta,
                                                            const double* __restrict__ gcoef,
                                                            const double* __restrict__ mcoef,
                                                            const double* __restrict__ tile_box,
                                                            const int16_t* __restrict__ face_group,
                                                            const GroupConst* __restrict__ groups, d3 fdir, double tau,
                                                            const int32_t* __restrict__ facets, int nfacets,
        int tiles_per_chunk, const int32_t* __restrict__ grp_sta_off,
        const int32_t* __restrict__ grp_tile_off, double* __restrict__ part) {
    const int lane = threadIdx.x & 31;
    const int w = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
    if (w >= nfacets) return;  // warp-uniform
    const int f = facets[w];
    if (grp_sta_off) {  // batched bodies: only the facet's own body's stations
        const int g = face_group[f], sb = grp_sta_off[g];
        S = grp_sta_off[g + 1] - sb;
        sta += 3 * (size_t)sb;
        if (gcoef) gcoef += sb;
        if (mcoef) mcoef += sb;
        tile_box += 6 * (size_t)grp_tile_off[g];
    }
    // this chunk's station tiles
    const int ntiles_all = (S + kStationTile - 1) / kStationTile;
    const int tbeg = blockIdx.y * tiles_per_chunk, ntiles = min(ntiles_all, tbeg + tiles_per_chunk);
    part += (size_t)blockIdx.y * 9 * T;
    // the facet's constants live in shared memory (one row per warp): the
    // per-lane FP64 sums and pair temporaries need the registers
    __shared__ double Csh[4][NGC], sums[4][32];
    double* C = Csh[threadIdx.x >> 5];
    if (lane < NGC) C[lane] = gc[(size_t)lane * T + f];
    __syncwarp();
    double outv[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (facet_grad_active(C)) {
        GradAcc A;
        grad_acc_zero(A);
        const double gsn = C[GC_GS], ms = C[GC_MS];
        const FarKey key = facet_far_key(C, tau);
        bool any = false;
        for (int t0 = tbeg; t0 < ntiles; t0 += 32) {
            const int t = t0 + lane;
            const bool nearT = t < ntiles && !tile_far(key, tile_box + 6 * (size_t)t);
            unsigned m = __ballot_sync(0xffffffffu, nearT);
            any |= m != 0;
            while (m) {
                const int b = __ffs(m) - 1;
                m &= m - 1;
                const int s0 = (t0 + b) * kStationTile;
#pragma unroll
                for (int k = 0; k < kStationTile; k += 32) {
                    const int j = s0 + k + lane;
                    if (j < S)
                        pair_gradient_fp64<GZ, TMI>(C, gsn, ms, sta[3 * j], sta[3 * j + 1], sta[3 * j + 2],
                                                    GZ ? gcoef[j] : 0.0, TMI ? mcoef[j] : 0.0, A);
                }
            }
        }
        if (any) {
            grad_acc_warp_sum(A, sums[threadIdx.x >> 5]);
            if (lane == 0) grad_finalize(C, A, groups[face_group[f]], fdir, outv);
        }
    }
    if (lane == 0)
        for (int k = 0; k < 9; ++k) part[(size_t)k * T + f] = outv[k];
}

// Finite-difference-XY partials (see k_face_prep_fdxy): one warp per listed
// facet x station chunk (tiles_per_chunk tiles of kStationTile stations),
// lanes over the chunk's stations.  Per station, the facet term of the base
// record and of the six moved copies (pair_forward_fp64), contracted with the station adjoints and the group
// scales of the analytic kernels (zero for collapsed facets):
//   sum_s (G_s (F_k - F_0) + T_s (M_k - M_0)) / h.
// Writes the x and y partials of the three corners, and zero z, into this
// chunk's slot of part ([chunk][9][T]).
__global__ void __launch_bounds__(128) k_gradient_fdxy(int T, int nf, const int32_t* __restrict__ facets,
                                                       const double* __restrict__ fcfd, const double* __restrict__ gc,
                                                       int S, const double* __restrict__ sta,
                                                       const double* __restrict__ gcoef,
                                                       const double* __restrict__ mcoef,
                                                       const int16_t* __restrict__ face_group, double inv_h,
                                                       int tiles_per_chunk, const int32_t* __restrict__ grp_sta_off,
                                                       double* __restrict__ part) {
    const int lane = threadIdx.x & 31;
    const int w = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
    if (w >= nf) return;  // warp-uniform
    const int f = facets[w];
    if (grp_sta_off) {  // batched bodies: only the facet's own body's stations
        const int g = face_group[f], sb = grp_sta_off[g];
        S = grp_sta_off[g + 1] - sb;
        sta += 3 * (size_t)sb;
        if (gcoef) gcoef += sb;
        if (mcoef) mcoef += sb;
    }
    const int s0 = blockIdx.y * tiles_per_chunk * kStationTile;
    const int s1 = min(S, s0 + tiles_per_chunk * kStationTile);
    part += (size_t)blockIdx.y * 9 * T;
    __shared__ __align__(16) double R[4][7 * NFC];
    double* rec = R[threadIdx.x >> 5];
    for (int q = lane; q < 7 * NFC; q += 32) rec[q] = fcfd[(size_t)w * 7 * NFC + q];
    __syncwarp();
    const double gs = gc[(size_t)GC_GS * T + f], ms = gc[(size_t)GC_MS * T + f];
    double acc[6] = {0, 0, 0, 0, 0, 0};
    if (gs != 0.0 || ms != 0.0) {
        for (int j = s0 + lane; j < s1; j += 32) {
            const double G = gcoef ? gcoef[j] * gs : 0.0, M = mcoef ? mcoef[j] * ms : 0.0;
            if (G == 0.0 && M == 0.0) continue;
            const d3 o = mk3(sta[3 * (size_t)j], sta[3 * (size_t)j + 1], sta[3 * (size_t)j + 2]);
            double g0 = 0.0, m0 = 0.0;
            pair_forward_fp64<true, true>(rec, o, &g0, &m0);
#pragma unroll 1
            for (int k = 0; k < 6; ++k) {
                double gk = 0.0, mk = 0.0;
                pair_forward_fp64<true, true>(rec + (k + 1) * NFC, o, &gk, &mk);
                acc[k] += G * (gk - g0) + M * (mk - m0);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) acc[k] = warp_sum(acc[k]);
    if (lane == 0)
        for (int c = 0; c < 3; ++c) {
            part[(size_t)(3 * c) * T + f] = acc[2 * c] * inv_h;
            part[(size_t)(3 * c + 1) * T + f] = acc[2 * c + 1] * inv_h;
            part[(size_t)(3 * c + 2) * T + f] = 0.0;
        }
}

// Sums facet partials into vertex gradients: one warp per listed vertex,
// lanes over its (chunk, incident facet corner) items, then a fixed warp
// reduction (deterministic).  Slots from fd_from on hold
// finite-difference-XY partials: when fd_from < nchunks, x and y come from
// those slots only and z from the slots before them.
__global__ void k_vertex_reduce(int nverts, const int32_t* __restrict__ verts, const int32_t* __restrict__ vf_off,
                                const int32_t* __restrict__ vf, int T, int nchunks, int fd_from,
                                const double* __restrict__ part, double* __restrict__ vgrad) {
    const int i = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= nverts) return;  // warp-uniform
    const int v = verts[i];
    const int b = vf_off[v], ninc = vf_off[v + 1] - b;
    const int items = nchunks * ninc;
    double gx = 0, gy = 0, gz = 0;
    for (int it = lane; it < items; it += 32) {
        const int c = it / ninc, k = b + it % ninc;
        const int f = vf[k] / 3, corner = vf[k] % 3;
        const double* p = part + ((size_t)c * 9 + 3 * corner) * T + f;
        const bool xy = fd_from >= nchunks || c >= fd_from;
        if (xy) {
            gx += p[0];
            gy += p[(size_t)T];
        }
        if (c < fd_from) gz += p[(size_t)2 * T];
    }
    gx = warp_sum(gx);
    gy = warp_sum(gy);
    gz = warp_sum(gz);
    if (lane == 0) {
        vgrad[3 * v] = gx;
        vgrad[3 * v + 1] = gy;
        vgrad[3 * v + 2] = gz;
    }
}

// grad[d] = sum_refs vgrad[vertex][axis] * axis scale + reference-model term
// (gather of gravity_forward.cpp:269-289 contracted; reference_model.cpp:22-25).
__global__ void k_dof_gather(int np, const int32_t* __restrict__ dof_off, const int32_t* __restrict__ ref_vertex,
                             const uint8_t* __restrict__ ref_axis, const double* __restrict__ ref_scale,
                             const double* __restrict__ vgrad, const double* __restrict__ params,
                             const double* __restrict__ ref_params, double ref_weight,
                             const double* __restrict__ vgrad_smooth, double smooth_weight,
                             double* __restrict__ grad) {
    int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= np) return;
    double acc = 0.0;
    for (int r = dof_off[d]; r < dof_off[d + 1]; ++r) acc += vgrad[3 * ref_vertex[r] + ref_axis[r]] * ref_scale[r];
    if (vgrad_smooth) {  // SurfaceSmoothness::gradient gather (smoothness.cpp:231-242), times its weight
        double s = 0.0;
        for (int r = dof_off[d]; r < dof_off[d + 1]; ++r)
            s += vgrad_smooth[3 * ref_vertex[r] + ref_axis[r]] * ref_scale[r];
        acc += smooth_weight * s;
    }
    if (ref_params) acc += ref_weight * (params[d] - ref_params[d]);
    grad[d] = acc;
}

// Chain gather (no reference counterpart; the reference reads the vertex
// gradient at the DOF vertices only, gravity_forward.cpp:270-289).  The
// scatter is DOF writes -> interpolation -> averaging; its adjoint runs the
// transposes in reverse.  The averaging's transpose is the averaging itself
// (k_sync_shared on the gradient: its matrix is symmetric).  The
// interpolation's transpose, out of place: a source receives w x the
// gradient of each row it feeds, a row keeps nothing (its position was
// overwritten), every other vertex keeps its own.  Fixed summation order,
// no atomics.  A warp per vertex, lanes over its entries; a control point that
// feeds more than kAdjointHeavy rows (a few drive thousands) takes the whole
// CTA.  106,000 vertices, a few sources with tens of thousands of rows between them: 3.8 ms
// with a thread per vertex, well under 0.1 ms now.
constexpr int kAdjointHeavy = 512, kAdjointThreads = 256;
__global__ void __launch_bounds__(kAdjointThreads) k_interp_adjoint(
    int V, const int32_t* __restrict__ interp_off, const int32_t* __restrict__ adj_off,
    const int32_t* __restrict__ adj_row, const double* __restrict__ adj_w, const double* __restrict__ vg,
    double* __restrict__ out) {
    constexpr int kWarps = kAdjointThreads / 32;
    __shared__ double part[kWarps][3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, first = blockIdx.x * kWarps;
    auto sum = [&](int b, int e, int start, int step) {
        d3 g = mk3(0.0, 0.0, 0.0);
        for (int k = b + start; k < e; k += step) {
            const double w = adj_w[k];
            const double* q = vg + 3 * (size_t)adj_row[k];
            g = mk3(g.x + w * q[0], g.y + w * q[1], g.z + w * q[2]);
        }
        return mk3(warp_sum(g.x), warp_sum(g.y), warp_sum(g.z));
    };
    auto store = [&](int v, d3 g) {
        const bool row = interp_off[v + 1] > interp_off[v];
        for (int k = 0; k < 3; ++k)
            out[3 * (size_t)v + k] = (row ? 0.0 : vg[3 * (size_t)v + k]) + (k == 0 ? g.x : k == 1 ? g.y : g.z);
    };
    auto heavy = [&](int v) { return v < V && adj_off[v + 1] - adj_off[v] > kAdjointHeavy; };
    const int mine = first + warp;
    if (mine < V && !heavy(mine)) {  // warp-uniform
        const d3 g = sum(adj_off[mine], adj_off[mine + 1], lane, 32);
        if (lane == 0) store(mine, g);
    }
    for (int v = first; v < first + kWarps; ++v) {
        if (!heavy(v)) continue;  // block-uniform
        const d3 g = sum(adj_off[v], adj_off[v + 1], (int)threadIdx.x, kAdjointThreads);
        if (lane == 0) { part[warp][0] = g.x; part[warp][1] = g.y; part[warp][2] = g.z; }
        __syncthreads();
        if (threadIdx.x == 0) {
            d3 t = mk3(0.0, 0.0, 0.0);
            for (int w = 0; w < kWarps; ++w) t = t + mk3(part[w][0], part[w][1], part[w][2]);
            store(v, t);
        }
        __syncthreads();
    }
}

// y += a x over n doubles (the smoothness vertex gradient into the misfit's
// before the chain gather).
__global__ void k_axpy(size_t n, double a, const double* __restrict__ x, double* __restrict__ y) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < n) y[i] += a * x[i];
}

// Dense Jacobian rows from per-station facet partials (one chunk per
// station): J[row[s]][d] = sum_refs (sum_{(f,c) of v} part) * scale, with the
// reference's |vertex gradient| < 1e-30 skip.  row nullptr: s itself.
__global__ void k_jacobian_gather(int nst, int np, const int32_t* __restrict__ row, const int32_t* __restrict__ dof_off,
                                  const int32_t* __restrict__ ref_vertex, const uint8_t* __restrict__ ref_axis,
                                  const double* __restrict__ ref_scale, const int32_t* __restrict__ vf_off,
                                  const int32_t* __restrict__ vf, int T, const double* __restrict__ part,
                                  double* __restrict__ J, int ld) {
    int d = blockIdx.x * blockDim.x + threadIdx.x;
    int s = blockIdx.y;
    if (d >= np || s >= nst) return;
    double acc = 0.0;
    for (int r = dof_off[d]; r < dof_off[d + 1]; ++r) {
        int v = ref_vertex[r], ax = ref_axis[r];
        double pg = 0.0;
        for (int k = vf_off[v]; k < vf_off[v + 1]; ++k) {
            int f = vf[k] / 3, corner = vf[k] % 3;
            pg += part[((size_t)s * 9 + 3 * corner + ax) * T + f];
        }
        if (fabs(pg) < 1e-30) continue;
        acc += pg * ref_scale[r];
    }
    J[(size_t)(row ? row[s] : s) * ld + d] = acc;
}

// Final deterministic reduction of block partials and objective assembly:
// out = {grav misfit, mag misfit, reg, 0, total}.
// ---------------------------------------------------------- smoothness ----
// SurfaceSmoothness (modules/litho-regularization/src/regularization/
// smoothness.cpp): every non-fixed vertex against the mean of its
// same-freedom mesh neighbours (nbr: CSR, ascending, built on the host like
// SurfaceMesh::buildNeighbors surface_mesh.cpp:265-286).

// Free axes of a VertexFreedom code (surface_mesh.h:9-19); ALONG_VECTOR is
// rejected on the host.
__device__ __forceinline__ void freedom_mask(int fr, bool m[3]) {
    m[0] = fr == 2 || fr == 5 || fr == 6 || fr == 8;
    m[1] = fr == 3 || fr == 5 || fr == 7 || fr == 8;
    m[2] = fr == 1 || fr == 6 || fr == 7 || fr == 8;
}

// diff_v = p_v - mean_v (evaluate :29-49) and the per-vertex penalty
// 0.5 |mask diff|^2 (:51-99), summed per block; same operation order as the
// reference.
__global__ void k_smooth_diff(int V, const double* __restrict__ pos, const uint8_t* __restrict__ freedom,
                              const int32_t* __restrict__ off, const int32_t* __restrict__ nbr,
                              double* __restrict__ diff, double* __restrict__ block_pen) {
    __shared__ double red[256];
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    double pen = 0.0;
    if (v < V) {
        const int b = off[v], e = off[v + 1];
        double d0 = 0.0, d1 = 0.0, d2 = 0.0;
        if (e > b) {
            double m0 = 0.0, m1 = 0.0, m2 = 0.0;
            for (int i = b; i < e; ++i) {
                const double* q = pos + 3 * (size_t)nbr[i];
                m0 = __dadd_rn(m0, q[0]); m1 = __dadd_rn(m1, q[1]); m2 = __dadd_rn(m2, q[2]);
            }
            const double n = static_cast<double>(e - b);
            m0 = __ddiv_rn(m0, n); m1 = __ddiv_rn(m1, n); m2 = __ddiv_rn(m2, n);
            d0 = __dsub_rn(pos[3 * (size_t)v], m0);
            d1 = __dsub_rn(pos[3 * (size_t)v + 1], m1);
            d2 = __dsub_rn(pos[3 * (size_t)v + 2], m2);
            auto sq = [](double d) { return __dmul_rn(d, d); };
            switch (freedom[v]) {
            case 1: pen = __dmul_rn(__dmul_rn(0.5, d2), d2); break;
            case 2: pen = __dmul_rn(__dmul_rn(0.5, d0), d0); break;
            case 3: pen = __dmul_rn(__dmul_rn(0.5, d1), d1); break;
            case 5: pen = __dmul_rn(0.5, __dadd_rn(sq(d0), sq(d1))); break;
            case 6: pen = __dmul_rn(0.5, __dadd_rn(sq(d0), sq(d2))); break;
            case 7: pen = __dmul_rn(0.5, __dadd_rn(sq(d1), sq(d2))); break;
            case 8: pen = __dmul_rn(0.5, __dadd_rn(__dadd_rn(sq(d0), sq(d1)), sq(d2))); break;
            default: break;
            }
        }
        diff[3 * (size_t)v] = d0; diff[3 * (size_t)v + 1] = d1; diff[3 * (size_t)v + 2] = d2;
    }
    red[threadIdx.x] = pen;
    __syncthreads();
    for (int k = blockDim.x / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) block_pen[blockIdx.x] = red[0];
}

// Per-vertex smoothness gradient (gradient :152-242): own term mask(diff_v),
// then -mask(diff_u) / n_u for every same-freedom neighbour u in ascending
// order (the neighbour relation and the freedom filter are symmetric, so the
// vertices that add to v are exactly v's own list).
__global__ void k_smooth_vgrad(int V, const uint8_t* __restrict__ freedom, const int32_t* __restrict__ off,
                               const int32_t* __restrict__ nbr, const double* __restrict__ diff,
                               double* __restrict__ vg) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    double g0 = 0.0, g1 = 0.0, g2 = 0.0;
    const int b = off[v], e = off[v + 1];
    if (e > b) {
        bool m[3];
        freedom_mask(freedom[v], m);
        if (m[0]) g0 = diff[3 * (size_t)v];
        if (m[1]) g1 = diff[3 * (size_t)v + 1];
        if (m[2]) g2 = diff[3 * (size_t)v + 2];
        for (int i = b; i < e; ++i) {
            const int u = nbr[i];
            const double nu = static_cast<double>(off[u + 1] - off[u]);
            if (m[0]) g0 = __dadd_rn(g0, __ddiv_rn(-diff[3 * (size_t)u], nu));
            if (m[1]) g1 = __dadd_rn(g1, __ddiv_rn(-diff[3 * (size_t)u + 1], nu));
            if (m[2]) g2 = __dadd_rn(g2, __ddiv_rn(-diff[3 * (size_t)u + 2], nu));
        }
    }
    vg[3 * (size_t)v] = g0; vg[3 * (size_t)v + 1] = g1; vg[3 * (size_t)v + 2] = g2;
}

// Objective components: misfits from the residual block sums; regularisation
// = smoothness (weight x block penalty sums) + reference-model term, in the
// order the runner registers them (runner.cpp:164-179).
__global__ void k_objective_final(int nbg, const double* __restrict__ bg, int nbm, const double* __restrict__ bm,
                                  double alpha, int np, const double* __restrict__ params,
                                  const double* __restrict__ ref_params, double ref_weight, int nbs,
                                  const double* __restrict__ bs, double smooth_weight, double* __restrict__ out5,
                                  double* __restrict__ f_out) {
    __shared__ double red[256];
    double reg = 0.0;
    if (ref_params)
        for (int d = threadIdx.x; d < np; d += blockDim.x) {
            double dd = params[d] - ref_params[d];
            reg += dd * dd;
        }
    red[threadIdx.x] = reg;
    __syncthreads();
    for (int k = blockDim.x / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        double g = 0.0, m = 0.0;
        for (int i = 0; i < nbg; ++i) g += bg[i];
        for (int i = 0; i < nbm; ++i) m += bm[i];
        double r = ref_params ? 0.5 * ref_weight * red[0] : 0.0;
        if (bs) {
            double sp = 0.0;
            for (int i = 0; i < nbs; ++i) sp += bs[i];
            r = smooth_weight * sp + r;
        }
        double total = g + alpha * m + r;
        out5[0] = g; out5[1] = m; out5[2] = r; out5[3] = 0.0; out5[4] = total;
        if (f_out) *f_out = total;
    }
}

}  // namespace litho_b200
