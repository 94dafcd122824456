// Mixed-precision (FP32 bulk, FP64 near field) forward and gradient kernels.
//
// Why the split: the facet formula of the reference (sum_i d_perp_i Lambda_i
// - h Omega, faceNagyContribution gravity_forward.cpp:13-42) is a
// cancellation.  Over a closed lithology surface the edge terms are ~100-500
// times larger than their sum, so FP32 rounding of Lambda and of the edge
// coefficients alone costs 1e-6..5e-6 relative in gz.  Two facts fix it:
//  * a facet far from a station tile (centroid distance >= tau x facet size)
//    is integrated directly: gz facet = n_z * integral of 1/r over the facet,
//    evaluated by quadrature in FP32 (positive terms, no cancellation):
//    Dunavant's 6-point degree-4 rule, 3 points beyond 4 tau, in the forward
//    and in the gradient;
//  * a facet near the tile uses the analytic formula in FP64, in the facet's
//    local frame (origin at a vertex, x along the longest edge, z along the
//    unit normal).
// The TMI facet term of the reference (magneticFacet magnetic_forward.cpp:
// 312-347) has no such cancellation; far facets evaluate it analytically in
// FP32, with Lambda from the symmetric form 2 atanh(L / (d1 + d2)).
#pragma once
#include "kernels_fp64.cuh"

namespace litho_b200 {

// Mixed facet constants, SoA [NMC][T] (FP64; FP32 copies are made in shared
// memory).  The local frame starts at vertex `a` of the facet rotated so that
// a->b is the longest edge; magnetic products follow that rotation.
enum MixedConst {
    MC_AX = 0, MC_AY, MC_AZ,          // local origin
    MC_XX, MC_XY, MC_XZ,              // local x axis
    MC_YX, MC_YY, MC_YZ,              // local y axis
    MC_ZX, MC_ZY, MC_ZZ,              // local z axis (unit normal)
    MC_L0, MC_CX, MC_CY,              // b = (L0, 0, 0), c = (CX, CY, 0)
    MC_E1X, MC_E1Y, MC_L1,            // edge b->c
    MC_E2X, MC_E2Y, MC_L2,            // edge c->a
    MC_SGZ,                           // n_z * G * rho * 1e3 * 1e5 (gz facet scale)
    MC_MF, MC_MT0, MC_MT1, MC_MT2,    // -amp*100/(4 pi) * direction products (TMI facet scales)
    MC_CENX, MC_CENY, MC_CENZ,        // centroid (near/far test)
    MC_SIZE,                          // longest edge
    MC_VALID,                         // 1: facet contributes (twice-area >= 1e-15)
    NMC
};

// Weights of Radon's 7-point degree-5 rule on the triangle (they sum to 1;
// multiply by the area): 9/40 at the centroid, (155 - sqrt 15)/1200 at the
// (a1, b1, b1) permutations with b1 = (6 - sqrt 15)/21, a1 = 1 - 2 b1, and
// (155 + sqrt 15)/1200 at the (a2, b2, b2) ones with b2 = (6 + sqrt 15)/21.
__constant__ float kRadonW[7] = {0.225f, 0.1259391805448271f, 0.1259391805448271f, 0.1259391805448271f,
                                 0.1323941527885062f, 0.1323941527885062f, 0.1323941527885062f};

// Dunavant's 6-point degree-4 rule (D. A. Dunavant, "High degree efficient
// symmetrical Gaussian quadrature rules for the triangle", IJNME 21, 1985):
// (a, b, b) permutations with a = 0.108103018168070, b = 0.445948490915965,
// weight 0.223381589678011, and a = 0.816847572980459, b = 0.091576213509771,
// weight 0.109951743655322.  Its degree-6 error term, which sets the error at
// the far-field distances, is as small as the 7-point rule's; one point fewer.
__constant__ float kDun6Bb[6] = {0.445948490915965f, 0.108103018168070f, 0.445948490915965f,
                                 0.091576213509771f, 0.816847572980459f, 0.091576213509771f};
__constant__ float kDun6Bc[6] = {0.445948490915965f, 0.445948490915965f, 0.108103018168070f,
                                 0.091576213509771f, 0.091576213509771f, 0.816847572980459f};
__constant__ float kDun6W[6] = {0.223381589678011f, 0.223381589678011f, 0.223381589678011f,
                                0.109951743655322f, 0.109951743655322f, 0.109951743655322f};
// 3-point degree-2 rule: (2/3, 1/6, 1/6) permutations, weights 1/3 (Strang &
// Fix).  Taken beyond 4 tau x size, where its (size / distance)^3 error term
// is below 1e-7 of the station total.
__constant__ float kTri3Bb[3] = {0.1666666666666667f, 0.6666666666666667f, 0.1666666666666667f};
__constant__ float kTri3Bc[3] = {0.1666666666666667f, 0.1666666666666667f, 0.6666666666666667f};

// Radon's rule on the four midpoint sub-triangles (a, ab, ca), (ab, b, bc),
// (ca, bc, c), (ab, bc, ca): 28 points in the parent's barycentric (beta_b,
// beta_c), weights kRadonW[q % 7] / 4.  Its error at distance ratio tau/2
// matches the 7-point rule's at tau (degree-5 error ~ (size / distance)^6),
// so it takes the mid field tau/2 <= distance / size < tau in FP32.
__constant__ float kRadon4Bb[28] = {
    0.1666666666666667f, 0.0506432536617282f, 0.3987134926765437f, 0.0506432536617282f, 0.2350710320525576f,
    0.0298579358948849f, 0.2350710320525576f, 0.6666666666666666f, 0.5506432536617281f, 0.8987134926765437f,
    0.5506432536617281f, 0.7350710320525575f, 0.5298579358948849f, 0.7350710320525576f, 0.1666666666666667f,
    0.0506432536617282f, 0.3987134926765437f, 0.0506432536617282f, 0.2350710320525576f, 0.0298579358948849f,
    0.2350710320525576f, 0.3333333333333334f, 0.4493567463382718f, 0.4493567463382718f, 0.1012865073234563f,
    0.2649289679474425f, 0.2649289679474425f, 0.4701420641051152f};
__constant__ float kRadon4Bc[28] = {
    0.1666666666666667f, 0.0506432536617282f, 0.0506432536617282f, 0.3987134926765437f, 0.2350710320525576f,
    0.2350710320525576f, 0.0298579358948849f, 0.1666666666666667f, 0.0506432536617282f, 0.0506432536617282f,
    0.3987134926765437f, 0.2350710320525576f, 0.2350710320525576f, 0.0298579358948849f, 0.6666666666666667f,
    0.5506432536617282f, 0.5506432536617282f, 0.8987134926765437f, 0.7350710320525575f, 0.7350710320525575f,
    0.5298579358948849f, 0.3333333333333333f, 0.1012865073234563f, 0.4493567463382718f, 0.4493567463382718f,
    0.4701420641051151f, 0.2649289679474425f, 0.2649289679474425f};

// ----------------------------------------------------------- FP32 pieces --
// sqrt for arguments known to be positive and normal (far-field distances):
// r2 * rsqrt(r2), within 2 ulp.
__device__ __forceinline__ float sqrt_pos(float r2) { return r2 * rsqrtf(r2); }

// Lambda of an edge of length L whose end points lie at distances d1, d2
// from the station: the line integral of 1/r along the edge,
//   Lambda = log((d1 + d2 + L) / (d1 + d2 - L)) = 2 atanh(v),  v = L / (d1 + d2),
// equal to the reference's oriented form log((s2 + d2) / (s1 + d1)) because
// d2^2 - d1^2 = s2^2 - s1^2 along the edge's line.  Away from the edge (every
// FP32 pair) d1 + d2 - L does not cancel.  For v <= 0.2 the series
// 2 (v + v^3/3 + ... + v^9/9) (Abramowitz & Stegun 4.1.28), whose first
// omitted term is below 2e-9 v, else log1pf(2v / (1 - v)).  The arguments are
// bounded away from zero and overflow, so the 2-ulp quotient is used.
// atanh(v) for 0 <= v <= 0.2 by the series above (Lambda = 2 atanh(v)).
__device__ __forceinline__ float atanh_series(float v) {
    const float v2 = v * v;
    const float p = fmaf(v2, fmaf(v2, fmaf(v2, fmaf(v2, 1.f / 9.f, 1.f / 7.f), 1.f / 5.f), 1.f / 3.f), 1.f);
    return v * p;
}

__device__ __forceinline__ float lam_f32(float d1, float d2, float L) {
    const float v = __fdividef(L, d1 + d2);
    if (v <= 0.2f) return 2.f * atanh_series(v);
    return log1pf(__fdividef(2.f * v, 1.f - v));
}

// atan(t) for |t| <= 1/8: the Maclaurin series through t^9 (Abramowitz &
// Stegun 4.4.42; first omitted term below 1e-10 t).
__device__ __forceinline__ float atan_series(float t) {
    const float t2 = t * t;
    const float p = fmaf(t2, fmaf(t2, fmaf(t2, fmaf(t2, 1.f / 9.f, -1.f / 7.f), 1.f / 5.f), -1.f / 3.f), 1.f);
    return t * p;
}

// atan2(y, x); for x > 0 and |y| <= x / 8 (every far pair's solid angle)
// atan_series(y / x), else atan2f.
__device__ __forceinline__ float atan2_far(float y, float x) {
    if (x > 0.f && fabsf(y) <= 0.125f * x) return atan_series(__fdividef(y, x));
    return atan2f(y, x);
}

// True when a far pair lies inside both series' ranges on all four terms:
// the solid angle's atan2(ny, den) (den > 0, |ny| <= den / 8) and the three
// edges' atanh (v_i <= 0.2).  Far pairs practically always do, so one test
// replaces four per-term branches; a pair that fails it takes atan2_far /
// lam_f32, which select per term, and both routes give the same bits.
__device__ __forceinline__ bool far_series_ok(float ny, float den, float v0, float v1, float v2) {
    return den > 0.f && fabsf(ny) <= 0.125f * den && fmaxf(v0, fmaxf(v1, v2)) <= 0.2f;
}

// Near pair in FP64, local frame: solidAngle's branch semantics, Lambda in
// the symmetric form (lambda_sym: the reference's value except exactly on an
// edge's line beyond its end, where the reference's branch gives 0).  Returns
// the gz and TMI contributions.  s: the facet's constants, (x, y, z) the
// station in its frame.
__device__ __noinline__ double2 pair_near_f64_close(const double* __restrict__ s, double x, double y, double z) {
    const double L0 = s[MC_L0], cx = s[MC_CX], cy = s[MC_CY];
    const double rbx = L0 - x, rcx = cx - x, rcy = cy - y, z2 = z * z;
    const double la = sqrt(x * x + y * y + z2), lb = sqrt(rbx * rbx + y * y + z2), lc = sqrt(rcx * rcx + rcy * rcy + z2);
    const double h = -z;
    double om = 0.0;
    if (!(la < kEps || lb < kEps || lc < kEps)) {
        double den = la * lb * lc + (-x * rbx + y * y + z2) * lc + (-x * rcx - y * rcy + z2) * lb +
                     (rbx * rcx - y * rcy + z2) * la;
        om = 2.0 * atan2(h * (L0 * cy), den);
    }
    bool live;
    const double lam0 = (L0 < kEps) ? 0.0 : lambda_sym(la, lb, L0, &live);
    const double e1x = s[MC_E1X], e1y = s[MC_E1Y], e2x = s[MC_E2X], e2y = s[MC_E2Y];
    const double lam1 = (s[MC_L1] < kEps) ? 0.0 : lambda_sym(lb, lc, s[MC_L1], &live);
    const double lam2 = (s[MC_L2] < kEps) ? 0.0 : lambda_sym(lc, la, s[MC_L2], &live);
    // d_perp_i = -(r1 . perp_i), perp_i = z x e_i = (-e_y, e_x, 0)
    const double dp0 = y, dp1 = rbx * e1y + y * e1x, dp2 = rcx * e2y - rcy * e2x;
    return make_double2(s[MC_SGZ] * (dp0 * lam0 + dp1 * lam1 + dp2 * lam2 - h * om),
                        s[MC_MF] * om + s[MC_MT0] * lam0 + s[MC_MT1] * lam1 + s[MC_MT2] * lam2);
}

// The same, by polynomials where every L / (d1 + d2) is below 1/2 (see
// pair_forward_fp64); adds the gz and TMI contributions.  About 3 % of the
// mixed forward's pairs come here, and through the library functions they
// cost four times a far pair: 19,076 facets x 4,096 stations 441 us with
// those, 424 us without (13,388 facets x 1,036 and 7,575 stations: 320, 300 us a launch).
__device__ __forceinline__ void pair_near_f64(const double* __restrict__ s, d3 o, double* gz, double* tmi) {
    const double dx = o.x - s[MC_AX], dy = o.y - s[MC_AY], dz = o.z - s[MC_AZ];
    const double x = dx * s[MC_XX] + dy * s[MC_XY] + dz * s[MC_XZ];
    const double y = dx * s[MC_YX] + dy * s[MC_YY] + dz * s[MC_YZ];
    const double z = dx * s[MC_ZX] + dy * s[MC_ZY] + dz * s[MC_ZZ];
    const double L0 = s[MC_L0], cx = s[MC_CX], cy = s[MC_CY], L1 = s[MC_L1], L2 = s[MC_L2];
    const double rbx = L0 - x, rcx = cx - x, rcy = cy - y;
    const double z2 = z * z, yz2 = fma(y, y, z2);
    const double a2 = fma(x, x, yz2), b2 = fma(rbx, rbx, yz2), c2 = fma(rcx, rcx, fma(rcy, rcy, z2));
    const double la = sqrt_pos64(a2), lb = sqrt_pos64(b2), lc = sqrt_pos64(c2);
    const double v0 = L0 * rcp_pos64(la + lb), v1 = L1 * rcp_pos64(lb + lc), v2 = L2 * rcp_pos64(lc + la);
    if (!(max_ratio_hi(v0, v1, v2) < 0x3fe00000u)) {
        const double2 r = pair_near_f64_close(s, x, y, z);
        *gz += r.x;
        *tmi += r.y;
        return;
    }
    // ra . rb etc. in the facet's frame
    const double dab = fma(-x, rbx, yz2), u = fma(-y, rcy, z2), dac = fma(-x, rcx, u), dbc = fma(rbx, rcx, u);
    const double den = fma(la * lb, lc, fma(dab, lc, fma(dac, lb, dbc * la)));
    const double om = atan_poly64(-z * (L0 * cy) * rcp_pos64(den));
    const double l0 = atanh_poly64(v0), l1 = atanh_poly64(v1), l2 = atanh_poly64(v2);  // Lambda / 2
    const double dp1 = fma(rbx, s[MC_E1Y], y * s[MC_E1X]), dp2 = fma(rcx, s[MC_E2Y], -rcy * s[MC_E2X]);
    *gz += 2.0 * s[MC_SGZ] * fma(y, l0, fma(dp1, l1, fma(dp2, l2, z * om)));
    *tmi += 2.0 * fma(s[MC_MF], om, fma(s[MC_MT0], l0, fma(s[MC_MT1], l1, s[MC_MT2] * l2)));
}

// Paired FP32 (two independent results per instruction, sm_100): each half is
// rounded as the scalar operation.
__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }

// ---------------------------------------------------- far-field gradient --
// Sums v[0..31] over the warp, transposed: on return lane L holds the warp
// total of v[L] in v[0] (31 shuffles for 32 sums instead of 32 x 5).
__device__ __forceinline__ float warp_transpose_sum32(float (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
        const bool upper = (lane & step) != 0;
#pragma unroll
        for (int i = 0; i < step; ++i) {
            const float send = upper ? v[i] : v[i + step];
            const float keep = upper ? v[i + step] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, step);
        }
    }
    return v[0];
}

// Class of a (facet, tile) in the far-field gradient: 0 near (the FP64
// kernel's), 1 far (6-point rule), 2 beyond 4 tau x size (3-point rule).
// The near / far decision is tile_far's, operation for operation.
__device__ __forceinline__ int tile_gradient_class(const FarKey& k, const double* __restrict__ bbox) {
    if (k.th2 < 0.0) return 0;
    const double d0 = fmax(0.0, fmax(__dadd_rn(bbox[0], -k.c0), __dadd_rn(k.c0, -bbox[3])));
    const double d1 = fmax(0.0, fmax(__dadd_rn(bbox[1], -k.c1), __dadd_rn(k.c1, -bbox[4])));
    const double d2 = fmax(0.0, fmax(__dadd_rn(bbox[2], -k.c2), __dadd_rn(k.c2, -bbox[5])));
    const double dd = __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2));
    return dd >= __dmul_rn(16.0, k.th2) ? 2 : (dd >= k.th2 ? 1 : 0);
}

constexpr int kFarFlushTiles = 4;  // far tiles summed per lane in FP32 between warp reductions

// Far-field objective gradient in FP32: one warp per facet, lanes over the
// stations of the facet's far tiles (exactly the tiles k_gradient_warp_fp64
// leaves out: both classify with facet_far_key / tile_far).  gz by Dunavant's
// 6-point rule, the 3-point rule beyond 4 tau x size (tile_gradient_class).
//  * gz: I = A sum_q w_q / r_q, so
//      sum_s G0 dI/dv = (dA/dv) Q0 - A sum_q beta_qv D_q,
//    Q0 = sum_s G0 sum_q w_q / r_q, D_q = sum_s G0 w_q (p_q - o) / r_q^3
//    (G0 = gravity adjoint x group scale, beta_qv = barycentric weight of
//    point q on vertex v; n_z enters at the end, its own derivative through
//    the shared finalisation);
//  * TMI: the closed-form d Omega / dv and d Lambda / dv of the FP64 kernel,
//    in its per-edge form (pair_gradient_fp64).
// Each lane sums up to kFarFlushTiles tiles (8 stations) in FP32; the 32
// sums are then reduced across the warp in one transposed pass and lane k
// adds sum k to its FP64 total (one per quadrature rule).  Lane 0 gathers the
// totals, forms the facet accumulators in FP64 and finalises.  Facet list and
// station chunks as in k_gradient_warp_fp64; part layout [chunk][9][T].
// Sums: 0-5, 6-11, 12-17 x, y, z of D_q; 18 Q0; 19-21, 22-24, 25-27 TMI vertex
// terms of a, b, c; 28 sum Ts Omega / 2; 29-31 sum Ts Lambda_i / 2.
// SHORT (tau >= 3): pair_far_f32's bounds on e and t hold, so that the series
// need no fall-back to library functions: through the seventh power beyond
// 4 tau x size (the omitted terms are below 2e-12), through the ninth nearer,
// and through the thirteenth for the few pairs with an e above 0.2.
//
// Bound by instruction issue and fixed latencies (62 % of the issue slots at
// 16 warps per SM).  The quadrature points, the series (three atanh
// and one atan) and edges 1 and 2 run in pairs through the sm_100 paired FP32
// instructions; pairing within one (station, facet) needs no more registers
// than the scalar form, where pairing two stations does.  The vertex sums keep
// the scalar form's order of additions.  With the adjoints rounded once per
// station, no range test with library fall-backs and no branch on a
// lane's adjoints: 250 warp instructions per 32 pairs instead of about 390,
// both gradient kernels of a 32-body batch (1.29e9 pairs) 18.3 -> 14.6 ms.
// Four CTAs per SM (128 registers, some spill): three without spill 5 %
// slower, five 5 %; the facet frame or points in shared memory instead of
// registers 2 %; the flush through shared memory instead of shuffles equal.
template <bool SHORT>
__global__ void __launch_bounds__(128, 4) k_gradient_warp_far32(
    int T, const double* __restrict__ gc, int S, const double* __restrict__ sta, const float* __restrict__ adj_g,
    const float* __restrict__ adj_t, const double* __restrict__ tile_box, const int16_t* __restrict__ face_group,
    const GroupConst* __restrict__ groups, d3 fdir, double tau, const int32_t* __restrict__ facets, int nfacets,
    int tiles_per_chunk, const int32_t* __restrict__ grp_sta_off, const int32_t* __restrict__ grp_tile_off,
    double* __restrict__ part) {
    const int lane = threadIdx.x & 31;
    const int w = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
    if (w >= nfacets) return;  // warp-uniform
    const int f = facets[w], grp = face_group[f];
    if (grp_sta_off) {  // batched bodies: only the facet's own body's stations
        const int sb = grp_sta_off[grp];
        S = grp_sta_off[grp + 1] - sb;
        sta += 3 * (size_t)sb;
        if (adj_g) adj_g += sb;
        if (adj_t) adj_t += sb;
        tile_box += 6 * (size_t)grp_tile_off[grp];
    } else {
        if (adj_g) adj_g += (size_t)grp * S;
        if (adj_t) adj_t += (size_t)grp * S;
    }
    // this chunk's station tiles
    const int ntiles_all = (S + kStationTile - 1) / kStationTile;
    const int tbeg = blockIdx.y * tiles_per_chunk, ntiles = min(ntiles_all, tbeg + tiles_per_chunk);
    part += (size_t)blockIdx.y * 9 * T;
    __shared__ double totals[4][2][32];  // per warp: six-point rule, three-point rule
    bool active, any = false;
    double tot = 0.0, tot3 = 0.0;
    {
        double C[NGC];
#pragma unroll
        for (int k = 0; k < NGC; ++k) C[k] = __ldg(&gc[(size_t)k * T + f]);
        active = facet_grad_active(C);
        if (active) {
            const float L0 = (float)C[GC_L0], cx = (float)C[GC_CX], cy = (float)C[GC_CY];
            const float L1 = (float)C[GC_L1], L2 = (float)C[GC_L2];
            const float2 ex = make_float2((float)C[GC_E1X], (float)C[GC_E2X]),  // edges 1 and 2
                         ey = make_float2((float)C[GC_E1Y], (float)C[GC_E2Y]);
            const float rx0 = (float)C[GC_XX], rx1 = (float)C[GC_XY], rx2 = (float)C[GC_XZ];
            const float ry0 = (float)C[GC_YX], ry1 = (float)C[GC_YY], ry2 = (float)C[GC_YZ];
            const float mf = (float)C[GC_MF], mt0 = (float)C[GC_MT0];
            const float2 mt = make_float2((float)C[GC_MT1], (float)C[GC_MT2]);
            const float A2 = L0 * cy;
            const double ax = C[GC_AX], ay = C[GC_AY], az = C[GC_AZ];
            const double zx = C[GC_ZX], zy = C[GC_ZY], zz = C[GC_ZZ];
            float2 qx[3], qy[3];  // points 2p, 2p + 1
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                qx[p] = make_float2(kDun6Bb[2 * p] * L0 + kDun6Bc[2 * p] * cx,
                                    kDun6Bb[2 * p + 1] * L0 + kDun6Bc[2 * p + 1] * cx);
                qy[p] = make_float2(kDun6Bc[2 * p] * cy, kDun6Bc[2 * p + 1] * cy);
            }
            const float2 zero = make_float2(0.f, 0.f);
            float q0 = 0.f;
            float2 dqx[3], dqy[3], dqz[3];
            // bc.x, bc.y: sums of vertices b and c; ca.y: of a.  ca.x stays zero: it pads the
            // flush, where c's sum is bc.y + ca.x
            float2 bcx = zero, bcy = zero, bcz = zero, cax = zero, cay = zero, caz = zero;
            float2 am01 = zero, am2f = zero;  // sums of Ts Lambda_{0,1} / 2; Ts Lambda_2 / 2, Ts Omega / 2
#pragma unroll
            for (int p = 0; p < 3; ++p) dqx[p] = dqy[p] = dqz[p] = zero;
            int pending = 0, rule = 0;  // rule of the pending point sums: 0 six-point, 1 three-point
            auto flush = [&]() {
                float v[32] = {dqx[0].x, dqx[0].y, dqx[1].x, dqx[1].y, dqx[2].x, dqx[2].y,
                               dqy[0].x, dqy[0].y, dqy[1].x, dqy[1].y, dqy[2].x, dqy[2].y,
                               dqz[0].x, dqz[0].y, dqz[1].x, dqz[1].y, dqz[2].x, dqz[2].y,
                               q0, cax.y, cay.y, caz.y, bcx.x, bcy.x, bcz.x,
                               bcx.y + cax.x, bcy.y + cay.x, bcz.y + caz.x, am2f.y, am01.x, am01.y, am2f.x};
                const double sum = (double)warp_transpose_sum32(v);
                if (rule) tot3 += sum;
                else tot += sum;
                q0 = 0.f;
                bcx = bcy = bcz = cax = cay = caz = am01 = am2f = zero;
#pragma unroll
                for (int p = 0; p < 3; ++p) dqx[p] = dqy[p] = dqz[p] = zero;
            };
            const bool doG = adj_g && C[GC_GS] != 0.0, doT = adj_t && C[GC_MS] != 0.0;
            const FarKey key = facet_far_key(C, tau);
            for (int t0 = tbeg; t0 < ntiles; t0 += 32) {
                const int t = t0 + lane;
                const int cls = t < ntiles ? tile_gradient_class(key, tile_box + 6 * (size_t)t) : 0;
                unsigned m = __ballot_sync(0xffffffffu, cls != 0);
                const unsigned mv = __ballot_sync(0xffffffffu, cls == 2);
                any |= m != 0;
                while (m) {
                    const int b = __ffs(m) - 1;
                    m &= m - 1;
                    const int r = (mv >> b) & 1u;  // warp-uniform
                    if (pending && r != rule) {  // the pending sums belong to the other rule
                        flush();
                        pending = 0;
                    }
                    rule = r;
                    const bool brief = SHORT && r;
                    const int s0 = (t0 + b) * kStationTile;
#pragma unroll
                    for (int k = 0; k < kStationTile; k += 32) {
                        // lanes past the last station repeat it with zero adjoints
                        const int j = min(s0 + k + lane, S - 1);
                        const bool in = s0 + k + lane < S;
                        const float G0 = doG && in ? adj_g[j] : 0.f, Ts = doT && in ? adj_t[j] : 0.f;
                        const double ox = sta[3 * j], oy = sta[3 * j + 1], oz = sta[3 * j + 2];
                        const double ddx = ox - ax, ddy = oy - ay, ddz = oz - az;
                        const float dx = (float)ddx, dy = (float)ddy, dzf = (float)ddz;
                        const float x = fmaf(dx, rx0, fmaf(dy, rx1, dzf * rx2));
                        const float y = fmaf(dx, ry0, fmaf(dy, ry1, dzf * ry2));
                        const float z = (float)(ddx * zx + ddy * zy + ddz * zz);
                        const float z2 = z * z;
                        const float2 zz2 = dup2(z2), nx = dup2(-x), ny = dup2(-y), nz = dup2(-z);
                        if (doG && r) {  // beyond 4 tau: the 3-point rule, weights 1/3
                            // points 0 and 1 paired, point 2 alone
                            const float2 px = fma2(make_float2(kTri3Bb[0], kTri3Bb[1]), dup2(L0),
                                                   fma2(make_float2(kTri3Bc[0], kTri3Bc[1]), dup2(cx), nx));
                            const float2 py = fma2(make_float2(kTri3Bc[0], kTri3Bc[1]), dup2(cy), ny);
                            const float2 r2 = fma2(px, px, fma2(py, py, zz2));
                            const float2 rs = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
                            const float2 w = mul2(dup2(1.f / 3.f), rs);
                            const float2 g3 = mul2(mul2(mul2(dup2(G0), w), rs), rs);
                            dqx[0] = fma2(g3, px, dqx[0]);
                            dqy[0] = fma2(g3, py, dqy[0]);
                            dqz[0] = fma2(g3, nz, dqz[0]);
                            const float px2 = fmaf(kTri3Bb[2], L0, fmaf(kTri3Bc[2], cx, -x));
                            const float py2 = fmaf(kTri3Bc[2], cy, -y);
                            const float rs2 = rsqrtf(fmaf(px2, px2, fmaf(py2, py2, z2)));
                            const float w2 = __fmul_rn(1.f / 3.f, rs2), h3 = G0 * w2 * rs2 * rs2;
                            dqx[1].x = fmaf(h3, px2, dqx[1].x);
                            dqy[1].x = fmaf(h3, py2, dqy[1].x);
                            dqz[1].x = fmaf(h3, -z, dqz[1].x);
                            q0 = fmaf(G0, __fadd_rn(__fadd_rn(w.x, w.y), w2), q0);
                        } else if (doG) {
                            float sw = 0.f;
#pragma unroll
                            for (int p = 0; p < 3; ++p) {
                                const float2 px = add2(qx[p], nx), py = add2(qy[p], ny);
                                const float2 r2 = fma2(px, px, fma2(py, py, zz2));
                                const float2 rs = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
                                const float2 w = mul2(make_float2(kDun6W[2 * p], kDun6W[2 * p + 1]), rs);
                                sw = __fadd_rn(sw, w.x);
                                sw = __fadd_rn(sw, w.y);
                                const float2 g3 = mul2(mul2(mul2(dup2(G0), w), rs), rs);
                                dqx[p] = fma2(g3, px, dqx[p]);
                                dqy[p] = fma2(g3, py, dqy[p]);
                                dqz[p] = fma2(g3, nz, dqz[p]);
                            }
                            q0 = fmaf(G0, sw, q0);
                        }
                        if (doT) {
                            const float2 rx = add2(make_float2(L0, cx), nx);   // b, c
                            const float2 ry = make_float2(-y, cy - y);         // b, c
                            const float2 yz = fma2(ry, ry, zz2);
                            const float2 bc2 = fma2(rx, rx, yz);
                            const float la2 = fmaf(x, x, yz.x);
                            const float la = sqrt_pos(la2);
                            const float2 lbc = mul2(bc2, make_float2(rsqrtf(bc2.x), rsqrtf(bc2.y)));
                            const float lb = lbc.x, lc = lbc.y;
                            const float ia = __fdividef(1.f, la), ib = __fdividef(1.f, lb), ic = __fdividef(1.f, lc);
                            const float2 ibc = make_float2(ib, ic), ica = make_float2(ic, ia);
                            const float u = fmaf(ry.x, ry.y, z2);
                            const float2 dad = fma2(nx, rx, make_float2(yz.x, u));  // ra.rb, ra.rc
                            const float dab = dad.x, dac = dad.y, dbc = fmaf(rx.x, rx.y, u);
                            const float den = fmaf(dbc, la, fmaf(dac, lb, fmaf(la * lb, lc, dab * lc)));
                            const float nyv = -z * A2;
                            const float t = __fdividef(nyv, den);
                            const float2 ea = make_float2(__fdividef(L0, la + lb), __fdividef(L1, lb + lc)),
                                         eb = make_float2(__fdividef(L2, lc + la), t);
                            float2 la01, la2f;  // (Lambda_0, Lambda_1) / 2, (Lambda_2, Omega) / 2
                            const float2 wa = mul2(ea, ea), wb = mul2(eb, eb);
                            const float2 s3 = make_float2(1.f / 3.f, -1.f / 3.f), s7 = make_float2(1.f / 7.f, -1.f / 7.f);
                            if (brief) {  // through e^7 and t^7; e < 0.045, |t| < 0.002
                                la01 = fma2(wa, fma2(wa, dup2(1.f / 7.f), dup2(0.2f)), dup2(1.f / 3.f));
                                la2f = fma2(wb, fma2(wb, s7, dup2(0.2f)), s3);
                            } else {
                                la01 = fma2(wa, fma2(wa, fma2(wa, dup2(1.f / 9.f), dup2(1.f / 7.f)), dup2(0.2f)), dup2(1.f / 3.f));
                                la2f = fma2(wb, fma2(wb, fma2(wb, dup2(1.f / 9.f), s7), dup2(0.2f)), s3);
                            }
                            if (SHORT && !brief && fmaxf(ea.x, fmaxf(ea.y, eb.x)) > 0.2f) {  // e < 0.215: through e^13
                                const float2 c = make_float2(1.f / 11.f, 1.f / 13.f);
                                la01 = fma2(wa, fma2(wa, fma2(wa, fma2(wa, fma2(wa, dup2(c.y), dup2(c.x)), dup2(1.f / 9.f)),
                                                              dup2(1.f / 7.f)), dup2(0.2f)), dup2(1.f / 3.f));
                                la2f.x = fmaf(wb.x, fmaf(wb.x, fmaf(wb.x, fmaf(wb.x, fmaf(wb.x, c.y, c.x), 1.f / 9.f),
                                                                    1.f / 7.f), 0.2f), 1.f / 3.f);
                            }
                            la01 = mul2(ea, fma2(wa, la01, dup2(1.f)));
                            la2f = mul2(eb, fma2(wb, la2f, dup2(1.f)));
                            if (!SHORT && !far_series_ok(nyv, den, ea.x, ea.y, eb.x)) {
                                la01 = make_float2(0.5f * lam_f32(la, lb, L0), 0.5f * lam_f32(lb, lc, L1));
                                la2f = make_float2(0.5f * lam_f32(lc, la, L2), atan2_far(nyv, den));
                            }
                            am01 = fma2(dup2(Ts), la01, am01);
                            am2f = fma2(dup2(Ts), la2f, am2f);
                            const float kom = Ts * mf;
                            // edge (p1 -> p2): W = L / (d1 d2 + r1.r2), q = r1 - s1 e, Z = e x r1,
                            // P = W (kom Z - kl q); p1 += (P - kl e)/d1, p2 += (P + kl e)/d2.
                            {  // edge 0: e = (1, 0), so q = (0, -y, -z) and Z = (0, z, -y)
                                const float kl = Ts * mt0, W = __fdividef(L0, fmaf(la, lb, dab));
                                const float Py = W * fmaf(kom, z, kl * y), Pz = W * fmaf(kom, -y, kl * z);
                                cax.y = fmaf(-kl, ia, cax.y);
                                cay.y = fmaf(Py, ia, cay.y);
                                caz.y = fmaf(Pz, ia, caz.y);
                                bcx.x = fmaf(kl, ib, bcx.x);
                                bcy.x = fmaf(Py, ib, bcy.x);
                                bcz.x = fmaf(Pz, ib, bcz.x);
                            }
                            // edges 1 (b->c) and 2 (c->a), paired
                            const float2 kl = mul2(dup2(Ts), mt), nkl = neg2(kl), kom2 = dup2(kom);
                            const float2 W = make_float2(__fdividef(L1, fmaf(lb, lc, dbc)), __fdividef(L2, fmaf(lc, la, dac)));
                            const float2 ns = neg2(fma2(rx, ex, mul2(ry, ey)));  // -(r1 . e)
                            const float2 kqx = mul2(nkl, fma2(ns, ex, rx)), kqy = mul2(nkl, fma2(ns, ey, ry));
                            const float2 Px = mul2(W, fma2(kom2, mul2(ey, nz), kqx)),
                                         Py = mul2(W, fma2(kom2, mul2(neg2(ex), nz), kqy)),
                                         Pz = mul2(W, fma2(kom2, fma2(ex, ry, mul2(neg2(ey), rx)), mul2(nkl, nz)));
                            const float2 t2x=fma2(kl, ex, Px), t2y=fma2(kl, ey, Py);
                            cax.y = fmaf(t2x.y, ia, cax.y); cay.y = fmaf(t2y.y, ia, cay.y); caz.y = fmaf(Pz.y, ia, caz.y);
                            bcx.y = fmaf(t2x.x, ic, bcx.y); bcy.y = fmaf(t2y.x, ic, bcy.y); bcz.y = fmaf(Pz.x, ic, bcz.y);
                            bcx = fma2(fma2(nkl, ex, Px), ibc, bcx);
                            bcy = fma2(fma2(nkl, ey, Py), ibc, bcy);
                            bcz = fma2(Pz, ibc, bcz);
                        }
                    }
                    if (++pending == kFarFlushTiles) {
                        flush();
                        pending = 0;
                    }
                }
            }
            if (pending) flush();
        }
    }
    double outv[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (active && any) {  // warp-uniform
        double(*v)[32] = totals[threadIdx.x >> 5];
        v[0][lane] = tot;
        v[1][lane] = tot3;
        __syncwarp();
        if (lane == 0) {
            double C[NGC];
#pragma unroll
            for (int k = 0; k < NGC; ++k) C[k] = __ldcg(&gc[(size_t)k * T + f]);
            const double nz = C[GC_ZZ], L0 = C[GC_L0], cx = C[GC_CX], cy = C[GC_CY];
            const double Ar = 0.5 * L0 * cy, q0 = v[0][18] + v[1][18];
            d3 Da = mk3(0, 0, 0), Db = Da, Dc = Da;  // sum_q beta_q{a,b,c} D_q over both rules
            for (int q = 0; q < 9; ++q) {
                const int rl = q >= 6, k = rl ? q - 6 : q;
                const double bb = rl ? kTri3Bb[k] : kDun6Bb[k], bc = rl ? kTri3Bc[k] : kDun6Bc[k];
                const d3 D = mk3(v[rl][k], v[rl][6 + k], v[rl][12 + k]);
                Da = Da + D * (1.0 - bb - bc);
                Db = Db + D * bb;
                Dc = Dc + D * bc;
            }
            auto both = [&](int k) { return v[0][k] + v[1][k]; };
            // dA/da = (-cy, cx - L0, 0)/2, dA/db = (cy, -cx, 0)/2, dA/dc = (0, L0, 0)/2
            GradAcc A;
            grad_acc_zero(A);
            A.va = mk3(nz * (-0.5 * cy * q0 - Ar * Da.x) + both(19), nz * (0.5 * (cx - L0) * q0 - Ar * Da.y) + both(20),
                       nz * (-Ar * Da.z) + both(21));
            A.vb = mk3(nz * (0.5 * cy * q0 - Ar * Db.x) + both(22), nz * (-0.5 * cx * q0 - Ar * Db.y) + both(23),
                       nz * (-Ar * Db.z) + both(24));
            A.vc = mk3(nz * (-Ar * Dc.x) + both(25), nz * (0.5 * L0 * q0 - Ar * Dc.y) + both(26),
                       nz * (-Ar * Dc.z) + both(27));
            A.ai = Ar * q0;
            A.amf = 2.0 * both(28);
            for (int i = 0; i < 3; ++i) A.amt[i] = 2.0 * both(29 + i);
            grad_finalize(C, A, groups[grp], fdir, outv);
        }
    }
    if (lane == 0)
        for (int k = 0; k < 9; ++k) part[(size_t)k * T + f] = outv[k];
}

// Per station: sum of chunk partials (facet scales are already applied).
// Blocks of 32 stations x 8 chunk lanes: lane y sums chunks y, y+8, ...
// (coalesced over stations), then the 8 lane sums are added in lane order.
// With block_nch, station s sums block_nch[s / block] chunks (the persistent
// patch forward), else nchunks.
__global__ void __launch_bounds__(256) k_forward_reduce_mixed(int S, int nchunks, const double* __restrict__ part_gz,
                                                              const double* __restrict__ part_tmi,
                                                              double* __restrict__ gz, double* __restrict__ tmi,
                                                              const int32_t* __restrict__ block_nch = nullptr,
                                                              int block = 1) {
    __shared__ double sg[8][33], st[8][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int s = blockIdx.x * 32 + tx;
    double g = 0.0, t = 0.0;
    if (block_nch && s < S) nchunks = block_nch[s / block];
    if (s < S) {
        if (part_gz) g = strided_sum8(ty, nchunks, g, [&](int c) { return part_gz[(size_t)c * S + s]; });
        if (part_tmi) t = strided_sum8(ty, nchunks, t, [&](int c) { return part_tmi[(size_t)c * S + s]; });
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

}  // namespace litho_b200
