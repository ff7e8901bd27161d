// hbg_statics.cu -- panel geometry and the frequency-independent influence data (FP64).
//
// Geometry: one thread per panel (geometry.rs:120-199 make_panel, panel_integrals.rs:145-217
// make_panel_geom).  Statics: one thread per (row k, panel j) pair computes the Rankine source and
// dipole of 1/r + 1/r' (finite depth: the six image terms) by the closed forms of
// panel_integrals.rs:226-275 and the log-singularity corrections dl, dd of lo_static.rs:99-117.
// Pairs whose log integral needs the adaptive rule (image within 2 radii and less than half a
// radius above the panel, panel_integrals.rs:407-449) are appended to a worklist and integrated by
// a second kernel with an explicit depth-first stack, in the reference's cell order.
//
// Layout: statics planes [4][N*N] (rs, rd, dl, dd), entry (k, j) at k + j*N (column-major, the
// layout of the matrices the assembly writes), so a warp of consecutive rows k writes coalesced.
//
// This file is its own translation unit, compiled without floating-point contraction (-fmad=false):
// the reference picks closed forms, Gauss orders and the adaptive rule by thresholds on geometric
// ratios (distance over panel radius, clearance, log_pair), which regular meshes put exactly on
// the thresholds; with the same IEEE operations in the same order as the reference, every such
// decision (and every geometric quantity) is the reference's to the bit.
#include "hbg_device.cuh"
#include "hbg_internal.h"

namespace hbg {

constexpr double COINCIDENCE_TOL = 1e-6;
constexpr double CONVEXITY_TOL = 1e-6;

__device__ __forceinline__ void bilinear(const double vt[4][3], double u, double v, double* x, double& jac) {
    double n0 = 0.25 * (1.0 - u) * (1.0 - v), n1 = 0.25 * (1.0 + u) * (1.0 - v);
    double n2 = 0.25 * (1.0 + u) * (1.0 + v), n3 = 0.25 * (1.0 - u) * (1.0 + v);
    double xu[3], xv[3], cr[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        x[d] = n0 * vt[0][d] + n1 * vt[1][d] + n2 * vt[2][d] + n3 * vt[3][d];
        xu[d] = (0.25 * (1.0 - v)) * (vt[1][d] - vt[0][d]) + (0.25 * (1.0 + v)) * (vt[2][d] - vt[3][d]);
        xv[d] = (0.25 * (1.0 - u)) * (vt[3][d] - vt[0][d]) + (0.25 * (1.0 + u)) * (vt[2][d] - vt[1][d]);
    }
    cross3(xu, xv, cr);
    jac = norm3(cr);
}

// ------------------------------------------------------------------ geometry
// The reference's production rule of the Rankine integrals (panel_integrals.rs:190-216, 288-363): per
// panel the float32 Gauss tiers of orders 3, 4, 5, 6 (points of the bilinear map relative to the
// centroid, weights scaled to the exact area), each block padded with zero weights to a multiple of 8:
// tier_len(t) points at tier_off(t), planes x, y, z, w of tier_len(t) floats each.
constexpr int TIER_FLOATS = 416;
static_assert(TIER_FLOATS == TIER_FLOATS_HOST, "the host's tier buffer size");
__device__ __forceinline__ int tier_off(int t) { return t == 0 ? 0 : t == 1 ? 64 : t == 2 ? 128 : 256; }
__device__ __forceinline__ int tier_len(int t) { return t <= 1 ? 16 : t == 2 ? 32 : 40; }

__global__ void k_panel_geometry(int N, const double* __restrict__ verts, const int32_t* __restrict__ kind,
                                 double* __restrict__ P, int32_t* __restrict__ bad, float* __restrict__ tiers,
                                 const int32_t* __restrict__ orig) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= N) return;
    double raw[4][3];
    bool ok = true;
    for (int i = 0; i < 4; i++)
        for (int d = 0; d < 3; d++) {
            raw[i][d] = verts[(size_t)j * 12 + 3 * i + d];
            ok = ok && isfinite(raw[i][d]);
        }
    auto fail = [&]() { atomicMin(bad, orig ? orig[j] : j); };  // the panel's index in the caller's order
    if (!ok) { fail(); return; }
    double t[3];
    double diameter = 0.0;
    for (int i = 0; i < 4; i++)
        for (int k = i + 1; k < 4; k++) {
            for (int d = 0; d < 3; d++) t[d] = raw[i][d] - raw[k][d];
            diameter = fmax(diameter, norm3(t));
        }
    if (diameter == 0.0) { fail(); return; }
    double tol = COINCIDENCE_TOL * diameter;
    int keep[4], m = 0;
    for (int i = 0; i < 4; i++) {
        for (int d = 0; d < 3; d++) t[d] = raw[i][d] - raw[(i + 1) % 4][d];
        if (norm3(t) > tol) keep[m++] = i;
    }
    if (m < 3) { fail(); return; }
    for (int a = 0; a < m; a++)
        for (int b = a + 1; b < m; b++) {
            for (int d = 0; d < 3; d++) t[d] = raw[keep[a]][d] - raw[keep[b]][d];
            if (norm3(t) <= tol) { fail(); return; }
        }
    double c[3], d1[3], d2[3], n[3];
    for (int d = 0; d < 3; d++) {
        c[d] = 0.25 * (raw[0][d] + raw[1][d] + raw[2][d] + raw[3][d]);
        d1[d] = raw[2][d] - raw[0][d];
        d2[d] = raw[3][d] - raw[1][d];
    }
    cross3(d1, d2, n);
    double nn = norm3(n);
    if (0.5 * nn <= COINCIDENCE_TOL * diameter * diameter) { fail(); return; }
    double inv = 1.0 / nn, nh[3] = {inv * n[0], inv * n[1], inv * n[2]};
    double q[4][3];
    for (int i = 0; i < 4; i++) {
        for (int d = 0; d < 3; d++) t[d] = raw[i][d] - c[d];
        double s = dot3(t, nh);
        for (int d = 0; d < 3; d++) q[i][d] = raw[i][d] - s * nh[d];
    }
    double poly[4][3];
    for (int a = 0; a < m; a++)
        for (int d = 0; d < 3; d++) poly[a][d] = q[keep[a]][d];
    for (int a = 0; a < m; a++) {
        double e1[3], e2[3], cr[3];
        for (int d = 0; d < 3; d++) {
            e1[d] = poly[(a + 1) % m][d] - poly[a][d];
            e2[d] = poly[(a + 2) % m][d] - poly[(a + 1) % m][d];
        }
        cross3(e1, e2, cr);
        double s = dot3(cr, nh) / (norm3(e1) * norm3(e2));
        if (!(s > CONVEXITY_TOL)) { fail(); return; }
    }
    double area = 0.0, mom[3] = {0, 0, 0};
    for (int a = 1; a < m - 1; a++) {
        double e1[3], e2[3], cr[3];
        for (int d = 0; d < 3; d++) {
            e1[d] = poly[a][d] - poly[0][d];
            e2[d] = poly[a + 1][d] - poly[0][d];
        }
        cross3(e1, e2, cr);
        double tt = 0.5 * dot3(cr, nh);
        area += tt;
        for (int d = 0; d < 3; d++) mom[d] += (tt / 3.0) * (poly[0][d] + poly[a][d] + poly[a + 1][d]);
    }
    double cent[3], normal[3] = {nh[0], nh[1], nh[2]};
    for (int d = 0; d < 3; d++) cent[d] = (1.0 / area) * mom[d];
    if (kind && kind[j] == 1) {
        // interior free surface: exactly in z = 0, normal +z (lo_geometry.rs:706-716)
        if (nh[2] < 0.0)
            for (int d = 0; d < 3; d++) {
                double s = q[1][d];
                q[1][d] = q[3][d];
                q[3][d] = s;
            }
        for (int i = 0; i < 4; i++) q[i][2] = 0.0;
        cent[2] = 0.0;
        normal[0] = 0.0;
        normal[1] = 0.0;
        normal[2] = 1.0;
    }
    auto W = [&](int plane, double val) { P[(size_t)plane * N + j] = val; };
    for (int d = 0; d < 3; d++) {
        W(P_C + d, cent[d]);
        W(P_N + d, normal[d]);
    }
    W(P_AREA, area);
    double diam = 0.0;
    for (int i = 0; i < 4; i++)
        for (int k = i + 1; k < 4; k++) {
            for (int d = 0; d < 3; d++) t[d] = q[i][d] - q[k][d];
            diam = fmax(diam, norm3(t));
        }
    double v[4][3] = {};
    int nv = 0;
    for (int i = 0; i < 4; i++) {
        for (int d = 0; d < 3; d++) t[d] = q[i][d] - q[(i + 1) % 4][d];
        if (norm3(t) > COINCIDENCE_TOL * diam) {
            for (int d = 0; d < 3; d++) v[nv][d] = q[i][d];
            nv++;
        }
    }
    double radius = 0.0;
    for (int i = 0; i < nv; i++) {
        for (int d = 0; d < 3; d++) t[d] = v[i][d] - cent[d];
        radius = fmax(radius, norm3(t));
    }
    W(P_RADIUS, radius);
    W(P_NV, (double)nv);
    for (int i = 0; i < 4; i++)
        for (int d = 0; d < 3; d++) W(P_V + 3 * i + d, v[i][d]);
    for (int e = 0; e < 4; e++) {
        double edge[3] = {0, 0, 0}, cr[3] = {0, 0, 0}, len = 0.0;
        if (e < nv) {
            for (int d = 0; d < 3; d++) edge[d] = v[(e + 1) % nv][d] - v[e][d];
            len = norm3(edge);
            cross3(edge, normal, cr);
            for (int d = 0; d < 3; d++) cr[d] *= 1.0 / len;
        }
        W(P_ELEN + e, len);
        for (int d = 0; d < 3; d++) W(P_EM + 3 * e + d, cr[d]);
    }
    double gw[9], sum = 0.0;
    for (int i = 0; i < 3; i++)
        for (int k = 0; k < 3; k++) {
            double x[3], jac;
            bilinear(q, c_glx[3][i], c_glx[3][k], x, jac);
            for (int d = 0; d < 3; d++) W(P_GX + 3 * (3 * i + k) + d, x[d]);
            gw[3 * i + k] = c_glw[3][i] * c_glw[3][k] * jac;
            sum += gw[3 * i + k];
        }
    for (int k = 0; k < 9; k++) W(P_GW + k, gw[k] * (area / sum));
    if (tiers) {
        float* tb = tiers + (size_t)j * TIER_FLOATS;
        for (int t = 0; t < 4; t++) {
            const int n = 3 + t, len = tier_len(t);
            float* b = tb + tier_off(t);
            double wsum = 0.0;
            for (int i = 0; i < n; i++)
                for (int k = 0; k < n; k++) {
                    double x[3], jac;
                    bilinear(q, c_glx[n][i], c_glx[n][k], x, jac);
                    wsum += c_glw[n][i] * c_glw[n][k] * jac;
                }
            for (int i = 0; i < n; i++)
                for (int k = 0; k < n; k++) {
                    double x[3], jac;
                    bilinear(q, c_glx[n][i], c_glx[n][k], x, jac);
                    const int e = i * n + k;
                    b[e] = (float)(x[0] - cent[0]);
                    b[len + e] = (float)(x[1] - cent[1]);
                    b[2 * len + e] = (float)(x[2] - cent[2]);
                    b[3 * len + e] = (float)(c_glw[n][i] * c_glw[n][k] * jac * area / wsum);
                }
            for (int e = n * n; e < len; e++) b[e] = b[len + e] = b[2 * len + e] = b[3 * len + e] = 0.f;
        }
    }
}

// ------------------------------------------------------------------ Rankine closed forms
struct PanelRegs {
    int nv;
    double c[3], n[3], area, radius;
    double v[4][3], em[4][3], elen[4];
};

__device__ __forceinline__ void load_panel(const PanelsView& pv, int j, PanelRegs& p) {
    p.nv = (int)pv.at(P_NV, j);
#pragma unroll
    for (int d = 0; d < 3; d++) {
        p.c[d] = pv.at(P_C + d, j);
        p.n[d] = pv.at(P_N + d, j);
    }
    p.area = pv.at(P_AREA, j);
    p.radius = pv.at(P_RADIUS, j);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        p.elen[i] = pv.at(P_ELEN + i, j);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            p.v[i][d] = pv.at(P_V + 3 * i + d, j);
            p.em[i][d] = pv.at(P_EM + 3 * i + d, j);
        }
    }
}

// panel_integrals.rs:226-275 (closed forms; beyond `far` radii the 3 x 3 rule: 1000 in the reference's
// double-precision mode, 12 in its production mode)
__device__ inline void rankine(const PanelsView& pv, int j, const PanelRegs& p, const double* x, double& S, double& D,
                               double far = 1000.0) {
    double rc[3] = {x[0] - p.c[0], x[1] - p.c[1], x[2] - p.c[2]};
    double dist = norm3(rc);
    if (dist > far * p.radius) {
        double s = 0.0, dd = 0.0;
        for (int k = 0; k < 9; k++) {
            double r[3];
            for (int d = 0; d < 3; d++) r[d] = x[d] - pv.at(P_GX + 3 * k + d, j);
            double ir = 1.0 / norm3(r), w = pv.at(P_GW + k, j);
            s += w * ir;
            dd += w * dot3(p.n, r) * ir * ir * ir;
        }
        S = s;
        D = dd;
        return;
    }
    double w = dot3(rc, p.n);
    int nv = p.nv;
    double av[4][3], r[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        for (int d = 0; d < 3; d++) av[i][d] = p.v[i][d] - x[d];
        r[i] = norm3(av[i]);
    }
    double omega = 0.0;
    if (fabs(w) > 1e-12 * p.radius) {
        for (int i = 1; i < nv - 1; i++) {
            double bc[3];
            cross3(av[i], av[i + 1], bc);
            double num = dot3(av[0], bc);
            double den = r[0] * r[i] * r[i + 1] + dot3(av[0], av[i]) * r[i + 1] + dot3(av[0], av[i + 1]) * r[i] +
                         dot3(av[i], av[i + 1]) * r[0];
            omega -= 2.0 * atan2(num, den);
        }
    }
    double s = 0.0;
    for (int e = 0; e < nv; e++) {
        int f = (e + 1) == nv ? 0 : e + 1;
        double d = dot3(av[e], p.em[e]);
        if (fabs(d) <= 1e-14 * p.radius) continue;
        double q = r[e] * r[f] + dot3(av[e], av[f]);
        if (!(q > 0.0)) continue;
        double sum = r[e] + r[f] + p.elen[e];
        s += d * log(sum * sum / (2.0 * q));
    }
    S = s - w * omega;
    D = omega;
}

__device__ __forceinline__ void psi_terms(const double* xi, const double* pp, const double* n, double& psi, double& dpsi) {
    double d[3] = {xi[0] - pp[0], xi[1] - pp[1], xi[2] - pp[2]};
    double R = norm3(d);
    double den = R - d[2];
    psi = log(den);
    dpsi = (dot3(d, n) / R - n[2]) / den;
}

__device__ __forceinline__ void panel_map(const PanelRegs& p, double m[4][3]) {
    for (int d = 0; d < 3; d++) {
        m[0][d] = p.v[0][d];
        m[1][d] = p.v[1][d];
        m[2][d] = p.v[2][d];
        m[3][d] = p.nv == 4 ? p.v[3][d] : p.v[2][d];
    }
}

// the Gauss order of the log integral by distance, 0 for the adaptive rule (panel_integrals.rs:407-432)
__device__ __forceinline__ int log_order(const PanelRegs& p, const double* image) {
    double t[3] = {image[0] - p.c[0], image[1] - p.c[1], image[2] - p.c[2]};
    double dist = norm3(t);
    double top = p.v[0][2];
    for (int i = 1; i < p.nv; i++) top = fmax(top, p.v[i][2]);
    double r = dist / p.radius;
    double clearance = (image[2] - top) / p.radius;
    if (clearance >= 0.5 || r >= 2.0) return r >= 6.0 ? 4 : r >= 3.0 ? 5 : r >= 2.0 ? 6 : r >= 1.5 ? 8 : r >= 1.0 ? 10 : 0;
    return 0;
}

// The points of the panel's order-4 rule (x, y, z and weight), formed once a panel: log_point4 of lane e < 16.
struct LogPoint {
    double x[3], w;
};
__device__ __forceinline__ LogPoint log_point4(const PanelRegs& p, int e) {
    double m[4][3], jac;
    panel_map(p, m);
    LogPoint q;
    bilinear(m, c_glx[4][e / 4], c_glx[4][e % 4], q.x, jac);
    q.w = c_glw[4][e / 4] * c_glw[4][e % 4] * jac;
    return q;
}
// log_gauss of order 4 on those points
__device__ __forceinline__ void log_gauss4(const LogPoint* lp, const PanelRegs& p, const double* image, double& L, double& Ld) {
    double l = 0.0, ld = 0.0;
#pragma unroll 2
    for (int e = 0; e < 16; e++) {
        double psi, dpsi;
        psi_terms(lp[e].x, image, p.n, psi, dpsi);
        l += lp[e].w * psi;
        ld += lp[e].w * dpsi;
    }
    L = l;
    Ld = ld;
}

// The Gauss rule of order n x n (5 to 10) at one image by a warp: the points spread over the lanes, the sums in every
// lane.  (A lane of its own for each image ran the orders of a warp's images one after another, up to
// 25 + 36 + 64 + 100 points of ~150 dependent FP64 instructions: 177 us for the whole of an 84-panel hull.)
__device__ __forceinline__ void log_gauss_warp(const PanelRegs& p, const double* image, int order, int lane, double& L,
                                               double& Ld) {
    double m[4][3];
    panel_map(p, m);
    double l = 0.0, ld = 0.0;
    for (int e = lane; e < order * order; e += 32) {
        const int i = e / order, j = e - i * order;
        double xi[3], jac, psi, dpsi;
        bilinear(m, c_glx[order][i], c_glx[order][j], xi, jac);
        psi_terms(xi, image, p.n, psi, dpsi);
        double ww = c_glw[order][i] * c_glw[order][j] * jac;
        l += ww * psi;
        ld += ww * dpsi;
    }
    for (int o = 16; o > 0; o >>= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, o);
        ld += __shfl_xor_sync(0xffffffffu, ld, o);
    }
    L = l;
    Ld = ld;
}

// ---- the mixed form's far-field shortcuts (its matrices are rounded to FP32 afterwards)
// A point farther than MIX_FAR panel radii from the panel: the Rankine integrals by the panel's 3 x 3
// Gauss rule (the rule the closed forms give way to beyond 1000 radii), in FP32 on FP64 differences.
// The rule's error falls as (radius / distance)^6, below FP32 rounding at 20 radii.
constexpr double MIX_FAR = 20.0;

// The images of a field point differ in z alone, so the horizontal differences of a Gauss point are formed once for
// all of them (bit i of any: some lane of the warp needs image i); the rule's points and weights in shared memory.
template <int NI>
__device__ __forceinline__ void rankine_gauss_f32(const double (*g)[3], const float* gw, const PanelRegs& p, const double* x,
                                                  const double (&z)[NI], unsigned any, double (&S)[NI], double (&D)[NI]) {
    const float n0 = (float)p.n[0], n1 = (float)p.n[1], n2 = (float)p.n[2];
    float s[NI], dd[NI];
#pragma unroll
    for (int i = 0; i < NI; i++) s[i] = dd[i] = 0.f;
#pragma unroll 3
    for (int k = 0; k < 9; k++) {
        const float r0 = (float)(x[0] - g[k][0]), r1 = (float)(x[1] - g[k][1]);
        const double gz = g[k][2];
        const float w = gw[k];
#pragma unroll
        for (int i = 0; i < NI; i++) {
            if (!(any >> i & 1)) continue;
            const float r2 = (float)(z[i] - gz);
            const float ir = rsqrtf(__fmaf_rn(r0, r0, __fmaf_rn(r1, r1, r2 * r2)));
            const float wi = w * ir;
            s[i] += wi;
            dd[i] = __fmaf_rn(wi * ir * ir, __fmaf_rn(n0, r0, __fmaf_rn(n1, r1, n2 * r2)), dd[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < NI; i++) S[i] = s[i], D[i] = dd[i];
}

// log_gauss with the integrand log(R - dz) and its normal derivative in FP32 (positions, weights and
// sums in FP64): R - dz = R + |dz| for an image above the panel, so no cancellation.
__device__ __forceinline__ void log_gauss4_f32(const LogPoint* lp, const PanelRegs& p, const double* image, double& L,
                                               double& Ld) {
    const float n0 = (float)p.n[0], n1 = (float)p.n[1], n2 = (float)p.n[2];
    double l = 0.0, ld = 0.0;
#pragma unroll 4
    for (int e = 0; e < 16; e++) {
        const double* xi = lp[e].x;
        const float d0 = (float)(xi[0] - image[0]), d1 = (float)(xi[1] - image[1]), d2 = (float)(xi[2] - image[2]);
        const float R = sqrtf(__fmaf_rn(d0, d0, __fmaf_rn(d1, d1, d2 * d2)));
        const float den = R - d2;
        const float psi = logf(den);
        const float dpsi = (__fmaf_rn(d0, n0, __fmaf_rn(d1, n1, d2 * n2)) / R - n2) / den;
        const double ww = lp[e].w;
        l += ww * (double)psi;
        ld += ww * (double)dpsi;
    }
    L = l;
    Ld = ld;
}

// ---- the reference's production rule (the mixed form)
// panel_integrals.rs:288-300 rankine_tier: 0 (order 3) beyond 8 radii, 1 (order 4) from 4, 2 (order 5)
// from 3, 3 (order 6) from 2; -1 (the closed forms) within 2
__device__ __forceinline__ int rankine_tier(double r) {
    return r >= 8.0 ? 0 : r >= 4.0 ? 1 : r >= 3.0 ? 2 : r >= 2.0 ? 3 : -1;
}

// panel_integrals.rs:305-357 rankine_gauss: the tier's rule in float32 on the point taken relative to the
// centroid in double, eight accumulator lanes summed in double (the reference's lane order)
__device__ inline void rankine_gauss_tier(const PanelRegs& p, const float* __restrict__ tq, const double* x, int t,
                                          double& S, double& D) {
    const int len = tier_len(t);
    const float* b = tq + tier_off(t);
    const float px = (float)(x[0] - p.c[0]), py = (float)(x[1] - p.c[1]), pz = (float)(x[2] - p.c[2]);
    const float nx = (float)p.n[0], ny = (float)p.n[1], nz = (float)p.n[2];
    float sacc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, dacc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int k = 0; k < len; k += 8)
#pragma unroll
        for (int l = 0; l < 8; l++) {
            const float rx = px - b[k + l], ry = py - b[len + k + l], rz = pz - b[2 * len + k + l];
            const float w = b[3 * len + k + l];
            const float r2 = __fmaf_rn(rz, rz, __fmaf_rn(rx, rx, ry * ry));
            const float ir = 1.0f / sqrtf(r2);
            const float nr = __fmaf_rn(nz, rz, __fmaf_rn(nx, rx, ny * ry));
            sacc[l] = __fmaf_rn(w, ir, sacc[l]);
            dacc[l] = __fmaf_rn(w * nr, ir * (ir * ir), dacc[l]);
        }
    double s = 0.0, d = 0.0;
#pragma unroll
    for (int l = 0; l < 8; l++) {
        s += (double)sacc[l];
        d += (double)dacc[l];
    }
    S = s;
    D = d;
}

// Rankine integrals at x by the production rule, panel_integrals.rs:359-363 rankine_any: the tiers, or the closed forms
// within 2 radii.
__device__ __forceinline__ void rankine_prod(const PanelsView& pv, int j, const PanelRegs& p, const double* x, double& S,
                                             double& D) {
    const double rc[3] = {x[0] - p.c[0], x[1] - p.c[1], x[2] - p.c[2]};
    const int t = rankine_tier(norm3(rc) / p.radius);
    if (t >= 0)
        rankine_gauss_tier(p, pv.tiers + (size_t)j * TIER_FLOATS, x, t, S, D);
    else
        rankine(pv, j, p, x, S, D);
}

// panel_integrals.rs:380-392: in the production mode the log integral of an image farther than 12 radii
// by the panel's 3 x 3 rule in double
__device__ inline void log_far_3x3(const PanelsView& pv, int j, const PanelRegs& p, const double* image, double& L,
                                   double& Ld) {
    double l = 0.0, ld = 0.0;
    for (int k = 0; k < 9; k++) {
        const double xi[3] = {pv.at(P_GX + 3 * k, j), pv.at(P_GX + 3 * k + 1, j), pv.at(P_GX + 3 * k + 2, j)};
        double psi, dpsi;
        psi_terms(xi, image, p.n, psi, dpsi);
        const double w = pv.at(P_GW + k, j);
        l += w * psi;
        ld += w * dpsi;
    }
    L = l;
    Ld = ld;
}

__device__ __forceinline__ double to_f32(double v) { return (double)(float)v; }

// lo_static.rs:47-55 log_pair
__device__ __forceinline__ bool log_pair(const PanelRegs& p, const double* x, double tol) {
    double dx = x[0] - p.c[0], dy = x[1] - p.c[1], zz = fabs(x[2] + p.c[2]);
    double d = sqrt(dx * dx + dy * dy + zz * zz) + zz;
    return d * d * tol < 0.6 * p.radius * p.radius;
}

// panel_integrals.rs:625-648 log_in_plane
__device__ inline double log_in_plane(const PanelRegs& p, const double* x) {
    double sum = 0.0;
    for (int i = 0; i < p.nv; i++) {
        int i1 = (i + 1) == p.nv ? 0 : i + 1;
        double ax[3], bx[3], e[3];
        for (int d = 0; d < 3; d++) {
            ax[d] = p.v[i][d] - x[d];
            bx[d] = p.v[i1][d] - x[d];
        }
        double h = dot3(ax, p.em[i]);
        if (h == 0.0) continue;
        for (int d = 0; d < 3; d++) e[d] = (1.0 / p.elen[i]) * (p.v[i1][d] - p.v[i][d]);
        double t1 = dot3(ax, e), t2 = dot3(bx, e);
        double q1 = h * h + t1 * t1, q2 = h * h + t2 * t2;
        double F1 = 0.5 * (t1 * log(q1) - 2.0 * t1 + 2.0 * h * atan(t1 / h)) - 0.5 * t1;
        double F2 = 0.5 * (t2 * log(q2) - 2.0 * t2 + 2.0 * h * atan(t2 / h)) - 0.5 * t2;
        sum += 0.5 * h * (F2 - F1);
    }
    return sum;
}

// One (row k, panel j) pair: rs, rd and (unless adaptive) dl, dd.  lo_static.rs:59-119
// Four planes of Nr x N (rows k < Nr = N / G, the sector's points, or the Nr field points; every panel
// j), entry at k + j Nr.
// MIXED: the mixed form's variant (far Rankine points and the order-4 log rule in FP32, above; with
// pv.tiers the reference's production rule instead, rows in float32).  The FP64 form runs the reference's double-precision
// arithmetic: its decisions, closed forms, 3 x 3 and order-4 rules in the reference's order of operations; the sums of the
// orders 5 to 10 (lanes, then shuffles) and of the adaptive cells (warps) are added in another order, so that those log
// integrals differ in their last bits.
// Bound by instruction issue and the conversions' pipe (per 32 pairs of the mixed form, infinite depth: 1800
// instructions, of them 440 FP64 and 150 conversions and reciprocals, before; FP64 closed forms near, the 3 x 3 and
// order-4 rules far).  Three CTAs an SM (80 registers, some spills) against two: 18496 panels 32.6 / 39.3 ms.  Measured, ms
// before / now: mixed 4096 panels, h = 5 m 4.2 / 2.6, 12288 panels 13.7 / 9.8, 18496 panels 50.0 / 33.5, FP64 4096
// panels 7.4 / 6.4; 84 panels 0.18 / 0.035, with the adaptive pairs 0.46 / 0.11.
// A warp has one panel; what depends on the panel alone (its data, the 3 x 3 rule, the points of the order-4 log rule
// with their FP64 bilinear map and Jacobian) is formed once by the warp, in shared memory.
template <bool MIXED, bool FINITE>
__global__ void __launch_bounds__(256, 3) k_statics(PanelsView pv, double depth, int logint, double tol, int rows,
                                                 double* __restrict__ st, int32_t* __restrict__ work,
                                                 int32_t* __restrict__ nwork, int work_cap) {
    constexpr int NI = FINITE ? 6 : 2;  // the point and its images
    // rows: the sector's panels (or the field points); columns: all panels
    const int N = pv.N, Nr = pv.rows ? pv.nrows : N / pv.G;
    int k = blockIdx.x * rows + threadIdx.x;  // a warp's first `rows` lanes hold a row each
    int j = blockIdx.y * 8 + threadIdx.y;
    // the panel of each warp (36 values every lane of the warp reads) in shared memory rather than in
    // 72 registers of every lane
    __shared__ PanelRegs sp[8];
    __shared__ LogPoint slp[8][16];
    __shared__ double sg[MIXED ? 8 : 1][9][3];
    __shared__ float sgw[MIXED ? 8 : 1][9];
    if (j >= N) return;  // (a whole warp)
    if (threadIdx.x == 0) load_panel(pv, j, sp[threadIdx.y]);
    __syncwarp();
    const PanelRegs& p = sp[threadIdx.y];
    if (threadIdx.x < 16) slp[threadIdx.y][threadIdx.x] = log_point4(p, threadIdx.x);
    if (MIXED && threadIdx.x < 9) {
        for (int d = 0; d < 3; d++) sg[threadIdx.y][threadIdx.x][d] = pv.at(P_GX + 3 * threadIdx.x + d, j);
        sgw[threadIdx.y][threadIdx.x] = (float)pv.at(P_GW + threadIdx.x, j);
    }
    __syncwarp();
    const LogPoint* lp = slp[threadIdx.y];
    const bool live = (int)threadIdx.x < rows && k < Nr;
    if (!live) k = min(k, Nr - 1);
    double x[3];
    for (int d = 0; d < 3; d++) x[d] = pv.rows ? pv.rows[3 * k + d] : pv.at(P_C + d, k);
    double xb[3] = {x[0], x[1], -x[2]};
    const double h = depth;
    double z[NI], S[NI], D[NI];
    z[0] = x[2];
    z[1] = -x[2];
    if constexpr (FINITE) {
        z[2] = -x[2] - 2.0 * h;
        z[3] = x[2] + 2.0 * h;
        z[4] = x[2] - 2.0 * h;
        z[5] = -x[2] - 4.0 * h;
    }
    if (MIXED && !pv.tiers) {  // the mixed form's own rule: the closed forms within MIX_FAR radii
        const double far = MIX_FAR * p.radius, t0 = x[0] - p.c[0], t1 = x[1] - p.c[1];
        unsigned mine = 0, any = 0;
#pragma unroll
        for (int i = 0; i < NI; i++) {
            const double t2 = z[i] - p.c[2];
            const bool f = t0 * t0 + t1 * t1 + t2 * t2 > far * far;
            mine |= (unsigned)f << i;
            any |= (unsigned)(__any_sync(0xffffffffu, f) != 0) << i;
        }
        rankine_gauss_f32<NI>(sg[threadIdx.y], sgw[threadIdx.y], p, x, z, any, S, D);
#pragma unroll
        for (int i = 0; i < NI; i++)
            if (live && !(mine >> i & 1)) {
                const double xi[3] = {x[0], x[1], z[i]};
                rankine(pv, j, p, xi, S[i], D[i]);
            }
    } else if (live) {
#pragma unroll
        for (int i = 0; i < NI; i++) {
            const double xi[3] = {x[0], x[1], z[i]};
            if (!MIXED)
                rankine(pv, j, p, xi, S[i], D[i]);
            else if (i >= 4)  // production: the two deep images by the 3 x 3 rule beyond 12 radii
                rankine(pv, j, p, xi, S[i], D[i], 12.0);  // (lo_static.rs:82-88)
            else
                rankine_prod(pv, j, p, xi, S[i], D[i]);
        }
    }
    double sr = S[0] + S[1], dr = D[0] + D[1];
    if constexpr (FINITE) {
        sr += (S[2] + S[3]) + S[4] + S[5];
        dr += (D[2] + D[3]) + D[4] + D[5];
    }
    const bool prod = MIXED && pv.tiers;  // the production rows are stored in float32
    size_t NN = (size_t)Nr * N, o = (size_t)k + (size_t)j * Nr;
    if (live) {
        st[o] = prod ? to_f32(sr) : sr;
        st[NN + o] = prod ? to_f32(dr) : dr;
    }
    double dl = 0.0, dd = 0.0;
    const bool use_log = live && logint && log_pair(p, x, tol);
    const bool plane = use_log && pv.kind[j] == 1 && x[2] == 0.0;
    int order = 4;
    bool far3 = false;
    if (use_log && !plane) {
        const double tb[3] = {xb[0] - p.c[0], xb[1] - p.c[1], xb[2] - p.c[2]};
        far3 = prod && norm3(tb) > 12.0 * p.radius;
        order = far3 ? 3 : log_order(p, xb);
    }
    // the near images one after another, each by the whole warp
    double L = 0.0, Ld = 0.0;
    for (unsigned near = __ballot_sync(0xffffffffu, order > 4); near; near &= near - 1) {
        const int src = __ffs(near) - 1;
        const double image[3] = {__shfl_sync(0xffffffffu, xb[0], src), __shfl_sync(0xffffffffu, xb[1], src),
                                 __shfl_sync(0xffffffffu, xb[2], src)};
        double l, ld;
        log_gauss_warp(p, image, __shfl_sync(0xffffffffu, order, src), threadIdx.x, l, ld);
        if ((int)threadIdx.x == src) L = l, Ld = ld;
    }
    if (!live) return;
    if (plane) {
        const double Lp = log_in_plane(p, x);
        double t[3] = {p.c[0] - x[0], p.c[1] - x[1], p.c[2] - x[2]};
        double Rr = norm3(t);
        dl = Rr > 0.0 ? Lp - p.area * log(Rr) : Lp;
    } else if (use_log && order > 0) {
        double psi, dpsi;
        if (far3)
            log_far_3x3(pv, j, p, xb, L, Ld);
        else if (order == 4 && MIXED && !prod)
            log_gauss4_f32(lp, p, xb, L, Ld);
        else if (order == 4)
            log_gauss4(lp, p, xb, L, Ld);
        psi_terms(p.c, xb, p.n, psi, dpsi);
        dl = L - p.area * psi;
        dd = Ld - p.area * dpsi;
    } else if (use_log) {
        int slot = atomicAdd(nwork, 1);
        if (slot < work_cap) {
            work[2 * slot] = k;
            work[2 * slot + 1] = j;
        }
    }
    st[2 * NN + o] = prod ? to_f32(dl) : dl;
    st[3 * NN + o] = prod ? to_f32(dd) : dd;
}

// The adaptive pairs: quadrisection to 1e-13 of the integrals' scale, at most 14 levels
// (panel_integrals.rs:100-120).  One CTA per pair: the cells wait on a stack in shared memory, each round the
// AD_WARPS topmost are taken, a warp each (the 32 lanes evaluate the 4 sub-cells x 16 Gauss points, two a lane, and
// reduce them per sub-cell by shuffles), and those to be split push their sub-cells.  A cell's decision depends on
// its own sums alone, so the cells are those of the reference's depth-first order; their sums are added per warp,
// then over the warps in order.  (One warp a pair took 0.29-0.39 ms for the few pairs of a small hull.)
// The stack's bound: the sub-cells of deeper cells go above those of shallower ones, so the stack stays sorted by depth
// and a round that pushes a level has taken every deeper cell before it.  A level then has at most 4 AD_WARPS cells, of
// which AD_WARPS went for a full next level: 3 AD_WARPS stay on each of the levels 3 .. 13 under a full level 14, 12
// on level 2 (of 16) and 3 on level 1 (of 4), 304 in all; a round that pushes two levels shares its cells between them.
constexpr int AD_WARPS = 8, AD_DEPTH = 14, AD_STACK = AD_WARPS * 48;
static_assert(16 + 3 * AD_WARPS * (AD_DEPTH - 2) <= AD_STACK, "the adaptive pairs' stack");

struct AdCell {
    double u0, u1, v0, v1, p0, p1;
    int depth;
};

__device__ __forceinline__ void log_point(const double m[4][3], const double* image, const double* n, double u0,
                                          double u1, double v0, double v1, int i, int j, double& a, double& b) {
    double hu = 0.5 * (u1 - u0), hv = 0.5 * (v1 - v0);
    double xi[3], jac, psi, dpsi;
    bilinear(m, u0 + hu * (c_glx[4][i] + 1.0), v0 + hv * (c_glx[4][j] + 1.0), xi, jac);
    double ww = c_glw[4][i] * c_glw[4][j] * hu * hv * jac;
    psi_terms(xi, image, n, psi, dpsi);
    a = ww * psi;
    b = ww * dpsi;
}

struct AdShared {
    AdCell stk[AD_STACK];
    PanelRegs p;
    double acc[AD_WARPS][2];
    int split[AD_WARPS];
    int entry;
};

// One adaptive pair (worklist entry t) by the calling CTA.
__device__ void adaptive_pair(const PanelsView& pv, const int32_t* __restrict__ work, int t, double* __restrict__ st,
                              AdShared& sh) {
    const int N = pv.N, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k = work[2 * t], j = work[2 * t + 1];
    if (threadIdx.x == 0) load_panel(pv, j, sh.p);
    __syncthreads();
    const PanelRegs& p = sh.p;
    double xb[3];
    for (int d = 0; d < 3; d++) xb[d] = pv.rows ? pv.rows[3 * k + d] : pv.at(P_C + d, k);
    xb[2] = -xb[2];
    double m[4][3];
    panel_map(p, m);
    double tt[3] = {xb[0] - p.c[0], xb[1] - p.c[1], xb[2] - p.c[2]};
    double dist = norm3(tt);
    double dmin = fmax(dist - p.radius, 1e-3 * p.radius);
    double scale = fabs(log(dist + p.radius)) + 1.0;
    double tol_l = 1e-13 * p.area * scale, tol_d = 1e-13 * p.area / dmin;
    if (warp == 0) {  // the whole square by one 4 x 4 cell (lanes 0..15 one point each)
        double wa = 0.0, wb = 0.0;
        if (lane < 16) log_point(m, xb, p.n, -1.0, 1.0, -1.0, 1.0, lane / 4, lane % 4, wa, wb);
        for (int o = 16; o > 0; o >>= 1) {
            wa += __shfl_xor_sync(0xffffffffu, wa, o);
            wb += __shfl_xor_sync(0xffffffffu, wb, o);
        }
        if (lane == 0) sh.stk[0] = AdCell{-1.0, 1.0, -1.0, 1.0, wa, wb, 0};
    }
    int sp = 1;
    double acc0 = 0.0, acc1 = 0.0;
    __syncthreads();
    while (sp > 0) {
        const int take = min(sp, AD_WARPS);
        sp -= take;
        bool split = false;
        AdCell c;
        double a0, b0, a1, b1, um, vm;
        if (warp < take) {
            c = sh.stk[sp + take - 1 - warp];
            um = 0.5 * (c.u0 + c.u1), vm = 0.5 * (c.v0 + c.v1);
            // lane l: point l % 16 of sub-cells (l / 16) and (l / 16) + 2, in the order (u0, v0), (um, v0), (um, vm), (u0, vm)
            const int sa = lane >> 4, q = lane & 15;
            const double ua = sa ? um : c.u0, ub = sa ? c.u1 : um;
            log_point(m, xb, p.n, ua, ub, c.v0, vm, q / 4, q % 4, a0, b0);
            log_point(m, xb, p.n, sa ? c.u0 : um, sa ? um : c.u1, vm, c.v1, q / 4, q % 4, a1, b1);
            for (int o = 8; o > 0; o >>= 1) {
                a0 += __shfl_xor_sync(0xffffffffu, a0, o);
                b0 += __shfl_xor_sync(0xffffffffu, b0, o);
                a1 += __shfl_xor_sync(0xffffffffu, a1, o);
                b1 += __shfl_xor_sync(0xffffffffu, b1, o);
            }
            // the sums of sub-cells 0, 1 (lanes 0, 16 of a0, b0) and 2, 3
            const double s0 = __shfl_sync(0xffffffffu, a0, 0) + __shfl_sync(0xffffffffu, a0, 16) +
                              __shfl_sync(0xffffffffu, a1, 0) + __shfl_sync(0xffffffffu, a1, 16);
            const double s1 = __shfl_sync(0xffffffffu, b0, 0) + __shfl_sync(0xffffffffu, b0, 16) +
                              __shfl_sync(0xffffffffu, b1, 0) + __shfl_sync(0xffffffffu, b1, 16);
            split = !(c.depth >= AD_DEPTH || (fabs(s0 - c.p0) <= tol_l && fabs(s1 - c.p1) <= tol_d));
            if (!split) acc0 += s0, acc1 += s1;
        }
        if (lane == 0) sh.split[warp] = split;
        __syncthreads();  // the cells are taken, the decisions known
        int at = sp, total = 0;
#pragma unroll
        for (int w = 0; w < AD_WARPS; w++) {
            if (w > warp) at += 4 * sh.split[w];  // (warp 0 has the deepest cell)
            total += sh.split[w];
        }
        if (split && (lane & 15) == 0) {  // lanes 0 and 16 hold the sums of sub-cells 0, 2 and 1, 3
            const int sa = lane >> 4;
            sh.stk[at + 3 - sa] = AdCell{sa ? um : c.u0, sa ? c.u1 : um, c.v0, vm, a0, b0, c.depth + 1};
            sh.stk[at + 1 - sa] = AdCell{sa ? c.u0 : um, sa ? um : c.u1, vm, c.v1, a1, b1, c.depth + 1};
        }
        sp += 4 * total;
        __syncthreads();
    }
    if (lane == 0) sh.acc[warp][0] = acc0, sh.acc[warp][1] = acc1;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < AD_WARPS; w++) acc0 += sh.acc[w][0], acc1 += sh.acc[w][1];
        double psi, dpsi;
        psi_terms(p.c, xb, p.n, psi, dpsi);
        const int Nr = pv.rows ? pv.nrows : N / pv.G;
        size_t NN = (size_t)Nr * N, o = (size_t)k + (size_t)j * Nr;
        const double vl = acc0 - p.area * psi, vd = acc1 - p.area * dpsi;
        st[2 * NN + o] = pv.tiers ? to_f32(vl) : vl;  // the production rows in float32
        st[3 * NN + o] = pv.tiers ? to_f32(vd) : vd;
    }
}

// One CTA per worklist entry, the entry count given by the host.
__global__ void __launch_bounds__(AD_WARPS * 32) k_statics_adaptive(PanelsView pv, const int32_t* __restrict__ work,
                                                                    int nwork, double* __restrict__ st) {
    __shared__ AdShared sh;
    if ((int)blockIdx.x < nwork) adaptive_pair(pv, work, blockIdx.x, st, sh);
}

// The same with the entry count in device memory (q[0], capped at work_cap) and the entries taken
// from a queue (cursor q[1], zero at launch), so that the host need not wait for the count.  No
// work when the geometry flagged an invalid panel (*bad != clean): the solve reports it.
__global__ void __launch_bounds__(AD_WARPS * 32) k_statics_adaptive_q(PanelsView pv, const int32_t* __restrict__ work,
                                                                      int32_t* q, int work_cap,
                                                                      const int32_t* __restrict__ bad, int32_t clean,
                                                                      double* __restrict__ st) {
    __shared__ AdShared sh;
    if (*bad != clean) return;
    const int nwork = min(*(volatile int32_t*)q, work_cap);
    for (;;) {
        if (threadIdx.x == 0) sh.entry = atomicAdd(q + 1, 1);
        __syncthreads();
        const int t = sh.entry;
        if (t >= nwork) return;
        adaptive_pair(pv, work, t, st, sh);
        __syncthreads();  // (the next entry overwrites the shared data)
    }
}

// ------------------------------------------------------------------ host launchers
void launch_panel_geometry(int N, const double* verts, const int32_t* kind, double* planes, int32_t* bad,
                           cudaStream_t s, float* tiers, const int32_t* orig) {
    k_panel_geometry<<<(N + 127) / 128, 128, 0, s>>>(N, verts, kind, planes, bad, tiers, orig);
}

// Pairs up to which a warp takes four rows instead of 32.  A warp costs the same with few rows, so they pay only while
// the device is nearly empty.  Measured, us with 4 / 32 rows: the FP64 form in deep water 42 panels 23 / 66, 81 29 / 66,
// 121 47 / 62, 144 54 / 64, 169 70 / 64, 240 117 / 64, 506 448 / 111; in depth 3 m (three times the images) 81 45 / 80,
// 121 78 / 76, 144 92 / 78; the mixed form 121 47 / 68 and 62 / 74, 169 68 / 67 and 79 / 68; a box hull of 84 35 / 51,
// 144 60 / 52.  The line (126 panels) is where the first of them cross; 8 and 16 rows are within 20 us of the better one
// between 100 and 240 panels.
constexpr double STATICS_SMALL = 1.6e4;

void launch_statics(const PanelsView& pv, double depth, int logint, double tol, double* st, int32_t* work,
                    int32_t* nwork, int work_cap, cudaStream_t s, bool mixed) {
    // few panels: fewer rows a warp, so that its near images (a warp's work each) are spread over the device
    const int Nr = pv.rows ? pv.nrows : pv.N / pv.G;
    const int rows = (double)Nr * pv.N < STATICS_SMALL ? 4 : 32;
    dim3 grid((Nr + rows - 1) / rows, (pv.N + 7) / 8);
    auto go = [&](auto kernel) {
        kernel<<<grid, dim3(32, 8), 0, s>>>(pv, depth, logint, tol, rows, st, work, nwork, work_cap);
    };
    if (mixed)
        depth > 0.0 ? go(k_statics<true, true>) : go(k_statics<true, false>);
    else
        depth > 0.0 ? go(k_statics<false, true>) : go(k_statics<false, false>);
}

void launch_statics_adaptive(const PanelsView& pv, const int32_t* work, int nwork, double* st, cudaStream_t s) {
    if (nwork > 0) k_statics_adaptive<<<nwork, AD_WARPS * 32, 0, s>>>(pv, work, nwork, st);
}

void launch_statics_adaptive_q(const PanelsView& pv, const int32_t* work, int32_t* q, int work_cap,
                               const int32_t* bad, int32_t clean, double* st, cudaStream_t s) {
    static int grid[16] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 16) dev = 0;
    if (grid[dev] == 0) {
        int sms = 0, per = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_statics_adaptive_q, AD_WARPS * 32, 0);
        grid[dev] = std::max(1, sms * std::max(per, 1));
    }
    k_statics_adaptive_q<<<grid[dev], AD_WARPS * 32, 0, s>>>(pv, work, q, work_cap, bad, clean, st);
}

void set_constants_statics(const double glx[17][16], const double glw[17][16]) {
    cudaMemcpyToSymbol(c_glx, glx, sizeof(double) * 17 * 16);
    cudaMemcpyToSymbol(c_glw, glw, sizeof(double) * 17 * 16);
}

}  // namespace hbg
