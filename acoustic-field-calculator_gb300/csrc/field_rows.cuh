// Grid field evaluation tiled by rows: the per-block body of field_rows_kernel.
//
// Each thread owns one first-axis index, one third-axis index and 2*PAIRS consecutive second-axis
// indices, so its points share two of their three coordinates; a warp's threads form a compact box
// (RowsMap: 8 x 8 x 4 points of a volume, 16 x 16 of a slice at 4 pairs).  Sources are staged with their coordinates and directions permuted into the
// grid's axis order; per source and thread, the offsets along the first and third axes, the
// sum of their squares and (for tiles of unequal directions) their part of n.d are computed
// once, and each point pair only adds the offset along the second axis: three fewer packed
// FP32 instructions per pair than the general body (field_body.cuh), whose math this is.
//
// Directivity.  Seen from one source, cos(theta) changes little over a warp's box.  Where the
// whole box lies inside one 10-degree bin of a source, D is one smooth function of c there, and
// the warp takes it from a quartic about the box centre's c (warp_dir_poly, one lane per source,
// 32 sources at a time): four packed FMAs a pair, no table load and no edge test.  Elsewhere it
// comes from the cos(theta)-indexed table (directivity2_ctab, about 12 instructions a point), and
// a thread keeps the smallest |c - L| of its points for the exact edge path.  What bounds it:
// instruction issue and the MUFU (7 lane slots a pair); 3,984 sources on 256^3 points went from
// 64.4 to 55.3 ms with the polynomials (91 % of the (warp, source) pairs), from 27 to 19
// instructions a pair, and to 54.7 ms with two sources a turn.  Points and the order of the sum
// over sources are the reference's (observe_area/grid/grid_area.rs:59-229,
// system/uniform_medium.rs:111-128).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "afc_internal.h"
#include "field_body.cuh"
#include "propagate.cuh"

namespace afc {
namespace fb {

__device__ __forceinline__ float pick3(float x, float y, float z, int a) {
    return a == 0 ? x : (a == 1 ? y : z);
}

// Per thread and source: offsets along the grid's first (v) and third (w) axes, v^2 + w^2,
// and n_v v + n_w w; for the far tiles also qb, qc with which the reference's
// (dx dx + dy dy) + dz dz is (du du + qb) + qc in the same rounding (see row_q2_parts).
struct RowShared {
    float dv, dw, vw2, nvw, qb, qc;
};

// The reference sums the squared offsets in x, y, z order (uniform_medium.rs:111-113); the rows
// body has the second grid axis's (u) per pair and the others' per source.  With a1 the xyz
// index of u and a0 that of v: u = z gives (du du + (sx + sy)) + 0, u = x gives
// (du du + sy) + sz and u = y gives (du du + sx) + sz, each rounding as the reference's sum
// (an addition commutes exactly, and adding +0 to a non-negative sum changes nothing).
__device__ __forceinline__ void row_q2_parts(float dv, float dw, int a0, int a1, float& qb,
                                             float& qc) {
    const float sv = __fmul_rn(dv, dv), sw = __fmul_rn(dw, dw);
    if (a1 == 2) {
        qb = __fadd_rn(sv, sw);
        qc = 0.f;
    } else {
        qb = a1 == 0 ? (a0 == 1 ? sv : sw) : (a0 == 0 ? sv : sw);  // y for u = x, x for u = y
        qc = a0 == 2 ? sv : sw;                                      // z
    }
}

// Point pair q of a thread against the staged source (t0 = its v[0], t2 = its v[2]): offset along
// the second axis, r^2, 1/r and the numerator of cos(theta), with the same operations on the hot
// loop and on its edge path.
struct RowGeom {
    float2 du, r2, rinv, cn;
    __device__ __forceinline__ RowGeom(float2 u, const RowShared& sh, float4 t0, float4 t2) {
        du = add2(u, lo2(t0));
        r2 = fma2(du, du, f2(sh.vw2));
        rinv = make_float2(mufu_rsqrt(r2.x), mufu_rsqrt(r2.y));
        cn = fma2(hi2(t2), du, f2(sh.nvw));
    }
    __device__ __forceinline__ float2 ct() const { return mul2(cn, rinv); }
};

// Edge correction for one point of the rows body (see edge_correction): the pair is
// recomputed from the offsets as the hot loop computed it; the reference's bin needs the
// offsets and the direction back in x, y, z order (a0, a1, a2: the xyz index of each grid
// axis).
static __device__ __noinline__ float2 edge_correction_rows(const float4* __restrict__ tab,
                                                           const float* __restrict__ cneg,
                                                           const float4* __restrict__ ccoef,
                                                           float du, float dv, float dw, float vw2,
                                                           float cn, float n_a0, float n_a1,
                                                           float n_a2, int a0, int a1, float k,
                                                           float phase, float a2c, float la) {
    const float r2 = fmaf(du, du, vw2);
    const float rinv = mufu_rsqrt(r2);
    const float ct = cn * rinv;
    float2 t;
    const float d_fast = directivity2_ctab(cneg, ccoef, make_float2(ct, ct), t).x;
    const float thc = theta2_centred(make_float2(ct, ct)).x;
    // back to x, y, z: the first grid axis carries v, the second u, the third w
    const float dx = a0 == 0 ? dv : (a1 == 0 ? du : dw);
    const float dy = a0 == 1 ? dv : (a1 == 1 ? du : dw);
    const float dz = a0 == 2 ? dv : (a1 == 2 ? du : dw);
    const float nx = a0 == 0 ? n_a0 : (a1 == 0 ? n_a1 : n_a2);
    const float ny = a0 == 1 ? n_a0 : (a1 == 1 ? n_a1 : n_a2);
    const float nz = a0 == 2 ? n_a0 : (a1 == 2 ? n_a1 : n_a2);
    const int i_exact = exact_bin(dx, dy, dz, nx, ny, nz);
    float2 r;
    const float red =
        ref_phase2(ref_dist2(f2(dx), f2(dy), f2(dz)), f2(rinv), f2(k), f2(phase), r).x;
    const float w0 = rinv * mufu_ex2(fmaf(a2c, r.x, la));
    const float corr = w0 * (dir_in_bin(tab, thc, i_exact) - d_fast);
    return make_float2(corr * mufu_cos(red), corr * mufu_sin(red));
}

// The PAIRS point pairs of one thread against staged source j (RowsTile).  p0, p2: the thread's
// coordinates along the first and third grid axes; U: its points' coordinates along the second.
// POLY: the directivity from the warp's polynomial for this source, whose three float4 lie 32
// apart from `poly`.
// Returns whether some point lies next to a bin edge (correct_rows).
template <int ST, int SUM, int PAIRS, int PH, bool POLY>
__device__ __forceinline__ bool accumulate_rows(const RowsTile& sm, const RowsTable& rt, int j,
                                                const float4* __restrict__ poly, float p0, float p2,
                                                int a0, int a1, float2 (&U)[PAIRS],
                                                float2 (&RE)[PAIRS], float2 (&IM)[PAIRS],
                                                float2 (&CRE)[PAIRS], float2 (&CIM)[PAIRS]) {
    const float4 t0 = sm.v[0][j], t1 = sm.v[1][j], t2 = sm.v[2][j], t3 = sm.v[3][j];
    RowShared sh;
    sh.dv = p0 + t3.x;
    sh.dw = p2 + t3.y;
    sh.vw2 = fmaf(sh.dw, sh.dw, sh.dv * sh.dv);
    sh.nvw = ST == SRC_T4010A1 ? fmaf(t3.w, sh.dw, t3.z * sh.dv) : 0.f;
    sh.qb = sh.qc = 0.f;
    if constexpr (PH == kPhaseRef) row_q2_parts(sh.dv, sh.dw, a0, a1, sh.qb, sh.qc);
    float4 w0, w1, w2;
    if constexpr (POLY) {
        w0 = poly[0];
        w1 = poly[32];
        w2 = poly[64];
    }
    float near_min = kCTabMargin;  // smallest |c - L| of the thread's points (the edge test)
#pragma unroll
    for (int q = 0; q < PAIRS; ++q) {
        const RowGeom p(U[q], sh, t0, t2);
        float2 r = mul2(p.r2, p.rinv);
        float2 red;
        if constexpr (PH == kPhaseRef) {
            const float2 q2 =
                make_float2(__fadd_rn(__fadd_rn(__fmul_rn(p.du.x, p.du.x), sh.qb), sh.qc),
                            __fadd_rn(__fadd_rn(__fmul_rn(p.du.y, p.du.y), sh.qb), sh.qc));
            red = ref_phase2(q2, p.rinv, hi2(t0), lo2(t2), r);
        } else if constexpr (PH == kPhaseMid) {
            red = mid_phase2(p.r2, p.rinv, hi2(t0), lo2(t2), r);
        } else {
            red = fma2(hi2(t0), r, lo2(t2));
        }
        const float2 ea = fma2(lo2(t1), r, hi2(t1));
        float2 w = mul2(p.rinv, make_float2(mufu_ex2(ea.x), mufu_ex2(ea.y)));
        if constexpr (POLY) {
            const float2 x = fma2(p.cn, p.rinv, hi2(w2));
            float2 d = fma2(lo2(w0), x, hi2(w0));
            d = fma2(d, x, lo2(w1));
            d = fma2(d, x, hi2(w1));
            d = fma2(d, x, lo2(w2));
            w = mul2(w, d);
        } else if constexpr (ST == SRC_T4010A1) {
            float2 t;
            w = mul2(w, directivity2_ctab(rt.cneg, rt.ccoef, p.ct(), t));
            near_min = fminf(near_min, fminf(fabsf(t.x), fabsf(t.y)));
        }
        const float2 sn = make_float2(mufu_sin(red.x), mufu_sin(red.y));
        const float2 cs = make_float2(mufu_cos(red.x), mufu_cos(red.y));
        if constexpr (SUM == SUM_PLAIN) {
            RE[q] = fma2(w, cs, RE[q]);
            IM[q] = fma2(w, sn, IM[q]);
        } else {
            neumaier_add2(RE[q], CRE[q], make_float2(__fmul_rn(w.x, cs.x), __fmul_rn(w.y, cs.y)));
            neumaier_add2(IM[q], CIM[q], make_float2(__fmul_rn(w.x, sn.x), __fmul_rn(w.y, sn.y)));
        }
    }
    return ST == SRC_T4010A1 && !POLY && near_min < kCTabMargin;
}

// Whether some cosine of a direction, seen from a box whose lowest n.(x - s) is `front`, may leave the table:
// a direction longer than 1 by more than rounding seen from behind, or one near 3 from anywhere.
__device__ __forceinline__ bool leaves_table(float nx, float ny, float nz, float front) {
    const float nn = fmaf(nz, nz, fmaf(ny, ny, nx * nx));
    return nn > 8.f || (nn > 1.000004f && !(front >= 0.f));
}

// The exact bins of the points that accumulate_rows found next to an edge for source j; where the tile's
// cosines may leave the table (LONG), also of those that do.
template <int SUM, int PAIRS, bool LONG>
__device__ __forceinline__ void correct_rows(const RowsTile& sm, const RowsTable& rt, int j, float p0,
                                             float p2, int a0, int a1, float2 (&U)[PAIRS],
                                             float2 (&RE)[PAIRS], float2 (&IM)[PAIRS],
                                             float2 (&CRE)[PAIRS], float2 (&CIM)[PAIRS]) {
    const float4 t0 = sm.v[0][j], t1 = sm.v[1][j], t2 = sm.v[2][j], t3 = sm.v[3][j];
    RowShared sh;
    sh.dv = p0 + t3.x;
    sh.dw = p2 + t3.y;
    sh.vw2 = fmaf(sh.dw, sh.dw, sh.dv * sh.dv);
    sh.nvw = fmaf(t3.w, sh.dw, t3.z * sh.dv);
#pragma unroll
    for (int q = 0; q < PAIRS; ++q) {
        const RowGeom p(U[q], sh, t0, t2);
        float2 t;
        directivity2_ctab(rt.cneg, rt.ccoef, p.ct(), t);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const bool out = LONG && (h ? p.ct().y < kBackAxisC || p.ct().y > 2.5f
                                        : p.ct().x < kBackAxisC || p.ct().x > 2.5f);
            if (!out && !near_edge_c(lane_of(t, h))) continue;
            const float2 c = edge_correction_rows(
                sm.dir, rt.cneg, rt.ccoef, lane_of(p.du, h), sh.dv, sh.dw, sh.vw2, lane_of(p.cn, h),
                t3.z, t2.z, t3.w, a0, a1, t0.z, t2.x, t1.x, t1.z);
            if constexpr (SUM == SUM_PLAIN) {
                lane_of(RE[q], h) += c.x;
                lane_of(IM[q], h) += c.y;
            } else {
                neumaier_add(lane_of(RE[q], h), lane_of(CRE[q], h), c.x);
                neumaier_add(lane_of(IM[q], h), lane_of(CIM[q], h), c.y);
            }
        }
    }
}

// A box of the grid (a warp's points) in grid axis order: its centre, half extents and the half
// diagonal.
struct RowsBox {
    float c0, c1, c2, h0, h1, h2, rho;
};

// The directivity of staged source j over a box as a polynomial in c = cos(theta), if it has one:
// true, and p[0..4], c0 with D(c) = p0 + x (p1 + x (p2 + x (p3 + x p4))), x = c - c0, where c0 is
// the box centre's c.
//
// Range of c over the box: with d from the source, g = (n - c0 d/|d|) / |d| its gradient at the
// centre and |n| 1.155 / r^2 a bound of its Hessian's norm (the eigenvalues for unit n are
// (-c +- sqrt(4 - 3 c^2)) / 2 r^2 and -c / r^2), |c - c0| <= h = sum_k |g_k| h_k + 0.6 |n| (rho / (|d| - rho))^2,
// plus kPolyMargin for the rounding of the pairs' own c and the edge margin of the table path.
// The box qualifies when [c0 - h, c0 + h] holds no bin edge (and no c next to -1, where the
// reference's bin is 0) and, outside the constant bins, h <= kPolyWidth (1 - c0^2).
//
// The polynomial is the bin's cubic in theta composed with the Taylor series of acos about c0, to
// degree 5, its last term economised over |x| <= h (x^5 ~ (20 h^2 x^3 - 5 h^4 x) / 16).  The truncation is
// within 6e-8 of D at the widest box and 1e-8 at half that width; evaluated in float32 it is within
// about 1.9e-7 at any width, since the rounding of its coefficients and steps decides, against 1.3e-7 for
// the table's entries, whose argument carries one rounding more.
constexpr float kPolyMargin = 1.5e-5f;
constexpr float kPolyWidth = 0.05f;

__device__ __forceinline__ bool warp_dir_poly(const RowsTile& sm, int j, const RowsBox& b,
                                              float (&p)[5], float& c0) {
    const float4 t3 = sm.v[3][j];
    const float dv = b.c0 + t3.x, du = b.c1 + sm.v[0][j].x, dw = b.c2 + t3.y;
    const float nv = t3.z, nu = sm.v[2][j].z, nw = t3.w;
    const float r2 = fmaf(dw, dw, fmaf(dv, dv, du * du));
    const float rinv = rsqrtf(r2);
    const float rmin = r2 * rinv - b.rho;
    c0 = fmaf(nw, dw, fmaf(nu, du, nv * dv)) * rinv;
    const float e = c0 * rinv;
    const float q = __fdividef(b.rho, rmin);
    const float nn = sqrtf(fmaf(nw, nw, fmaf(nu, nu, nv * nv)));
    float h = fabsf(fmaf(-e, dv, nv)) * b.h0 + fabsf(fmaf(-e, du, nu)) * b.h1 +
              fabsf(fmaf(-e, dw, nw)) * b.h2;
    h = fmaf(h, rinv, fmaf(0.6f * nn, q * q, kPolyMargin));
    // the bin of c0 and its bounds on c (bins 0 to 2 as one: D = 1; bin 10: D = 0)
    constexpr float kEdge[8] = {kBinCos3, kBinCos4, kBinCos5, kBinCos6,
                                kBinCos7, kBinCos8, kBinCos9, kBinCos10};
    int bin = 2;
    float hi = __int_as_float(0x7f800000), lo = kEdge[0];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        if (c0 <= kEdge[k]) {
            bin = k + 3;
            hi = kEdge[k];
            lo = k < 7 ? kEdge[k + 1] : kBackAxisC;
        }
    }
    const float s2 = (1.f - c0) * (1.f + c0);
    const bool flat = bin == 2 || bin == 10;
    const bool ok = rmin > 0.f && c0 + h < hi && c0 - h > lo && (flat || h <= kPolyWidth * s2);
    p[0] = bin == 2 ? 1.f : 0.f;
    p[1] = p[2] = p[3] = p[4] = 0.f;
    if (ok && !flat) {
        const float th = acosf(c0), i1 = rsqrtf(s2), i2 = i1 * i1, cc = c0 * c0;
        // acos(c0 + x) = th + t1 x + t2 x^2 + ...
        const float t1 = -i1, i3 = i1 * i2, i5 = i3 * i2, i7 = i5 * i2, i9 = i7 * i2;
        const float t2 = -0.5f * c0 * i3, t3 = fmaf(cc, -1.f / 3.f, -1.f / 6.f) * i5;
        const float t4 = -c0 * fmaf(cc, 0.25f, 0.375f) * i7;
        const float t5 = -fmaf(cc, fmaf(cc, 0.2f, 0.6f), 0.075f) * i9;
        const float4 k = sm.dir[bin];  // the bin's cubic about its centre
        const float xc = fmaf(static_cast<float>(bin) - 0.5f, -kAngleDiv, th);
        const float d1 = fmaf(fmaf(3.f * k.w, xc, 2.f * k.z), xc, k.y);
        const float d2 = fmaf(3.f * k.w, xc, k.z), d3 = k.w;
        const float t11 = t1 * t1;
        p[0] = fmaf(fmaf(fmaf(k.w, xc, k.z), xc, k.y), xc, k.x);
        p[1] = d1 * t1;
        p[2] = fmaf(d2, t11, d1 * t2);
        p[3] = fmaf(d3 * t11, t1, fmaf(2.f * d2 * t1, t2, d1 * t3));
        p[4] = fmaf(3.f * d3 * t11, t2, fmaf(d2, fmaf(t2, t2, 2.f * t1 * t3), d1 * t4));
        const float p5 = fmaf(3.f * d3 * t1, fmaf(t1, t3, t2 * t2),
                              fmaf(2.f * d2, fmaf(t1, t4, t2 * t3), d1 * t5));
        const float hh = h * h;
        p[3] = fmaf(p5 * 1.25f, hh, p[3]);
        p[1] = fmaf(p5 * -0.3125f * hh, hh, p[1]);
    }
    return ok;
}

// Sources 0 .. cnt - 1 of the staged tile against the thread's points (accumulate_rows) with the
// phase variant PH, in source order: each source with the warp's directivity polynomial where it
// has one, else with the table (one pair a thread: always, two points do not pay for setting
// polynomials up).  tile_long: some cosines may leave the table (then PH is kPhaseRef).
template <int ST, int SUM, int PAIRS, int PH>
__device__ __forceinline__ void rows_source_loop(int cnt, RowsSmem& rs, float p0, float p2, int a0,
                                                 int a1, int a2, float2 (&U)[PAIRS],
                                                 float2 (&RE)[PAIRS], float2 (&IM)[PAIRS],
                                                 float2 (&CRE)[PAIRS], float2 (&CIM)[PAIRS],
                                                 bool tile_long = false) {
    const RowsTile& sm = rs.sm;
    if constexpr (ST == SRC_T4010A1 && PH != kPhaseRef && PAIRS > 1) {
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        float4(*w)[32] = rs.poly.w[wid];
#pragma unroll 1
        for (int j0 = 0; j0 < cnt; j0 += 32) {
            bool ok = false;
            if (j0 + lane < cnt) {
                const float* box = sm.box[wid];  // the warp's own bounds, in x, y, z slots
                RowsBox b;
                b.h0 = 0.5f * (box[3 + a0] - box[a0]);
                b.h1 = 0.5f * (box[3 + a1] - box[a1]);
                b.h2 = 0.5f * (box[3 + a2] - box[a2]);
                b.c0 = box[a0] + b.h0;
                b.c1 = box[a1] + b.h1;
                b.c2 = box[a2] + b.h2;
                b.rho = sqrtf(fmaf(b.h2, b.h2, fmaf(b.h1, b.h1, b.h0 * b.h0)));
                float p[5], c0;
                ok = warp_dir_poly(sm, j0 + lane, b, p, c0);
                w[0][lane] = make_float4(p[4], p[4], p[3], p[3]);
                w[1][lane] = make_float4(p[2], p[2], p[1], p[1]);
                w[2][lane] = make_float4(p[0], p[0], -c0, -c0);
            }
            const unsigned mask = __ballot_sync(0xffffffffu, ok);
            __syncwarp();
            const int e = cnt - j0 < 32 ? cnt - j0 : 32;
#pragma unroll 1
            for (int j = 0; j < e; ++j) {
                // two sources at a time where both have one: half the loop's branches, and two
                // sources' chains to interleave (128^3: 7.36 -> 7.17 ms; four: 7.16)
                if (((mask >> j) & 3u) == 3u) {
                    accumulate_rows<ST, SUM, PAIRS, PH, true>(sm, rs.rt, j0 + j, &w[0][j], p0, p2, a0,
                                                              a1, U, RE, IM, CRE, CIM);
                    ++j;
                    accumulate_rows<ST, SUM, PAIRS, PH, true>(sm, rs.rt, j0 + j, &w[0][j], p0, p2, a0,
                                                              a1, U, RE, IM, CRE, CIM);
                } else if ((mask >> j) & 1u) {
                    accumulate_rows<ST, SUM, PAIRS, PH, true>(sm, rs.rt, j0 + j, &w[0][j], p0, p2, a0,
                                                              a1, U, RE, IM, CRE, CIM);
                } else if (accumulate_rows<ST, SUM, PAIRS, PH, false>(sm, rs.rt, j0 + j, nullptr, p0, p2,
                                                                      a0, a1, U, RE, IM, CRE, CIM)) {
                    correct_rows<SUM, PAIRS, false>(sm, rs.rt, j0 + j, p0, p2, a0, a1, U, RE, IM, CRE, CIM);
                }
            }
            __syncwarp();  // the next 32 sources' polynomials replace these
        }
    } else {
        constexpr int G = PH == kPhaseRef ? 1 : source_group<ST, PAIRS>();
        int j = 0;
        if constexpr (G > 1) {
#pragma unroll 1
            for (; j + G <= cnt; j += G) {
                bool near = false;
#pragma unroll
                for (int u = 0; u < G; ++u)
                    near |= accumulate_rows<ST, SUM, PAIRS, PH, false>(sm, rs.rt, j + u, nullptr, p0, p2,
                                                                       a0, a1, U, RE, IM, CRE, CIM);
                if (near) {
#pragma unroll 1
                    for (int u = 0; u < G; ++u)
                        correct_rows<SUM, PAIRS, false>(sm, rs.rt, j + u, p0, p2, a0, a1, U, RE, IM, CRE, CIM);
                }
            }
        }
#pragma unroll 1
        for (; j < cnt; ++j)
            if (accumulate_rows<ST, SUM, PAIRS, PH, false>(sm, rs.rt, j, nullptr, p0, p2, a0, a1, U, RE,
                                                           IM, CRE, CIM) ||
                (PH == kPhaseRef && tile_long))
                correct_rows<SUM, PAIRS, PH == kPhaseRef>(sm, rs.rt, j, p0, p2, a0, a1, U, RE, IM, CRE,
                                                          CIM);
    }
}

// Coordinate of index i along grid axis k (xyz index a), bit-identical to the reference's
// o + (i as f32 * res); a fixed axis (count 1) stays at its origin.
__device__ __forceinline__ float axis_coord(const GridDev& g, int k, int a, int64_t i) {
    const float o = pick3(g.origin[0], g.origin[1], g.origin[2], a);
    return g.count[k] > 1 ? __fadd_rn(o, __fmul_rn(__ll2float_rn(i), g.res)) : o;
}

// The grid indices of the calling thread's points in tile `tile`: first axis i0, second axis i1 ..
// i1 + ppt - 1, third axis i2 (any of them may lie past the grid's edge).
struct RowsCell {
    int64_t i0, i1, i2;
    __device__ __forceinline__ RowsCell(const RowsMap& map, int64_t tile, int ppt) {
        const int lane = threadIdx.x & 31;
        const int64_t wt = tile * (kThreads / 32) + (threadIdx.x >> 5);
        int64_t t0, t1, t2, rest;
        div_rem(wt, map.tiles0, rest, t0);
        div_rem(rest, map.tiles1, t2, t1);
        i0 = (t0 << map.bits[0]) + (lane & ((1 << map.bits[0]) - 1));
        i1 = ((t1 << map.bits[1]) +
              ((lane >> map.bits[0]) & ((1 << map.bits[1]) - 1))) * ppt;
        i2 = (t2 << map.bits[2]) + (lane >> (map.bits[0] + map.bits[1]));
    }
};

// One tile of the rows tiling: the sums of sources s_lo .. s_hi - 1 at the thread's points, in RE,
// IM (CRE, CIM: compensations).  MID: whether the mid phase tier is compiled in; without it, mid
// tiles take the careful variant.
template <int ST, int SUM, int PAIRS, bool MID = false>
__device__ __forceinline__ void rows_accumulate(RowsSmem& rs,
                                                const PackedSource* __restrict__ src,
                                                int64_t n, int64_t s_lo, int64_t s_hi,
                                                const GridDev& g, const RowsMap& map,
                                                int64_t tile, float2 (&RE)[PAIRS],
                                                float2 (&IM)[PAIRS], float2 (&CRE)[PAIRS],
                                                float2 (&CIM)[PAIRS]) {
    constexpr int kPPT = 2 * PAIRS;
    RowsTile& sm = rs.sm;
    const RowsCell cell(map, tile, kPPT);
    const int64_t c0 = g.count[0], c1 = g.count[1], c2 = g.count[2];
    const int64_t i1b = cell.i1;
    const int a0 = g.axis[0], a1 = g.axis[1], a2 = g.axis[2];
    // points past the grid's edges are computed at its last index, and never stored
    const float p0 = axis_coord(g, 0, a0, cell.i0 < c0 ? cell.i0 : c0 - 1);
    const float p2 = axis_coord(g, 2, a2, cell.i2 < c2 ? cell.i2 : c2 - 1);

    float2 U[PAIRS];
#pragma unroll
    for (int k = 0; k < kPPT; ++k) {
        const int64_t i1 = i1b + k < c1 ? i1b + k : c1 - 1;
        lane_of(U[k >> 1], k & 1) = axis_coord(g, 1, a1, i1);
    }
#pragma unroll
    for (int q = 0; q < PAIRS; ++q) {
        RE[q] = f2(0.f);
        IM[q] = f2(0.f);
        CRE[q] = f2(0.f);
        CIM[q] = f2(0.f);
    }

    // bounding box of the block's points in x, y, z (for the phase bound of each source tile)
    {
        float umin = U[0].x, umax = U[0].x;
#pragma unroll
        for (int k = 1; k < kPPT; ++k) {
            umin = fminf(umin, lane_of(U[k >> 1], k & 1));
            umax = fmaxf(umax, lane_of(U[k >> 1], k & 1));
        }
        float lo[3], hi[3];
        lo[0] = p0, hi[0] = p0, lo[1] = umin, hi[1] = umax, lo[2] = p2, hi[2] = p2;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
                hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
            }
        }
        if ((threadIdx.x & 31) == 0) {
            // grid-axis order (0: first, 1: second, 2: third) -> x, y, z slots
            const int ax[3] = {a0, a1, a2};
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                sm.box[threadIdx.x >> 5][ax[c]] = lo[c];
                sm.box[threadIdx.x >> 5][3 + ax[c]] = hi[c];
            }
        }
        __syncthreads();
        if (threadIdx.x < 6) {
            const int a = threadIdx.x;
            float v = sm.box[0][a];
#pragma unroll
            for (int w = 1; w < kThreads / 32; ++w)
                v = a < 3 ? fminf(v, sm.box[w][a]) : fmaxf(v, sm.box[w][a]);
            sm.bbox[a] = v;
        }
        __syncthreads();
    }

    for (int64_t s0 = s_lo; s0 < s_hi; s0 += kTile) {
        const int cnt = static_cast<int>((s_hi - s0) < kTile ? (s_hi - s0) : kTile);
        __syncthreads();
        bool small_phase = true, mid_phase = true, any_long = false;
        for (int j = threadIdx.x; j < cnt; j += kThreads) {
            const PackedSource s = src[s0 + j];
            bool is_long = false;
            if (ST == SRC_T4010A1) {
                const float lx = s.b.x >= 0.f ? sm.bbox[0] : sm.bbox[3];
                const float ly = s.b.y >= 0.f ? sm.bbox[1] : sm.bbox[4];
                const float lz = s.b.z >= 0.f ? sm.bbox[2] : sm.bbox[5];
                is_long = leaves_table(s.b.x, s.b.y, s.b.z,
                                       fmaf(s.b.z, lz - s.a.z, fmaf(s.b.y, ly - s.a.y, s.b.x * (lx - s.a.x))));
            }
            any_long = any_long || is_long;
            const float fx = fmaxf(fabsf(sm.bbox[0] - s.a.x), fabsf(sm.bbox[3] - s.a.x));
            const float fy = fmaxf(fabsf(sm.bbox[1] - s.a.y), fabsf(sm.bbox[4] - s.a.y));
            const float fz = fmaxf(fabsf(sm.bbox[2] - s.a.z), fabsf(sm.bbox[5] - s.a.z));
            const float rmax = sqrtf(fmaf(fz, fz, fmaf(fy, fy, fx * fx)));
            const float bound = fmaf(fabsf(s.a.w), rmax, fabsf(s.c.y));
            small_phase = small_phase && !is_long && bound <= kUnreducedPhaseMax;
            mid_phase = mid_phase && !is_long && bound <= kMidPhaseMax;
            const float sv = pick3(s.a.x, s.a.y, s.a.z, a0), su = pick3(s.a.x, s.a.y, s.a.z, a1),
                        sw = pick3(s.a.x, s.a.y, s.a.z, a2);
            const float nv = pick3(s.b.x, s.b.y, s.b.z, a0), nu = pick3(s.b.x, s.b.y, s.b.z, a1),
                        nw = pick3(s.b.x, s.b.y, s.b.z, a2);
            sm.v[0][j] = make_float4(-su, -su, s.a.w, s.a.w);
            sm.v[1][j] = make_float4(s.b.w, s.b.w, s.c.x, s.c.x);
            sm.v[2][j] = make_float4(s.c.y, s.c.y, nu, nu);
            sm.v[3][j] = make_float4(-sv, -sw, nv, nw);
        }
        const bool tile_small = __syncthreads_and(small_phase);
        const bool tile_mid = __syncthreads_and(mid_phase);
        if (tile_small)
            rows_source_loop<ST, SUM, PAIRS, kPhaseFast>(cnt, rs, p0, p2, a0, a1, a2, U, RE, IM, CRE,
                                                         CIM);
        else if (MID && tile_mid)
            rows_source_loop<ST, SUM, PAIRS, kPhaseMid>(cnt, rs, p0, p2, a0, a1, a2, U, RE, IM, CRE,
                                                        CIM);
        else
            rows_source_loop<ST, SUM, PAIRS, kPhaseRef>(cnt, rs, p0, p2, a0, a1, a2, U, RE, IM, CRE,
                                                        CIM, ST == SRC_T4010A1 && __syncthreads_or(any_long));
    }
}

// Store the thread's sums of one tile of the rows tiling (field transform applied); points
// whose sum is NaN are then passed to fix_coincident with the n sources src.
template <int SUM, int PAIRS>
__device__ __forceinline__ void rows_store(const PackedSource* __restrict__ src, int64_t n,
                                           const GridDev& g, const RowsMap& map,
                                           int64_t tile, float2 (&RE)[PAIRS], float2 (&IM)[PAIRS], float2 (&CRE)[PAIRS],
                                           float2 (&CIM)[PAIRS], int field,
                                           void* __restrict__ out) {
    constexpr int kPPT = 2 * PAIRS;
    const RowsCell cell(map, tile, kPPT);
    const int64_t c0 = g.count[0], c1 = g.count[1];
    const int64_t i0 = cell.i0, i1b = cell.i1, i2 = cell.i2;
    if (i0 >= c0 || i2 >= g.count[2]) return;
    bool bad = false;
#pragma unroll
    for (int k = 0; k < kPPT; ++k) {
        const int64_t i1 = i1b + k;
        if (i1 >= c1) break;
        const int64_t p = (i2 * c1 + i1) * c0 + i0;
        float vr = lane_of(RE[k >> 1], k & 1);
        float vi = lane_of(IM[k >> 1], k & 1);
        if constexpr (SUM == SUM_COMPENSATED) {
            vr = __fadd_rn(vr, lane_of(CRE[k >> 1], k & 1));
            vi = __fadd_rn(vi, lane_of(CIM[k >> 1], k & 1));
        }
        bad |= isnan(vr) || isnan(vi);
        store_field(out, p, field, vr, vi);
    }
    if (bad) {
#pragma unroll 1
        for (int k = 0; k < kPPT; ++k) {
            const int64_t i1 = i1b + k;
            if (i1 >= c1) break;
            const int64_t p = (i2 * c1 + i1) * c0 + i0;
            float x, y, z;
            grid_point(g, p, x, y, z);
            fix_coincident(src, n, x, y, z, p, field, out);
        }
    }
}

// The partial sums of one tile of the rows tiling, without the field transform, at its points of
// `part` (one entry per grid point).
template <int PAIRS>
__device__ __forceinline__ void rows_store_partial(const GridDev& g, const RowsMap& map,
                                                   int64_t tile, float2 (&RE)[PAIRS],
                                                   float2 (&IM)[PAIRS], float2* __restrict__ part) {
    constexpr int kPPT = 2 * PAIRS;
    const RowsCell cell(map, tile, kPPT);
    const int64_t c0 = g.count[0], c1 = g.count[1];
    if (cell.i0 >= c0 || cell.i2 >= g.count[2]) return;
#pragma unroll
    for (int k = 0; k < kPPT; ++k) {
        const int64_t i1 = cell.i1 + k;
        if (i1 >= c1) break;
        part[(cell.i2 * c1 + i1) * c0 + cell.i0] =
            make_float2(lane_of(RE[k >> 1], k & 1), lane_of(IM[k >> 1], k & 1));
    }
}

// One tile of the rows tiling, all n sources, stored.
template <int ST, int SUM, int PAIRS, bool MID = false>
__device__ __forceinline__ void block_rows(RowsSmem& rs, const PackedSource* __restrict__ src,
                                           int64_t n, const GridDev& g, const RowsMap& map,
                                           int64_t tile, int field, void* __restrict__ out) {
    float2 RE[PAIRS], IM[PAIRS], CRE[PAIRS], CIM[PAIRS];
    rows_accumulate<ST, SUM, PAIRS, MID>(rs, src, n, 0, n, g, map, tile, RE, IM, CRE, CIM);
    rows_store<SUM, PAIRS>(src, n, g, map, tile, RE, IM, CRE, CIM, field, out);
}

}  // namespace fb
}  // namespace afc
