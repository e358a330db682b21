// The blend's cull: which groups of a tile's samples a Gaussian may reach, and a lower bound of the
// depth of its core fragments.  Apart from the two approximate instructions this is plain C++, so
// that the host can compile it (with its own rcp_approx, sqrt_approx and intrinsics) and count the
// fragments it would lose.
#pragma once
#include "fhtgs_math.cuh"
#include "fhtgs_types.cuh"

namespace fhtgs {
namespace FHTGS_FLAVOR {
using namespace fhtgs::vm;

#ifdef __CUDACC__
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
#endif

// Pixel-space bounding box of a Gaussian's cutoff ellipse (rc = 2 ln(255 opacity)), evaluated about
// the projected mean (x0 = P1.w / P4.w) so that no large terms cancel.  Returns false when the box is
// unbounded (camera inside the cutoff quadric or mean behind it): no culling then.
__device__ __forceinline__ bool cutoff_box(const float4 P1, const float4 P2, const float4 P4, float rc, float4& box) {
    if (!(P4.w > 0.0f) || !(rc > 0.0f)) return false;
    const float3 n4 = xyz(P4);
    const float a = P4.w * P4.w - rc * dot(n4, n4);
    if (!(a > 0.0f)) return false;
    const float ia = 1.0f / a;
    const float x0 = P1.w / P4.w, y0 = P2.w / P4.w;
    const float3 q1 = xyz(P1) - x0 * n4, q2 = xyz(P2) - y0 * n4;
    const float cx = -rc * dot(q1, n4) * ia, cy = -rc * dot(q2, n4) * ia;
    const float ex = sqrtf(fmaxf(cx * cx + rc * dot(q1, q1) * ia, 0.0f));
    const float ey = sqrtf(fmaxf(cy * cy + rc * dot(q2, q2) * ia, 0.0f));
    if (!(isfinite(ex) && isfinite(ey) && isfinite(x0) && isfinite(y0))) return false;
    const float mx = 1.0f + 1e-4f * (fabsf(x0) + ex), my = 1.0f + 1e-4f * (fabsf(y0) + ey);
    box = make_float4(x0 + cx - ex - mx, x0 + cx + ex + mx, y0 + cy - ey - my, y0 + cy + ey + my);
    return true;
}

// The cutoff ellipse of a Gaussian as a conic F(x', y') <= 0 about its projected mean
// (x' = x - x0, y' = y - y0).  With Q1 = VPMT1 - x0 VPMT4 and Q2 = VPMT2 - y0 VPMT4 (both with
// zero w) the blend's moment vector is m = w4 (y' q1 - x' q2) and its direction vector
// d = q1 x q2 + x' (q2 x n4) + y' (n4 x q1), so rho^2 <= rc  <=>
//   w4^2 |y' q1 - x' q2|^2 - rc |d|^2 <= 0.
// rc is inflated by kCullRcInflation and the rectangles by kCullPixelMargin, so that a
// rectangle reported empty holds no pixel the blend could accept.  Of the conic itself, measured on
// B200 over 1.8 G accepted fragments of five scenes (1M-Gaussian stereo 2064x2208, 100k SH0
// 1280x720, a camera inside a 300k cloud, 20k Gaussians 25x the benchmark size, 4096x1024):
// evaluated at the accepted pixel with rc not inflated it rejects 3,052 of them (float rounding of
// the blend's plane arithmetic); inflated by 0.1 % it rejects none.  0.5 % keeps 5x that margin; the
// 0.02 px covers the rounding of the interval's edges for sub-pixel ellipses.  Of reached_groups as
// a whole, counted on the CPU over 213 M accepted fragments (seven kinds of scene, 523x411 to
// 16384x16384, all classes and shapes, the approximate instructions pushed off by 2^-22 either
// way): none lies outside its reached groups, no core fragment before its depth bound.
constexpr float kCullRcInflation = 1.005f;
constexpr float kCullPixelMargin = 0.02f;

struct Conic {
    float x0, y0, A, B, C, D, E, F0, det;
};

__device__ __forceinline__ bool cutoff_conic(const float4 P1, const float4 P2, const float4 P4, float opacity, Conic& q) {
    const float rc = 2.0f * __logf(opacity * kMinAlphaRcp) * kCullRcInflation;
    const float3 n4 = xyz(P4);
    const float w4 = P4.w;
    if (!(rc > 0.0f) || !(w4 > 0.0f)) return false;
    q.x0 = P1.w / w4;
    q.y0 = P2.w / w4;
    const float3 q1 = xyz(P1) - q.x0 * n4, q2 = xyz(P2) - q.y0 * n4;
    const float3 c0 = cross(q1, q2), cx = cross(q2, n4), cy = cross(n4, q1);
    const float ww = w4 * w4;
    q.A = ww * dot(q2, q2) - rc * dot(cx, cx);
    q.C = ww * dot(q1, q1) - rc * dot(cy, cy);
    q.B = -2.0f * (ww * dot(q1, q2) + rc * dot(cx, cy));
    q.D = -2.0f * rc * dot(c0, cx);
    q.E = -2.0f * rc * dot(c0, cy);
    q.F0 = -rc * dot(c0, c0);
    q.det = 4.0f * q.A * q.C - q.B * q.B;
    // an ellipse, clearly: positive definite quadratic part
    return q.A > 0.0f && q.C > 0.0f && q.det > 1e-4f * (4.0f * q.A * q.C) && isfinite(q.det) && isfinite(q.F0) &&
           isfinite(q.D) && isfinite(q.E) && isfinite(q.x0) && isfinite(q.y0);
}

// 2 ln(255 / 20) = 2 ln(kMinAlphaRcp kMinAlphaCore) rounded down, so that rc - kCoreCutoff bounds
// 2 ln(20 opacity) from above.
constexpr float kCoreCutoff = 5.0910620f;

// How a tile's samples map onto threads.  A warp walks groups of 16 samples, each along its own
// list of the Gaussians that may reach the group's rectangle: four groups, one per 8 lanes with
// two samples a lane (PX 2), or two groups, one per 16 lanes (PX 1, half items).  CLS 0: a
// full-resolution tile (16 x 16 samples, 16 groups: the whole block, or half of them for a half
// item); CLS 1: a periphery tile (8 x 8 samples at stride 2, four groups, one warp); CLS 2: a
// ring-mode quarter tile (4 x 4 samples at stride 4, one group: a warp blends four tiles, or with
// PX 1 one whose list is long).
// RW (fhtgs_tuning.blend_warp_width) gives the group rectangle: 8: 4 x 4, 16: 8 x 2, 4: 2 x 8.
template <int RW, int CLS>
struct GroupShape {
    static constexpr int S = CLS == 0 ? 1 : CLS == 1 ? kStride : kQuarterStride;
    static constexpr int SIDE = kTileLarge / S;  // samples per tile row
    static constexpr int GW = CLS == 2 ? 4 : RW == 16 ? 8 : RW == 4 ? 2 : 4, GH = 16 / GW;
    static constexpr int COLS = SIDE / GW, ROWS = SIDE / GH;
};

// Which sample groups of the tile at pixel (ox, oy) the Gaussian may reach: bit row * COLS + col,
// among `valid`.  The cutoff ellipse about its centre is x = slope y +- hx sqrt(1 - (y / ymax)^2);
// its x extent over a row of groups gives that row's bits at once (one test per row of groups
// instead of one per group).  Ellipses that are not clearly ellipses, or out of the range of the
// approximate arithmetic (both math flavours use it here: it gates pairs within the margins and
// reaches no pixel), are tested by their bounding box; unbounded ones reach every group, and
// so do Gaussians so small (rc |d|^2 at the mean) that the blend's 1 / |d|^2 may overflow:
// 0 x inf makes their alpha 1 at any pixel of their tiles.
// Rows row0 .. row0 + ROWS_USED - 1 of groups are tested (a half item's).
// `zmin` receives a depth that no fragment of the core (alpha >= 1/20) undercuts: the depth is
// w4 + n4 . e with |e| = rho, and alpha >= 1/20 needs rho^2 <= 2 ln(20 opacity); 25 % of rho,
// 0.5 |n4| and 1e-4 w4 cover its rounding.
template <int RW, int CLS, int ROWS_USED>
__device__ __forceinline__ uint32_t reached_groups(const float4 P1, const float4 P2, const float4 P4, float opacity,
                                                   float ox, float oy, int row0, uint32_t valid, float& zmin) {
    using G = GroupShape<RW, CLS>;
    constexpr float fS = static_cast<float>(G::S);
    zmin = -3.402823466e+38f;
    const float rc = 2.0f * __logf(opacity * kMinAlphaRcp);
    if (rc < 0.0f) return 0u;  // alpha <= opacity < 1/255 everywhere
    const float3 n4 = xyz(P4);
    const float nn = dot(n4, n4);
    if (!(P4.w > 0.0f) || !(rc > 0.0f) || !(P4.w * P4.w - rc * nn > 0.0f)) return valid;
    Conic q;
    const bool ell = cutoff_conic(P1, P2, P4, opacity, q) && q.det > 1e-3f * (4.0f * q.A * q.C) && q.A < 1e30f &&
                     q.C < 1e30f && q.det < 1e30f && q.A > 1e-30f && q.C > 1e-30f && q.det > 1e-30f && q.F0 < -1e-28f;
    uint32_t m = 0u;
    if (ell) {
        const float idet = rcp_approx(q.det), i2a = 0.5f * rcp_approx(q.A), i2c = 0.5f * rcp_approx(q.C);
        const float xc = (q.B * q.E - 2.0f * q.C * q.D) * idet, yc = (q.B * q.D - 2.0f * q.A * q.E) * idet;
        const float Fc = -(q.F0 + 0.5f * (q.D * xc + q.E * yc));  // >= -F0 > 0
        const float ymax = sqrt_approx(4.0f * q.A * Fc * idet), xmax = sqrt_approx(4.0f * q.C * Fc * idet);
        const float iy = rcp_approx(ymax);
        const float hx = sqrt_approx(2.0f * Fc * i2a), slope = -q.B * i2a;
        const float ystar = -q.B * i2c * xmax;  // where the right extreme x = xmax lies
        const float X = q.x0 + xc - ox, Y = q.y0 + yc - oy;  // centre relative to the tile
        constexpr float pitch = static_cast<float>(G::GW * G::S), width = static_cast<float>((G::GW - 1) * G::S);
        constexpr float ipitch = 1.0f / pitch;
#pragma unroll
        for (int i = 0; i < ROWS_USED; ++i) {
            const int r = row0 + i;
            const float Y0 = static_cast<float>(r * G::GH) * fS - Y - kCullPixelMargin;
            const float Y1 = Y0 + static_cast<float>(G::GH - 1) * fS + 2.0f * kCullPixelMargin;
            const float a = fmaxf(Y0, -ymax), e = fminf(Y1, ymax);
            const float ta = a * iy, te = e * iy;
            const float ha = hx * sqrt_approx(fmaxf(1.0f - ta * ta, 0.0f)), he = hx * sqrt_approx(fmaxf(1.0f - te * te, 0.0f));
            const float R = ystar >= a && ystar <= e ? xmax : fmaxf(slope * a + ha, slope * e + he);
            const float L = -ystar >= a && -ystar <= e ? -xmax : fminf(slope * a - ha, slope * e - he);
            // columns whose samples [c pitch, c pitch + width] meet [X + L, X + R]
            const int c0 = max(0, __float2int_ru(fmaxf((X + L - kCullPixelMargin - width) * ipitch, -1.0f)));
            const int c1 = min(G::COLS - 1, __float2int_rd(fminf((X + R + kCullPixelMargin) * ipitch, 32.0f)));
            if (a <= e && c0 <= c1) m |= ((2u << c1) - (1u << c0)) << (r * G::COLS);
        }
        const float rho2 = rc - kCoreCutoff;  // 2 ln(20 opacity) = rc - 2 ln(255 / 20)
        if (rho2 < -0.01f) zmin = 3.402823466e+38f;  // opacity < 1/20: no core fragment
        else
            zmin = P4.w - (1.25f * sqrt_approx(fmaxf(rho2, 0.0f)) + 0.5f) * sqrt_approx(nn) - 1e-4f * P4.w;
        return m & valid;
    }
    const float ix = P1.w / P4.w, iy = P2.w / P4.w;
    const float3 c0 = cross(xyz(P1) - ix * n4, xyz(P2) - iy * n4);  // the direction vector d at the mean
    float4 box;
    if (!(rc * dot(c0, c0) > 1e-28f) || !cutoff_box(P1, P2, P4, rc, box)) return valid;
    for (int g = 0; g < G::COLS * G::ROWS; ++g) {
        const float ax0 = ox + static_cast<float>((g % G::COLS) * G::GW) * fS, ax1 = ax0 + static_cast<float>(G::GW - 1) * fS;
        const float ay0 = oy + static_cast<float>((g / G::COLS) * G::GH) * fS, ay1 = ay0 + static_cast<float>(G::GH - 1) * fS;
        if (box.y >= ax0 && box.x <= ax1 && box.w >= ay0 && box.z <= ay1) m |= 1u << g;
    }
    return m & valid;
}

}  // namespace FHTGS_FLAVOR
}  // namespace fhtgs
