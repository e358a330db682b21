"""The blend's cull (csrc/fhtgs_cull.cuh), compiled with g++ and counted against what it may not lose.

For every Gaussian and tile the cull returns the sample groups that may hold a fragment and a depth
that no core fragment undercuts.  Here every sample of the tiles around a Gaussian is evaluated with
the blend's FP32 arithmetic (fused as in the kernel, both for the whole tile and its halves, all
three tile classes and group shapes), and each accepted fragment (rho^2 <= cutoff, alpha >= 1/255)
must lie in a reached group, each core fragment (alpha >= 1/20) at or behind the bound.  The two
approximate instructions are replaced by exact results pushed off by 2^-22 either way, more than
their documented error (rcp.approx.ftz: 1 ulp; sqrt.approx.ftz: 2^-23 relative).
"""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "foveatedhtgscudabackend_b200", "csrc")

WRAPPER = r"""
#include <cmath>
#include <cstring>
#include <algorithm>
#include <cuda_runtime.h>
using std::isfinite; using std::max; using std::min;
static float g_push = 0.0f;  // relative error of the approximate instructions
static inline float host_logf(float x) { return std::log(x); }
#define __logf host_logf
static inline float rsqrtf(float x) { return 1.0f / std::sqrt(x); }
static inline int clip_int(float x) { return x != x ? 0 : x >= 2147483648.0f ? 2147483647 : x <= -2147483648.0f ? (-2147483647 - 1) : int(x); }
static inline int __float2int_ru(float x) { return clip_int(std::ceil(x)); }
static inline int __float2int_rd(float x) { return clip_int(std::floor(x)); }
static inline float ftz(float x) { return std::fabs(x) < 1.17549435e-38f ? std::copysign(0.0f, x) : x; }
namespace fhtgs { namespace host {
static inline float rcp_approx(float x) { return ftz(float((1.0 / double(ftz(x))) * (1.0 + g_push))); }
static inline float sqrt_approx(float x) { return ftz(float(std::sqrt(double(ftz(x))) * (1.0 + g_push))); }
} }
#define FHTGS_FLAVOR host
#include "fhtgs_cull.cuh"
using namespace fhtgs;
using namespace fhtgs::host;

extern "C" float core_cutoff() { return kCoreCutoff; }

static float mulsub(float a, float b, float c, float d) { return std::fma(a, b, -(c * d)); }
static float dot3(float3 a, float3 b) { return std::fma(a.z, b.z, std::fma(a.x, b.x, a.y * b.y)); }
static float3 cross3(float3 a, float3 b) {
    return make_float3(mulsub(a.y, b.z, a.z, b.y), mulsub(a.z, b.x, a.x, b.z), mulsub(a.x, b.y, a.y, b.x));
}

struct Counts { long long fragments, lost, core, undercut, reached, groups; };

// The Gaussian in the tile at (ox, oy): its samples against the cull of the tile (PX 2) and of its
// halves (PX 1).
template <int RW, int CLS, int PX>
static void check(const float4 P1, const float4 P2, const float4 P4, float opacity, int ox, int oy, Counts& n) {
    using G = GroupShape<RW, CLS>;
    constexpr int NG = CLS == 2 ? 1 : G::COLS * G::ROWS * PX / 2, ROWS_USED = NG >= G::COLS ? NG / G::COLS : 1;
    for (int half = 0; half < (CLS == 2 ? 1 : 2 / PX); ++half) {
        const uint32_t valid = ((1u << NG) - 1u) << (half * NG);
        float zmin;
        const uint32_t m = reached_groups<RW, CLS, ROWS_USED>(P1, P2, P4, opacity, float(ox), float(oy),
                                                              half * NG / G::COLS, valid, zmin);
        for (int g = half * NG; g < (half + 1) * NG; ++g) {
            n.groups += 1;
            n.reached += (m >> g) & 1;
            for (int k = 0; k < 16; ++k) {
                const float px = float(ox + ((g % G::COLS) * G::GW + k % G::GW) * G::S);
                const float py = float(oy + ((g / G::COLS) * G::GH + k / G::GW) * G::S);
                const float3 nx = make_float3(std::fma(-P4.x, px, P1.x), std::fma(-P4.y, px, P1.y), std::fma(-P4.z, px, P1.z));
                const float3 ny = make_float3(std::fma(-P4.x, py, P2.x), std::fma(-P4.y, py, P2.y), std::fma(-P4.z, py, P2.z));
                const float wx = std::fma(-P4.w, px, P1.w), wy = std::fma(-P4.w, py, P2.w);
                const float3 mm = make_float3(mulsub(wx, ny.x, nx.x, wy), mulsub(wx, ny.y, nx.y, wy), mulsub(wx, ny.z, nx.z, wy));
                const float3 d = cross3(nx, ny);
                const float num = dot3(mm, mm), den = dot3(d, d);
                if (num > kMaxCutoffSq * den) continue;
                const float rcp = 1.0f / den;
                const float alpha = std::fmin(opacity * std::exp(-0.5f * num * rcp), kMaxFragmentAlpha);
                if (alpha < kMinAlpha) continue;
                n.fragments += 1;
                if (!((m >> g) & 1)) { n.lost += 1; continue; }
                if (alpha < kMinAlphaCore) continue;
                const float3 e = cross3(d, mm);
                const float depth = dot3(make_float3(P4.x, P4.y, P4.z), make_float3(e.x * rcp, e.y * rcp, e.z * rcp)) + P4.w;
                n.core += 1;
                n.undercut += depth < zmin;
            }
        }
    }
}

template <int RW, int CLS>
static void both(const float4 P1, const float4 P2, const float4 P4, float o, int ox, int oy, Counts& n) {
    check<RW, CLS, 2>(P1, P2, P4, o, ox, oy, n);
    if constexpr (CLS != 2) check<RW, CLS, 1>(P1, P2, P4, o, ox, oy, n);
}

// n records (P1, P2, P4: 12 floats), opacities, and per record `per` tile origins.
extern "C" void cull_counts(const float* rec, const float* opacity, const int* origin, int n, int per, float push,
                            long long* out) {
    g_push = push;
    Counts c = {};
    for (int i = 0; i < n; ++i) {
        float4 P[3];
        std::memcpy(P, rec + 12 * i, sizeof(P));
        for (int t = 0; t < per; ++t) {
            const int ox = origin[2 * (i * per + t)], oy = origin[2 * (i * per + t) + 1];
            both<8, 0>(P[0], P[1], P[2], opacity[i], ox, oy, c);
            both<16, 0>(P[0], P[1], P[2], opacity[i], ox, oy, c);
            both<4, 0>(P[0], P[1], P[2], opacity[i], ox, oy, c);
            both<8, 1>(P[0], P[1], P[2], opacity[i], ox, oy, c);
            both<16, 1>(P[0], P[1], P[2], opacity[i], ox, oy, c);
            both<4, 1>(P[0], P[1], P[2], opacity[i], ox, oy, c);
            both<8, 2>(P[0], P[1], P[2], opacity[i], ox, oy, c);
        }
    }
    std::memcpy(out, &c, sizeof(c));
}
"""


@pytest.fixture(scope="module")
def cull(tmp_path_factory):
    d = tmp_path_factory.mktemp("cull")
    src = d / "cull.cpp"
    src.write_text(WRAPPER)
    so = d / "libcull.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-mfma", "-ffp-contract=off", "-w", "-shared", "-fPIC", "-I" + CSRC,
                    "-I/usr/local/cuda/include", str(src), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.core_cutoff.restype = C.c_float
    f32, i32, i64 = (np.ctypeslib.ndpointer(t, flags="C") for t in (np.float32, np.int32, np.int64))
    lib.cull_counts.argtypes = [f32, f32, i32, C.c_int, C.c_int, C.c_float, i64]
    return lib


def records(kind: str, n: int, rng, width: int, height: int):
    """P1, P2, P4 rows of n Gaussians before a pinhole camera, their opacities and depths > 0.2."""
    f = 0.5 * height / math.tan(math.radians(30.0))
    pos = rng.normal(size=(n, 3))
    pos *= 2.0 / np.abs(pos).max()
    pos[:, 2] += {"inside": 0.5, "near": 2.2}.get(kind, 6.0)
    s = np.exp(rng.normal(size=(n, 3)) * 0.5 - 4.5)
    if kind == "needles":
        s[:, 0] *= 30.0
        s[:, 1:] *= 0.03
    elif kind == "subpixel":
        s *= 10.0 ** rng.uniform(-4.0, -1.0, (n, 1))
    elif kind == "huge":
        s *= 12.0
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    r, x, y, z = q.T
    R = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - r * z), 2 * (x * z + r * y), 2 * (x * y + r * z),
                  1 - 2 * (x * x + z * z), 2 * (y * z - r * x), 2 * (x * z - r * y), 2 * (y * z + r * x),
                  1 - 2 * (x * x + y * y)], 1).reshape(n, 3, 3)
    T = np.concatenate([R * s[:, None, :], pos[:, :, None]], 2)
    VP = np.array([[f, 0, 0.5 * width], [0, f, 0.5 * height], [0, 0, 1]])
    P = np.einsum("rk,nkc->nrc", VP, T).astype(np.float32)
    opacity = 1.0 / (1.0 + np.exp(-1.5 * rng.normal(size=n)))
    if kind == "faint":
        opacity = np.where(rng.random(n) < 0.5, rng.uniform(1 / 254.9, 1 / 240, n), rng.uniform(0.049, 0.052, n))
    keep = P[:, 2, 3] > 0.2
    return P[keep], opacity[keep].astype(np.float32)


@pytest.mark.parametrize("size", [(523, 411), (2064, 2208), (16384, 16384)])
@pytest.mark.parametrize("kind", ["plain", "needles", "subpixel", "huge", "faint", "near", "inside"])
def test_no_fragment_outside_the_reached_groups(cull, kind, size):
    width, height = size
    rng = np.random.default_rng(width + len(kind))
    P, opacity = records(kind, 1500, rng, width, height)
    n, per = len(P), 6
    # tiles at the projected mean and around it, near and up to a footprint away
    w = P[:, 2, 3:4]
    mean = P[:, :2, 3] / w
    reach = 3.5 * np.sqrt((P[:, :2, :3] ** 2).sum(2)) / w + 16.0
    at = mean[:, None, :] + rng.uniform(-1.0, 1.0, (n, per, 2)) * reach[:, None, :] * np.linspace(0.0, 1.0, per)[None, :, None]
    origin = (np.clip(np.nan_to_num(at), 0, np.array(size) - 1) // 16 * 16).astype(np.int32)
    total = np.zeros(6, np.int64)
    for push in (2.0 ** -22, -(2.0 ** -22)):
        out = np.zeros(6, np.int64)
        cull.cull_counts(np.ascontiguousarray(P.reshape(n, 12)), opacity, np.ascontiguousarray(origin), n, per, push, out)
        total += out
    fragments, lost, core, undercut, reached, groups = (int(x) for x in total)
    print(f"{kind} {size}: {fragments} fragments ({core} core), {lost} lost, {undercut} under the bound, "
          f"{reached / groups:.3f} of the groups reached")
    assert fragments > 100  # (sub-pixel Gaussians seldom hold a sample)
    assert lost == 0 and undercut == 0


def test_core_cutoff_bounds_the_core_radius(cull):
    """A core fragment needs rho^2 <= 2 ln(20 opacity) = rc - 2 ln(255 / 20): what is taken off rc may
    not exceed that, and by no more than float spacing falls short of it."""
    exact = 2.0 * math.log(255.0 / 20.0)
    assert exact - 2e-6 <= cull.core_cutoff() <= exact
