"""The blend's work items, group shapes and culling at their edges (GPU).

The three group rectangles (`blend_warp_width` 8: 4x4, 16: 8x2, 4: 2x8) cull different pairs, and
the frames below force every kind of work item: full-resolution tiles whole and as halves (a few
long lists), periphery tiles in fours and quarter tiles in sixteens with remainders, tiles cut by
the image edge.  Culling may only skip pairs that cannot contribute, so the images of the three
shapes are bit-identical (tolerance: none); against the FP32 oracle the repository's bar of 50 dB
holds.
"""
import numpy as np
import pytest

from helpers import REF_PSNR_DB, psnr

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import foveatedhtgscudabackend_b200 as F  # noqa: E402
from foveatedhtgscudabackend_b200 import scene  # noqa: E402
import oracle as O  # noqa: E402


def scene_of(kind: str, n: int, seed: int) -> scene.Gaussians:
    g = scene.make_gaussians(n, 1, seed)
    rng = np.random.default_rng(seed + 1)
    if kind == "needles":       # scale ratios up to 1e3
        g.scales[:, 0] *= 30.0
        g.scales[:, 1:] *= np.float32(0.03) * rng.uniform(0.5, 2.0, (n, 2)).astype(np.float32)
    elif kind == "subpixel":    # far below a pixel, some of them around 1e-10
        g.scales[:] = (g.scales * 10.0 ** rng.uniform(-8.0, -1.0, (n, 1))).astype(np.float32)
    elif kind == "huge":        # footprints over many tiles, the camera inside some
        g.scales[:] *= 12.0
    elif kind == "faint":       # opacities around 1/255 and 1/20
        g.opacities[:] = np.where(rng.random((n, 1)) < 0.5, rng.uniform(1 / 260, 1 / 240, (n, 1)),
                                  rng.uniform(0.04, 0.06, (n, 1))).astype(np.float32)
    elif kind == "centre":      # one dense spot: a few tiles hold most of the instances
        g.positions[: n // 2] *= np.float32(0.02)
    return g


def render_all(g, v, foveation, K, fast=True):
    dev = torch.device("cuda", 0)
    r = F.Renderer(dev)
    r.set_foveation(foveation)
    gt = F.gaussians_to_torch(g, dev)
    st = [F.settings_from_view(v, K=K, active_sh_bases=4, device=dev)]
    out = {}
    for width in (8, 16, 4):
        r.set_tuning(blend_warp_width=width)
        out[width] = r.render(*gt, st, fast_math=fast)[0].cpu().numpy()
    r.set_tuning(blend_blocks_per_sm=1)
    out["one block"] = r.render(*gt, st, fast_math=fast)[0].cpu().numpy()
    r.close()
    return out


@pytest.mark.parametrize("foveation", ["reference", "rings", "none"])
@pytest.mark.parametrize("kind", ["plain", "needles", "subpixel", "huge", "faint", "centre"])
def test_group_shapes_agree_bit_for_bit(kind, foveation):
    g = scene_of(kind, 6000, seed=11)
    v = scene.make_view(523, 411, position=(0.3, 0.2, -3.0), gaze_ndc=(0.2, -0.1))
    for fast in (True, False):
        out = render_all(g, v, foveation, K=4, fast=fast)
        for k in out:
            assert np.array_equal(out[8], out[k]), f"{kind}/{foveation}: shape {k} differs"


@pytest.mark.parametrize("K", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("size", [(1, 1), (16, 16), (17, 15), (250, 33), (401, 399)])
def test_items_vs_oracle(K, size):
    g = scene_of("centre", 3000, seed=K)
    v = scene.make_view(*size)
    for foveation in ("reference", "rings", "none"):
        img = render_all(g, v, foveation, K)[8]
        ref = O.render(g, v, K=K, active_sh_bases=4, precision=32, foveation=foveation)
        assert psnr(img, ref) >= REF_PSNR_DB, f"{foveation}: {psnr(img, ref):.1f} dB"


def test_degenerate_records_agree_bit_for_bit():
    """NaN and infinite attributes reach every pixel of their tiles whatever the group shape."""
    g = scene_of("plain", 500, seed=3)
    g.opacities[::50] = np.float32(np.inf)
    g.sh_0[5::60] = np.float32(np.nan)
    g.scales[7::70] = np.float32(0.0)
    v = scene.make_view(160, 120)
    out = render_all(g, v, "none", K=8)
    for k in out:
        assert np.array_equal(out[8], out[k], equal_nan=True)
