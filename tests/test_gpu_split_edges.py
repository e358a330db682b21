"""The split blend at the image's edge (GPU): a tile that the edge cuts has samples outside the
image.  They are walked with their group but resolve to nothing, so what they record may neither
count as a record overflow (which would blend the whole tile again) nor show in the statistics.
"""
import dataclasses

import numpy as np
import pytest
import torch

import foveatedhtgscudabackend_b200 as F
from foveatedhtgscudabackend_b200 import scene

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)
INSIDE = 1  # columns (or rows) of the last tile that lie inside the image


def spot(view: scene.View, x: float, y: float, n: int, sigma_px: float, seed: int) -> scene.Gaussians:
    """n round Gaussians of one pixel size about pixel (x, y), at random depths, in random order."""
    rng = np.random.default_rng(seed)
    g = scene.make_gaussians(n, 0, seed)
    z = rng.uniform(4.0, 8.0, n)
    px, py = x + rng.uniform(-0.2, 0.2, n), y + rng.uniform(-0.2, 0.2, n)
    cam = np.stack([(px - view.center_x) / view.focal_x * z, (py - view.center_y) / view.focal_y * z, z], 1)
    g.positions[:] = (cam - view.M[:, 3]) @ view.M[:, :3]  # view = R p + t
    g.scales[:] = (sigma_px * z / view.focal_x)[:, None]
    g.opacities[:] = 0.9
    return g


@pytest.mark.parametrize("axis", ["right", "bottom"])
@pytest.mark.parametrize("K", [1, 8])
def test_samples_outside_the_image_record_nothing(axis, K):
    full = scene.make_view(320, 240)
    # the same camera, the last tile cut after INSIDE columns (rows): the spot lies two samples
    # further, in the same 4x4 group, and its cutoff radius (1 px) does not reach the image
    cut = 16 - INSIDE
    view = dataclasses.replace(full, **({"width": 320 - cut} if axis == "right" else {"height": 240 - cut}))
    at = (view.width + 1.0, 88.0) if axis == "right" else (88.0, view.height + 1.0)
    gt = F.gaussians_to_torch(spot(full, *at, 3000, 0.3, K), DEV)
    out = []
    for share, v in ((0.0, view), (0.1, view), (0.1, full)):
        r = F.Renderer(DEV)
        r.set_foveation("none")
        r.set_blend_split(share, 1)
        img = r.render(*gt, [F.settings_from_view(v, K=K, active_sh_bases=1, device=DEV)])[0].clone()
        out.append((img, r.blend_split_stats() if share else None))
        r.close()
    (whole, _), (split, stats), (_, all_inside) = out
    # inside the image the same spot overflows its one record: the cut view's tile is split too
    assert all_inside["split_tiles"] == 1 and all_inside["max_records"] > 1 and all_inside["whole_fallbacks"] == 1
    assert stats["split_tiles"] == 1
    assert stats["max_records"] == 0 and stats["whole_fallbacks"] == 0
    assert torch.equal(whole, split)
