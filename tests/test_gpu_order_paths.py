"""The two walks of a tile against each other (GPU): whole or as two halves (full-resolution and
periphery tiles), among sixteen or alone on a warp (quarter tiles).

The work order takes a tile apart when its list is long against the frame's instances, so the same
view is rendered alone, where its long lists are taken apart, and in a batch of copies, where none
is.  That they are, and are not, is asserted from the lists and the order's own constants.  Both
walks evaluate the same pairs with the same operations in the same order: the images agree bit for
bit (tolerance: none), for all three group shapes and both math flavours.
"""
import os
import re

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import foveatedhtgscudabackend_b200 as F  # noqa: E402
from foveatedhtgscudabackend_b200 import scene  # noqa: E402

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MANY = 250  # copies of the view in the batch
# every tile of one class: foveation, its ring radii, the factor of its list in the order's rule
CLASSES = {"full": ("none", (0.15, 0.4), None), "periphery": ("rings", (0.0, 100.0), "kCostLow"),
           "quarter": ("rings", (0.0, 0.0), "kCostQuarter")}


def constant(name: str) -> float:
    with open(os.path.join(ROOT, "foveatedhtgscudabackend_b200", "csrc", "fhtgs_order.h")) as f:
        return float(re.search(rf"\b{name} = ([0-9.]+)f", f.read()).group(1))


def longest_and_total(r, view) -> tuple[int, int]:
    """The view's longest tile list and its stored instances, from the Gaussians' tile bounds."""
    m = r.intermediates(0)
    gw, gh = view.grid_large
    count = np.zeros((gh, gw), np.int64)
    for (x0, x1, y0, y1), n in zip(m["screen_bounds"].astype(int), m["n_touched"]):
        if n:
            count[y0:y1, x0:x1] += 1
    assert count.sum() == m["n_instances_stored"]
    return int(count.max()), int(count.sum())


@pytest.mark.parametrize("K", [1, 8, 32])
@pytest.mark.parametrize("size", [(170, 130), (251, 171)])
@pytest.mark.parametrize("cls", sorted(CLASSES))
def test_whole_and_apart_agree(cls, size, K):
    foveation, rings, factor = CLASSES[cls]
    g = scene.make_gaussians(12_000, 1, seed=K)
    g.positions[:] = np.random.default_rng(K).uniform(-2.0, 2.0, g.positions.shape)  # no tile holds most instances
    g.opacities[::7] = np.float32(1.0)  # (K-buffer entries of alpha 1, and ties of evicted colours)
    dev = torch.device("cuda", 0)
    gt = F.gaussians_to_torch(g, dev)
    v = scene.make_view(*size, position=(0.3, 0.2, -5.0))
    st = F.settings_from_view(v, K=K, active_sh_bases=4, device=dev)
    r = F.Renderer(dev)
    r.set_foveation(foveation, *rings)
    r.render(*gt, [st])
    longest, total = longest_and_total(r, v)
    longest *= constant(factor) if factor else 1.0
    share = constant("kHalfShare") / torch.cuda.get_device_properties(dev).multi_processor_count
    assert longest > 1.01 * share * total            # alone: the longest list is taken apart
    assert longest < 0.99 * share * total * MANY     # in the batch: no list is
    for width in (8, 16, 4):
        r.set_tuning(blend_warp_width=width)
        for fast in (True, False):
            one = r.render(*gt, [st], fast_math=fast)[0].clone()
            many = r.render(*gt, [st] * MANY, fast_math=fast)
            for i in (0, MANY // 2, MANY - 1):
                assert torch.equal(one, many[i]), f"width {width}, fast {fast}, copy {i}"
    r.close()
