"""Instance creation where a block loops over several chunks of Gaussians (GPU).

A frame of many views has fewer creation blocks a view than chunks of 256 Gaussians; the same view
alone has one block a chunk and never loops.  The stored instances and the images must agree bit for
bit (tolerance: none), with bounds of one tile, of up to 16 (a thread's own) and of more (a warp's),
and a last chunk that is not full.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import foveatedhtgscudabackend_b200 as F  # noqa: E402
from foveatedhtgscudabackend_b200 import scene  # noqa: E402

VIEWS = 128


@pytest.mark.parametrize("n", [20_017, 10_240])
def test_looping_blocks_store_what_single_chunks_store(n):
    dev = torch.device("cuda", 0)
    blocks_per_view = -(-32 * torch.cuda.get_device_properties(dev).multi_processor_count // VIEWS)
    assert -(-n // 256) > blocks_per_view  # the batch loops, the single view does not
    g = scene.make_gaussians(n, 0, seed=5)
    g.scales[::3] *= np.float32(15.0)  # footprints of many tiles
    g.scales[1::3] *= np.float32(0.1)
    gt = F.gaussians_to_torch(g, dev)
    views = scene.make_batched_views(VIEWS, seed=2, resolutions=((170, 130), (208, 160), (33, 250)))
    st = [F.settings_from_view(v, K=4, active_sh_bases=1, device=dev) for v in views]
    r = F.Renderer(dev)
    many = [x.clone() for x in r.render(*gt, st)]
    picked = (0, 1, VIEWS // 2, VIEWS - 1)
    loop = {i: r.intermediates(i) for i in picked}
    for i in picked:
        one = r.render(*gt, [st[i]])[0]
        alone = r.intermediates(0)
        assert alone["n_instances_stored"] == loop[i]["n_instances_stored"] > n
        bounds = alone["screen_bounds"].astype(int)
        tiles = (bounds[:, 1] - bounds[:, 0]) * (bounds[:, 3] - bounds[:, 2])
        assert (tiles > 16).any() and ((tiles > 1) & (tiles <= 16)).any()
        for what in ("keys", "values", "instance_ranges"):
            assert np.array_equal(alone[what], loop[i][what]), f"view {i}: {what}"
        assert torch.equal(one, many[i]), f"view {i}"
    r.close()
