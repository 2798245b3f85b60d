"""A batch whose scans lay out a CTA's shared memory differently (few and many
detector rows, views per slab, half-turn angles): work items of one scan follow
items of another in the same persistent CTA, so that one tile's view slots lie
where the tile before had its records and lists. Every volume equals its scan's
own wfbp_run, in repeated runs."""
import numpy as np
import pytest

from freect_b200 import abi_types as T
from freect_b200 import scans, wfbp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)


@pytest.mark.parametrize("precision", [T.PRECISION_FP32, T.PRECISION_MIXED])
def test_alternating_layouts(precision):
    ctxs, raws, refs = [], [], []
    for i, (nr, P, nx, feed) in enumerate([(48, 60, 96, 28.8), (4, 64, 88, 2.0), (33, 40, 120, 12.0), (8, 90, 64, 4.8),
                                           (48, 52, 72, 20.0), (6, 72, 104, 2.4)]):
        spec = scans.tiny(nch=120 + 8 * i, nr=nr, P=P, rotations=4, nx=nx, n_slices=10 + i, seed=i)
        spec.feed = feed
        tube, table = spec.views()
        cg, _ = wfbp.configure_geometry(spec.meta(), table)
        c = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(precision=precision), device=0)
        c.set_views(tube, table)
        raw = c.alloc("raw")
        wfbp.synth_project(spec.synth(), spec.ellipsoids(), raw)
        v = c.alloc("volume")
        c.run(raw, v)
        torch.cuda.synchronize()
        ctxs.append(c)
        raws.append(raw)
        refs.append(v.cpu().numpy())
    batch = wfbp.Batch(ctxs)
    s = torch.cuda.Stream()
    for cfg in [batch.bp_config()] + batch.bp_configs()[-1:]:
        batch.set_bp_config(cfg)
        vols = [c.alloc("volume") for c in ctxs]
        for _ in range(3):
            with torch.cuda.stream(s):
                batch.run(raws, vols)
            s.synchronize()
            batch.check_device_status()
            for v, ref in zip(vols, refs):
                assert np.array_equal(v.cpu().numpy(), ref, equal_nan=True), cfg.key()
    batch.close()
