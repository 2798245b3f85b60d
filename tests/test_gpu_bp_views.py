"""The lists of views that a lane of the staged backprojection walks, at the
edges of their rule: no list (every staged view reaches every slice), lists of
a few views, stages of more views than a list can name, slabs of 16 and of 32
slices, a last slab of one slice, descending slices. A view off a lane's list
gives that slice exactly nothing, so the launch shapes (whose slabs stage
different views) must agree bit for bit; against the FP32 transcript the parity
test's 0.05 HU RMS holds, for mixed precision against the FP32 volume
test_gpu_mixed's 1 HU RMS. There is no bound on the largest difference from the
transcript: in the first of these scans one view's sample of one voxel lies on
a detector edge and falls on the other side of it in the transcript, which is
worth 2.3 HU in the two slices around it, with lists and without.
"""
import numpy as np
import pytest

from freect_b200 import abi_types as T
from freect_b200 import scans, wfbp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("feed,rotations,n_slices,pitch", [(9.6, 4, 33, 0.5), (4.8, 8, 33, 0.5), (4.0, 8, 17, 0.9),
                                                           (3.0, 11, 34, 0.5), (2.0, 16, 20, 0.5), (9.6, 4, 3, -0.7)])
def test_view_lists(orc, feed, rotations, n_slices, pitch):
    spec = scans.tiny(nch=96, nr=8, P=64, rotations=rotations, nx=40, n_slices=n_slices)
    spec.feed, spec.slice_thickness, spec.slice_pitch = feed, abs(pitch), abs(pitch)
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    raw = orc.synth_project(spec.synth(), spec.ellipsoids())
    ref = orc.reconstruct_ref32(spec, raw, q8=False)["volume"]
    raw_d, base = torch.from_numpy(raw).to(DEV), None
    for precision in (T.PRECISION_FP32, T.PRECISION_MIXED):
        ctx = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(precision=precision), device=0)
        ctx.set_views(tube, table)
        if pitch < 0:
            nat, req = ctx.slices()
            ctx.set_slices(nat[::-1].copy(), req[::-1].copy())
        first = None
        for cfg in [None] + list(ctx.bp_configs()):
            if cfg is not None:
                ctx.set_bp_config(cfg)
            v = ctx.alloc("volume")
            ctx.run(raw_d, v)
            torch.cuda.synchronize()
            ctx.check_device_status()
            v = v.cpu().numpy()
            if first is None:
                first = v
            assert np.array_equal(v, first, equal_nan=True), cfg and cfg.key()
        ctx.close()
        got = first[::-1] if pitch < 0 else first
        if base is None:
            rms, _, n = orc.hu_error(got, ref)
            assert n > 0.5 * got.size and rms <= 0.05
            base = got
        else:
            rms, _, n = orc.hu_error(got, base)
            assert n > 0.5 * got.size and rms <= 1.0
