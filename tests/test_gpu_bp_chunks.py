"""Backprojection in chunks of half-turn angles (a cluster of CTAs per column
tile; work items of a persistent batch): the chunk sums must be added in the
same order by every launch shape, by a window of slices and by the batch, and
the volume must stay within the parity bound of the transcript (0.05 HU RMS,
1 HU max, as test_gpu_parity's stage test). Sizes around the rule's edges: one
tile, several tiles, matrices that leave tile columns empty or outside the field
of view, fewer angles than chunks could use, and a matrix without chunks.
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


def setup(orc, nx, ny, P, nr, n_slices, fov, precision):
    spec = scans.tiny(nch=96, nr=nr, P=P, rotations=4, nx=nx, n_slices=n_slices)
    spec.ny, spec.fov = ny, fov
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    ext = wfbp.make_ext(precision=precision)
    raw = torch.from_numpy(orc.synth_project(spec.synth(), spec.ellipsoids())).to(DEV)

    def ctx():
        c = wfbp.Context(cg, spec.recon_config(), ext, device=0)
        c.set_views(tube, table)
        return c
    return spec, ctx, raw


def run(c, raw):
    v = c.alloc("volume")
    c.run(raw, v)
    torch.cuda.synchronize()
    c.check_device_status()
    return v.cpu().numpy()


@pytest.mark.parametrize("precision", [T.PRECISION_FP32, T.PRECISION_MIXED])
@pytest.mark.parametrize("nx,ny,P,nr,n_slices,fov", [(8, 16, 96, 8, 3, 60.0), (33, 17, 130, 5, 6, 250.0),
                                                     (40, 40, 14, 8, 5, 250.0), (64, 48, 300, 16, 9, 520.0),
                                                     (160, 150, 64, 8, 12, 250.0)])
def test_chunks_same_order_everywhere(orc, nx, ny, P, nr, n_slices, fov, precision):
    spec, make, raw = setup(orc, nx, ny, P, nr, n_slices, fov, precision)
    c = make()
    ref = run(c, raw)
    assert np.isfinite(ref).mean() > 0.5
    for cfg in c.bp_configs():
        c.set_bp_config(cfg)
        assert np.array_equal(run(c, raw), ref, equal_nan=True), cfg.key()
    # a window of the slices, as a shard reconstructs it
    nat, req = c.slices()
    w = make()
    keep = req[1:-1] if req.size > 2 else req
    near = nat[(nat > keep.min() - spec.slice_thickness) & (nat < keep.max() + spec.slice_thickness)]
    w.set_slices(near, keep)
    assert np.array_equal(run(w, raw), ref[1:-1] if req.size > 2 else ref, equal_nan=True)
    # the batch, from device and host buffers
    cs = [make(), make()]
    b = wfbp.Batch(cs)
    vols = [x.alloc("volume") for x in cs]
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        b.run([raw, raw], vols)
    s.synchronize()
    b.check_device_status()
    host = [torch.empty(ref.shape, dtype=torch.float32, pin_memory=True) for _ in cs]
    b.run_host([raw.cpu().pin_memory()] * 2, host)
    for v in vols + host:
        assert np.array_equal(v.cpu().numpy(), ref, equal_nan=True)
    out = torch.empty(ref.shape, dtype=torch.float32, pin_memory=True)
    assert np.array_equal(make().run_host(raw.cpu().pin_memory(), out).numpy(), ref, equal_nan=True)


@pytest.mark.parametrize("nx,P", [(24, 96), (64, 200)])
def test_chunks_against_transcript(orc, nx, P):
    spec, make, raw = setup(orc, nx, nx, P, 8, 5, 250.0, T.PRECISION_FP32)
    got = run(make(), raw)
    ref = orc.reconstruct_ref32(spec, raw.cpu().numpy(), q8=False)["volume"]
    rms, mx, n = orc.hu_error(got, ref)
    assert n > 0.9 * got.size and rms <= 0.05 and mx <= 1.0
