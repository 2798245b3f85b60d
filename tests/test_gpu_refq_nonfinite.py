"""Filtered rows with samples that are not finite through wfbp_backproject on
reference-layout rows: a sample enters the voxels whose view and row it is in
and no other, so every voxel that k_bp (a captured call; it also lets rows
beyond the detector's edges in with weight 0) leaves finite is finite, with k_bp's
value to the rounding of sums of the same terms (2 (P / 2) u pi max|row|,
u = 2^-24). Rows of NaN at the detector's first and last row and single channels
at its ends, where a tile's columns beyond the channels have no sample."""
import math

import pytest

from freect_b200 import abi_types as T
from freect_b200 import scans, wfbp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("precision", [T.PRECISION_FP32, T.PRECISION_MIXED])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("nr,nx,n_slices,where", [(8, 64, 12, "last"), (8, 64, 12, "first"), (16, 40, 9, "last"),
                                                  (8, 64, 12, "channel"), (13, 200, 20, "last")])
def test_nonfinite_samples(nr, nx, n_slices, where, value, precision):
    spec = scans.tiny(nch=96, nr=nr, P=48, rotations=4, nx=nx, n_slices=n_slices)
    spec.fov = 520.0
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    ctx = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(precision=precision), device=0)
    ctx.set_views(tube, table)
    d = ctx.dims
    gen = torch.Generator(device=DEV).manual_seed(nr)
    rows = torch.randn((d.n_views, d.n_rows, d.n_channels), device=DEV, generator=gen)
    top = rows.abs().max().item()
    scales = None
    if precision == T.PRECISION_MIXED:
        rows, scales = rows.half(), torch.ones(d.n_views * d.n_rows, device=DEV)
    views = [d.n_views // 2, d.n_views // 2 + 7]
    for j in views:
        if where == "channel":
            rows[j, :, 0] = value
            rows[j, :, -3:] = value
        else:
            rows[j, -1 if where == "last" else 0] = value
    got, ref = ctx.alloc("native"), ctx.alloc("native")
    ctx.backproject(rows, got, row_scales=scales)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        ctx.backproject(rows, ref, row_scales=scales)
    g.replay()
    torch.cuda.synchronize()
    ctx.check_device_status()
    ok = torch.isfinite(ref)
    assert ok.any()
    assert torch.isfinite(got[ok]).all()
    assert (got[ok] - ref[ok]).abs().max().item() <= 2 * 24 * 2.0 ** -24 * math.pi * top
