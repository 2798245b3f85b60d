"""A reconstruction grid that reaches past the source's orbit: a tile corner
there has |p_hat| > the source's distance, where the arcsine of the slice range
of a view does not exist. A tile that also holds voxels inside the acquisition
field must keep its views: the voxels the reference kernel's form (k_bp, which a
captured call runs) leaves finite are finite, and as close to its volume as
sums of the same terms are (the bound of the reference layout's test: 2 (P / 2)
u pi max|row| for P / 2 angles of one rounding each, u = 2^-24).
"""
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
@pytest.mark.parametrize("nx,fov,x0,y0,nr", [(36, 900.0, 0.0, 250.0, 8), (36, 900.0, -250.0, 0.0, 16),
                                             (40, 1400.0, 30.0, -20.0, 8)])
def test_tiles_beyond_the_source(nx, fov, x0, y0, nr, precision):
    spec = scans.tiny(nch=96, nr=nr, P=96, rotations=4, nx=nx, n_slices=9)
    spec.fov = fov
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    rp = spec.recon_config()
    rp.x_origin, rp.y_origin = x0, y0
    ctx = wfbp.Context(cg, rp, wfbp.make_ext(precision=precision), device=0)
    ctx.set_views(tube, table)
    ctx.bp_config()  # a tile fits: the staged kernel runs
    raw = torch.empty((spec.V, spec.nr, spec.nch), dtype=torch.float32, device=DEV)
    wfbp.synth_project(spec.synth(), spec.ellipsoids(), raw)
    reb, rows = ctx.alloc("rebinned"), ctx.alloc("filtered")
    sc = ctx.alloc("row_scales") if precision == T.PRECISION_MIXED else None
    ctx.rebin(raw, reb)
    ctx.filter(reb, rows, row_scales=sc)
    ref, got = ctx.alloc("native"), ctx.alloc("native")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        ctx.backproject(rows, ref, row_scales=sc)
    g.replay()
    ctx.backproject(rows, got, row_scales=sc)
    want, run = ctx.alloc("volume"), ctx.alloc("volume")
    ctx.thicken(ref, want)
    ctx.run(raw, run)
    torch.cuda.synchronize()
    ctx.check_device_status()
    assert (torch.isfinite(ref) & (ref != 0)).sum() > 100
    assert torch.equal(torch.isnan(got), torch.isnan(ref))
    assert torch.equal(torch.isnan(run), torch.isnan(want))
    full = rows.double() if sc is None else rows.double() * sc.double().view(rows.shape[0], rows.shape[1], 1)
    tol = 2 * (spec.P // 2) * 2.0 ** -24 * math.pi * full.abs().max().item()
    assert (got - ref).nan_to_num(0.0).abs().max().item() <= tol
