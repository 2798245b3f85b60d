"""k_rebin_adjoint at the edges of its split (blocks of 128 raw channels, threads of 8
rows): channel counts around the block, row counts around the thread's, against
the FP64 oracle's adjoint with test_gpu_adjoint's bound (1e-4 of the largest value).
"""
import numpy as np
import pytest

from freect_b200 import scans, wfbp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("nch,nr", [(96, 2), (127, 7), (128, 8), (129, 9), (257, 17)])
def test_rows_and_channels(orc, nch, nr):
    spec = scans.tiny(nch=nch, nr=nr, P=48, rotations=3, nx=16, n_slices=2)
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    ctx = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(), device=0)
    ctx.set_views(tube, table)
    d = ctx.dims
    g = np.random.default_rng(nch).standard_normal((d.n_views, d.n_rows, d.n_channels)).astype(np.float32)
    out = torch.full((d.n_readings, d.raw_rows, d.raw_channels), float("nan"), device=DEV)
    ctx.rebin_adjoint(torch.from_numpy(g).to(DEV), out)
    torch.cuda.synchronize()
    ctx.check_device_status()
    ref = orc.rebin_adjoint_f64(cg, g)
    assert np.abs(out.cpu().numpy() - ref).max() <= 1e-4 * np.abs(ref).max()
