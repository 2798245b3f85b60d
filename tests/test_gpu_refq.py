"""wfbp_backproject on reference-layout rows: the transposed, TMA-staged form
(k_bp_tma_refq) against k_bp, which a captured call still runs, on the same
rows: tile edges, odd and padded row counts, FP16 rows with scales, a table feed
so low that the reference's z cull binds, and chunked and unchunked matrices.

Both sum the same terms, at most dtheta max|row| each for P / 2 half-turn
angles, with one rounding per angle (u = 2^-24): the sums differ by at most
2 (P / 2) u times their terms' sum, pi max|row|. A sample that fell on the other
side of a detector edge would differ by its angle's whole term, 2 pi / P max|row|.
"""
import math

import numpy as np
import pytest

from freect_b200 import abi_types as T
from freect_b200 import scans, wfbp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("precision", [T.PRECISION_FP32, T.PRECISION_MIXED])
@pytest.mark.parametrize("nch,nr,P,nx,ny,n_slices,feed", [(96, 8, 96, 32, 32, 4, 9.6), (90, 5, 100, 33, 17, 3, 9.6),
                                                          (97, 18, 64, 70, 61, 6, 9.6), (128, 67, 48, 24, 40, 5, 9.6),
                                                          (96, 8, 96, 32, 32, 4, 4.0), (96, 6, 40, 200, 190, 9, 6.0)])
def test_refq_equals_k_bp(nch, nr, P, nx, ny, n_slices, feed, precision):
    spec = scans.tiny(nch=nch, nr=nr, P=P, rotations=3.3, nx=nx, n_slices=n_slices)
    spec.ny, spec.feed = ny, feed
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    ctx = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(precision=precision), device=0)
    ctx.set_views(tube, table)
    d = ctx.dims
    gen = torch.Generator(device=DEV).manual_seed(nch + nr)
    rows = torch.randn((d.n_views, d.n_rows, d.n_channels), device=DEV, generator=gen)
    scales, top = None, rows.abs().max().item()
    if precision == T.PRECISION_MIXED:
        rows = rows.half()
        e = torch.randint(-2, 3, (d.n_views, d.n_rows), device=DEV, generator=gen)
        scales = torch.exp2(e.float()).reshape(-1)
        top *= 4.0
    vols, counts = [], []
    for captured in (False, True):
        v = torch.full((d.n_slices_native, d.ny, d.nx), float("nan"), device=DEV)
        n = torch.zeros(1, dtype=torch.int64, device=DEV)
        if captured:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                ctx.backproject(rows, v, row_scales=scales, update_count=n)
            n.zero_()
            g.replay()
        else:
            ctx.backproject(rows, v, row_scales=scales, update_count=n)
        torch.cuda.synchronize()
        ctx.check_device_status()
        vols.append(v.double().cpu().numpy())
        counts.append(int(n.item()))
    a, b = vols
    assert counts[0] == counts[1] > 0
    assert np.array_equal(np.isnan(a), np.isnan(b)) and np.isfinite(b).mean() > 0.5
    assert np.nanmax(np.abs(a - b)) <= 2 * (P // 2) * 2.0 ** -24 * math.pi * top
