"""The FFT filter transforms two detector rows at a time. Smooth rows beside rough
ones must not take on the rough rows' rounding: against FP64, every kind of row is
at least as exact (2-norm over the rows of that kind) as the Toeplitz product on
the same rows, which a context with wfbp_set_taps runs."""
import numpy as np
import pytest

from freect_b200 import scans, wfbp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)


def both_forms(nch, nr, rows):
    """FFT filter and Toeplitz product of rows [V][nr][nch], and the FP64 convolution."""
    spec = scans.tiny(nch=nch, nr=nr, P=24, rotations=2.5, nx=8, n_slices=1)
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    ctx = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(), device=0)
    ctx.set_views(tube, table)
    x = np.ascontiguousarray(rows(spec.V), np.float32)
    out = []
    for product in (False, True):
        if product:
            ctx.set_taps(ctx.get_taps())
        y = ctx.alloc("filtered")
        ctx.filter(torch.from_numpy(x).cuda(), y)
        torch.cuda.synchronize()
        out.append(y.cpu().numpy())
    n = np.arange(nch)
    half = wfbp.filter_taps(ctx.cg, n=nch).astype(np.float64)
    return out[0], out[1], x.astype(np.float64) @ half[np.abs(n[:, None] - n[None, :])]


@pytest.mark.parametrize("nch", [96, 120, 300, 700, 888, 1472, 2047])
def test_smooth_rows_beside_rough_ones(nch):
    n, rng = np.arange(nch), np.random.default_rng(nch)
    smooth = [np.ones(nch), np.sqrt(np.maximum(0, 1 - ((n - nch / 2) / (0.35 * nch)) ** 2)), n / nch,
              np.exp(-((n - nch / 2) / (0.1 * nch)) ** 2)]
    rough = [1.99 * (-1.0) ** n, 0.6 * rng.standard_normal(nch)]
    kinds = [(a, b) for a in range(len(smooth)) for b in range(len(rough))]

    def rows(V):  # pair i of every view: smooth row beside rough row, either first
        x = np.empty((V, 2 * len(kinds), nch))
        for v in range(V):
            for i, (a, b) in enumerate(kinds):
                s = smooth[a] * rng.uniform(0.5, 2.0) * 10.0 ** rng.integers(-3, 4)
                r = rough[b] * rng.uniform(0.5, 2.0) * 10.0 ** rng.integers(-3, 4)
                x[v, 2 * i + v % 2], x[v, 2 * i + 1 - v % 2] = s, r
        return x

    y, t, ref = both_forms(nch, 2 * len(kinds), rows)
    scale = np.linalg.norm(ref, axis=-1)
    ey, et = (np.linalg.norm(a - ref, axis=-1) / scale for a in (y, t))
    for i in range(2 * len(kinds)):
        for first in (0, 1):  # the smooth row first, or second
            assert np.linalg.norm(ey[first::2, i]) <= np.linalg.norm(et[first::2, i]), (i, first)
