"""FP32 filter of rows that are 0 but for a few samples (a lone reading, an impulse
response, the gradient of a small region): up to 64 samples such a row is the
Toeplitz product's sum, bit for bit, whatever row shares its transform; above, the
transform is at least as exact as the product against FP64 (2-norm over the rows of
one count of samples)."""
import numpy as np
import pytest

from freect_b200 import scans, wfbp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("nch", [40, 96, 127, 200, 500, 888, 1472, 2047])
def test_few_samples(nch, adjoint):
    counts = [c for c in (1, 2, 17, 63, 64, 65, 96, 200) if c <= nch]
    nr = 2 * len(counts) + 1
    spec = scans.tiny(nch=nch, nr=nr, P=24, rotations=2.5, nx=8, n_slices=1)
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    ctx = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(), device=0)
    ctx.set_views(tube, table)
    rng = np.random.default_rng(nch)
    x = rng.standard_normal((spec.V, nr, nch)).astype(np.float32)  # dense rows between the sparse ones
    x[::3, 1] = 0.0
    for v in range(spec.V):
        for i, c in enumerate(counts):
            keep = rng.permutation(nch)[:c] if v % 2 else rng.integers(0, nch - c + 1) + np.arange(c)
            row = np.zeros(nch, np.float32)
            row[keep] = x[v, 2 * i, keep]
            x[v, 2 * i] = row
    xd, fft, product = torch.from_numpy(x).cuda(), ctx.alloc("filtered"), ctx.alloc("filtered")
    if adjoint:
        ctx.filter_adjoint(xd, fft)
    else:
        ctx.filter(xd, fft)
    ctx.set_taps(ctx.get_taps())
    ctx.filter(xd, product)
    torch.cuda.synchronize()
    y, t = fft.cpu().numpy(), product.cpu().numpy()
    n = np.arange(nch)
    ref = x.astype(np.float64) @ wfbp.filter_taps(ctx.cg, n=nch).astype(np.float64)[np.abs(n[:, None] - n[None, :])]
    assert not y[::3, 1].any()
    for i, c in enumerate(counts):
        if c <= 64:
            assert np.array_equal(y[:, 2 * i], t[:, 2 * i]), c
        else:
            scale = np.linalg.norm(ref[:, 2 * i], axis=-1, keepdims=True)
            ey, et = (np.linalg.norm((a[:, 2 * i] - ref[:, 2 * i]) / scale) for a in (y, t))
            assert ey <= et, (c, ey, et)
