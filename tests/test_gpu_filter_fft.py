"""FP32 filter by FFT (k_filter_fft.cu) against the linear convolution in FP64,
at the edges of its transform lengths (2 nch < 256, 512, ...),
with row pairs that straddle views (odd row counts), rows of very different
size next to each other, rows of zeros, and rows with samples that are not
finite or so large that only the direct sum stays in range.

Tolerance: a radix FFT's rounding error grows at most with log2 N factors of
the unit roundoff u = 2^-24 in the 2-norm (Higham, Accuracy and Stability of
Numerical Algorithms, 24.1); forward, spectrum and inverse together stay below
u (8 log2 N + 4) |A|max ||d|| for the transformed sequence d and kernel a (the
row's differences and the taps' running sums), and an element is at most the
norm.
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


def make_ctx(nch, nr, layout, P=8, rotations=2.5):
    spec = scans.tiny(nch=nch, nr=nr, P=P, rotations=rotations, nx=8, n_slices=1)
    spec.fov = 8.0  # a channel window that every shape holds
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    ctx = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(filtered_layout=layout), device=0)
    ctx.set_views(tube, table)
    return ctx


def run_filter(ctx, x, layout):
    d = ctx.dims
    out = ctx.alloc("filtered")
    ctx.filter(torch.from_numpy(x).to(DEV), out)
    torch.cuda.synchronize()
    y = out.cpu().numpy()
    if layout == T.LAYOUT_BACKPROJECTION:
        y = y.reshape(d.n_views, d.n_channels, -1)[:, :, :d.n_rows].transpose(0, 2, 1)
    return y.reshape(d.n_views, d.n_rows, d.n_channels)


def conv64(x, half):
    n = np.arange(half.size)
    return x.astype(np.float64) @ half[np.abs(n[:, None] - n[None, :])]


def bound(x, half):
    nch = half.size
    N = 256
    while N <= 2 * nch:
        N *= 2
    a = np.cumsum(half) - half[0] / 2
    full = np.zeros(N)
    full[:nch] = a
    full[N - nch:] = -a[::-1]
    amax = np.abs(np.fft.fft(full)).max()
    z = np.zeros(x.shape[:-1] + (1,))
    d = np.diff(x.astype(np.float64), axis=-1, prepend=z, append=z)
    return 2.0 ** -24 * (8 * np.log2(N) + 4) * amax * np.linalg.norm(d, axis=-1)


@pytest.mark.parametrize("layout", [T.LAYOUT_REFERENCE, T.LAYOUT_BACKPROJECTION])
@pytest.mark.parametrize("nch,nr", [(16, 2), (127, 5), (128, 4), (255, 3), (256, 8), (511, 5), (512, 2), (701, 7),
                                    (1023, 5), (1024, 3), (2047, 5), (2048, 3)])
def test_filter_fft_edges(nch, nr, layout):
    ctx = make_ctx(nch, nr, layout)
    d = ctx.dims
    if layout == T.LAYOUT_BACKPROJECTION:
        try:
            ctx.bp_config()
        except wfbp.WfbpError:
            pytest.skip("no backprojection-layout launch fits this geometry")
    rng = np.random.default_rng(nch + nr)
    x = rng.standard_normal((d.n_views, d.n_rows, nch)).astype(np.float32)
    x *= np.float32(10.0) ** rng.integers(-9, 10, (d.n_views, d.n_rows, 1)).astype(np.float32)
    x[1, 0] = 0.0
    x[2, -1] = 0.0
    x[3, 0] = 0.0
    x[3, 0, nch // 2] = 1e-40  # a subnormal sample
    half = wfbp.filter_taps(ctx.cg, n=nch).astype(np.float64)
    y = run_filter(ctx, x, layout)
    ref = conv64(x, half)
    err = np.abs(y - ref).max(axis=-1)
    tol = bound(x, half) + 1e-42
    if nch > 2047:  # the Toeplitz product: a chain of nch FMAs
        tol = 2.0 ** -24 * nch * np.abs(x.astype(np.float64)).max(axis=-1) * np.abs(half).sum() * 2
    assert (err <= tol).all(), (err / tol).max()
    assert not y[1, 0].any() and not y[2, -1].any()


@pytest.mark.parametrize("nch", [96, 300, 888, 1472])
def test_filter_fft_rows_out_of_range(nch):
    # a row that is not finite, or whose transform would overflow, leaves every
    # other row as it is, its pair's other row too, and gives the direct sum
    nr = 6
    ctx = make_ctx(nch, nr, T.LAYOUT_REFERENCE)
    d = ctx.dims
    rng = np.random.default_rng(nch)
    x = rng.standard_normal((d.n_views, nr, nch)).astype(np.float32)
    half = wfbp.filter_taps(ctx.cg, n=nch).astype(np.float64)
    clean = run_filter(ctx, x, T.LAYOUT_REFERENCE)
    z = x.copy()
    z[0, 1, 3] = np.nan
    z[1, 2, nch - 1] = np.inf
    z[2, 4] = x[2, 4] * np.float32(1e36)
    y = run_filter(ctx, z, T.LAYOUT_REFERENCE)
    touched = np.zeros((d.n_views, nr), bool)
    touched[0, :2] = touched[1, 2:4] = touched[2, 4:6] = True
    assert (y[~touched] == clean[~touched]).all()
    direct = 2.0 ** -24 * nch * np.abs(x).max(axis=-1) * np.abs(half).sum() * 2
    ref = conv64(x, half)
    for v, r in ((0, 0), (1, 3), (2, 5)):  # the other rows of those pairs
        assert np.abs(y[v, r] - ref[v, r]).max() <= direct[v, r]
    assert not np.isfinite(y[0, 1]).any() and not np.isfinite(y[1, 2]).any()
    big = conv64(z[2:3, 4], half)[0]
    assert np.abs(y[2, 4] - big).max() <= direct[2, 4] * 1.0001e36


def test_filter_follows_new_taps():
    # after wfbp_set_taps: the forward filter (Toeplitz product, a chain of nch
    # FMAs) and the adjoint (FFT) both use the taps that were set last
    nch, nr = 200, 4
    ctx = make_ctx(nch, nr, T.LAYOUT_REFERENCE)
    d = ctx.dims
    rng = np.random.default_rng(5)
    x = rng.standard_normal((d.n_views, nr, nch)).astype(np.float32)
    for k in range(2):
        half = rng.standard_normal(nch).astype(np.float32)
        ctx.set_taps(torch.from_numpy(half).to(DEV))
        h64 = half.astype(np.float64)
        chain = 2.0 ** -24 * nch * np.abs(x).max(axis=-1) * np.abs(h64).sum() * 2
        err = np.abs(run_filter(ctx, x, T.LAYOUT_REFERENCE) - conv64(x, h64)).max(axis=-1)
        assert (err <= chain).all()
        g = torch.empty(x.shape, dtype=torch.float32, device=DEV)
        ctx.filter_adjoint(torch.from_numpy(x).to(DEV), g)
        torch.cuda.synchronize()
        err = np.abs(g.cpu().numpy() - conv64(x, h64)).max(axis=-1)
        assert (err <= bound(x, h64)).all()
