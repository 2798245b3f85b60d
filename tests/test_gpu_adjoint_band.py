"""The table form of the backprojection adjoint (k_bp_adjoint_band and its weight
table) at the edges of its splits: row counts around the window sizes, voxels
wider and finer than a channel (lanes alone in a channel, or taking turns),
one native slice, slices finer than the detector rows, descending and unevenly
spaced slices, matrices that leave lanes idle, and a table computed in groups
of angles. Each result is held against the form without a table
(adjoint_scale_table = -1), which evaluates the same weights in the same
order: FP32 sums of the same terms in another order, so within n u of the
largest sum for the n ~ 1e3 terms of a sample (2^-24 x 1e3 = 6e-5), taken as
the tolerance of test_gpu_adjoint's table test, 1e-5 of the largest value.
"""
import numpy as np
import pytest

from freect_b200 import scans, wfbp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

DEV = torch.device("cuda", 0)


def both(spec, slices=None):
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    out = []
    for mode in (0, -1):
        ctx = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(adjoint_scale_table=mode), device=0)
        ctx.set_views(tube, table)
        if slices is not None:
            ctx.set_slices(slices, slices)
        d = ctx.dims
        gen = torch.Generator(device=DEV).manual_seed(7)
        g = torch.randn((d.n_slices_native, d.ny, d.nx), device=DEV, generator=gen)
        o = torch.full((d.n_views, d.n_rows, d.n_channels), float("nan"), device=DEV)
        for _ in range(2):
            ctx.backproject_adjoint(g, o)
        torch.cuda.synchronize()
        out.append(o)
        ctx.close()
    a, b = out
    assert torch.isfinite(a).all() and (spec.nr == 2 or b.abs().max() > 0)  # two rows: no row coordinate in [0, 0]
    assert (a - b).abs().max().item() <= 1e-5 * b.abs().max().item()


@pytest.mark.parametrize("nr", [2, 5, 16, 17, 33, 64, 100])
@pytest.mark.parametrize("fov,nx,ny", [(250.0, 32, 32), (60.0, 40, 25), (30.0, 33, 64)])
def test_rows_and_voxel_sizes(nr, fov, nx, ny):
    spec = scans.tiny(nch=100, nr=nr, P=48, rotations=3, nx=nx, n_slices=4)
    spec.ny, spec.fov = ny, fov
    both(spec)


@pytest.mark.parametrize("slices", [[0.3], np.linspace(-3, 3, 90), np.linspace(2.5, -2.5, 11),
                                    [-2.0, -1.9, -0.5, 0.1, 0.2, 1.7]])
def test_slices(slices):
    spec = scans.tiny(nch=96, nr=12, P=64, rotations=3, nx=24, n_slices=4)
    both(spec, np.asarray(slices, np.float32))


def test_table_in_groups_of_angles():
    # 1024 half-turn angles x 512 x 512 x 7 slices: a 7.5 GB table
    spec = scans.tiny(nch=64, nr=4, P=2048, rotations=1.5, nx=512, n_slices=1)
    both(spec, np.linspace(-1.5, 1.5, 7).astype(np.float32))
