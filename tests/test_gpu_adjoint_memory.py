"""The backprojection adjoint's weight table where memory is short, with the
shortage made on the host (wfbp_selftest_adjoint_table): the table shrinks to as
many half-turn angles as fit and is refilled group by group, a call that may not
allocate (captured) uses the table that is there or none. With a table the gradient
is the same bit for bit however its angles are grouped; without one it is the
gradient of a context that never has one (adjoint_scale_table = -1), and the two
agree to 1e-5 of the largest value, the tolerance of the table tests."""
import pytest

from freect_b200 import scans, wfbp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

DEV = torch.device("cuda", 0)


def make(table=0):
    spec = scans.tiny(nch=96, nr=12, P=64, rotations=3, nx=40, n_slices=6)
    tube, views = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), views)
    ctx = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(adjoint_scale_table=table), device=0)
    ctx.set_views(tube, views)
    d = ctx.dims
    g = torch.randn((d.n_slices_native, d.ny, d.nx), device=DEV, generator=torch.Generator(device=DEV).manual_seed(3))
    return ctx, g, 4 * g.numel()


def gradient(ctx, g, captured=False):
    d = ctx.dims
    out = torch.full((d.n_views, d.n_rows, d.n_channels), float("nan"), device=DEV)
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            ctx.backproject_adjoint(g, out)
        graph.replay()
    else:
        ctx.backproject_adjoint(g, out)
    torch.cuda.synchronize()
    return out


def test_table_shrinks_to_the_memory():
    ctx, g, per_angle = make()
    whole = gradient(ctx, g)
    assert ctx.selftest_adjoint_angles() == 32
    none = gradient(make(-1)[0], g)
    assert (whole - none).abs().max().item() <= 1e-5 * none.abs().max().item()
    for limit, free, angles in ((0, 20 * per_angle, 16), (0, 5 * per_angle, 4), (0, per_angle, 1),
                                (7 * per_angle, 0, 7), (7 * per_angle, 3 * per_angle, 2)):
        ctx.selftest_adjoint_table(limit, free)
        for _ in range(2):
            assert torch.equal(gradient(ctx, g), whole), (limit, free)
            assert ctx.selftest_adjoint_angles() == angles
    ctx.selftest_adjoint_table(0, per_angle - 1)
    assert torch.equal(gradient(ctx, g), none) and ctx.selftest_adjoint_angles() == 0


def test_captured_calls_allocate_nothing():
    none = gradient(make(-1)[0], make()[1])
    ctx, g, per_angle = make()
    assert torch.equal(gradient(ctx, g, captured=True), none)  # the context's first call
    assert ctx.selftest_adjoint_angles() == 0
    whole = gradient(ctx, g)
    assert torch.equal(gradient(ctx, g, captured=True), whole)
    # a fill that is captured belongs to its graph: a call before the replay fills for itself
    z, _ = ctx.slices()
    ctx.set_slices(z + 0.25, z + 0.25)
    other = torch.empty((ctx.dims.n_views, ctx.dims.n_rows, ctx.dims.n_channels), device=DEV)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.backproject_adjoint(g, other)
    moved = gradient(ctx, g)
    assert not torch.equal(moved, whole)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(other, moved)
