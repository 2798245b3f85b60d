"""Stage calls of one context may overlap on several streams: the FP32 filter must
write its output and nothing of the context. A captured filter call is one kernel
(the taps' spectrum is computed with the taps), and overlapping calls on two
streams, after new taps too, give what each gives alone."""
import pytest

from freect_b200 import scans, wfbp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)


def make(nch=300, nr=6):
    spec = scans.tiny(nch=nch, nr=nr, P=64, rotations=3, nx=8, n_slices=1)
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    ctx = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(), device=0)
    ctx.set_views(tube, table)
    gen = torch.Generator(device="cuda").manual_seed(1)
    xs = [torch.randn((spec.V, nr, nch), device="cuda", generator=gen) for _ in range(2)]
    return ctx, xs


@pytest.mark.parametrize("call", ["filter", "filter_adjoint"])
def test_captured_filter_is_one_kernel(call):
    rt = pytest.importorskip("cuda.bindings.runtime")
    ctx, xs = make()
    y = torch.empty_like(xs[0])
    try:
        g = torch.cuda.CUDAGraph(keep_graph=True)
    except TypeError:
        pytest.skip("this torch does not hand out its graphs")
    with torch.cuda.graph(g):
        getattr(ctx, call)(xs[0], y)
    graph = rt.cudaGraph_t(g.raw_cuda_graph())
    err, _, n = rt.cudaGraphGetNodes(graph, 0)
    assert int(err) == 0 and n == 1
    g.replay()
    ref = torch.empty_like(y)
    getattr(ctx, call)(xs[0], ref)
    torch.cuda.synchronize()
    assert torch.equal(y, ref)


def test_overlapping_calls():
    ctx, xs = make()
    streams = [torch.cuda.Stream() for _ in xs]
    for new_taps in (False, True):
        if new_taps:
            ctx.set_taps(torch.randn(40, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2)))
        alone = [torch.empty_like(x) for x in xs]
        for x, y in zip(xs, alone):
            ctx.filter_adjoint(x, y)
        torch.cuda.synchronize()
        ys = [[torch.empty_like(x) for _ in range(8)] for x in xs]
        for i in range(8):
            for s, x, y in zip(streams, xs, ys):
                ctx.filter_adjoint(x, y[i], stream=s)
        torch.cuda.synchronize()
        for a, y in zip(alone, ys):
            assert all(torch.equal(a, b) for b in y)
