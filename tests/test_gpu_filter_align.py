"""wfbp_filter into the backprojection layout at every float of a buffer: the
transform's two-row stores must not need more than a float's alignment, and
write the same rows, and nothing else, wherever the output begins."""
import pytest

from freect_b200 import abi_types as T
from freect_b200 import scans, wfbp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)


@pytest.mark.parametrize("nch,nr", [(90, 5), (300, 8), (888, 6), (1472, 3)])
def test_output_at_any_float(nch, nr):
    spec = scans.tiny(nch=nch, nr=nr, P=16, rotations=2.5, nx=8, n_slices=1)
    spec.fov = 8.0
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    ctx = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(filtered_layout=T.LAYOUT_BACKPROJECTION), device=0)
    ctx.set_views(tube, table)
    x = torch.randn(spec.V * nr * nch, device="cuda", generator=torch.Generator(device="cuda").manual_seed(nch))
    n = ctx.alloc("filtered").numel()
    outs = []
    for shift in range(4):
        buf = torch.full((n + 8,), 7.0, device="cuda")
        ctx.filter(x, buf[shift:shift + n])
        torch.cuda.synchronize()
        assert (buf[:shift] == 7.0).all() and (buf[shift + n:] == 7.0).all()
        y = buf[shift:shift + n].view(spec.V, nch, -1)
        assert (y[:, :, nr:] == 7.0).all()  # the rows' padding is not written
        outs.append(y[:, :, :nr].clone())
    for y in outs[1:]:
        assert torch.equal(y, outs[0])
