"""Device memory of wfbp_backproject on reference-layout rows: what a call takes for
the transposed rows goes back to the device, up to the 256 MiB that the context's
pool may keep, and a context that refuses the memory (backproject_scratch = -1)
takes none and gives the gather kernel's volume, as a captured call does."""
import threading

import pytest

from freect_b200 import scans, wfbp

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

KEEP = 256 << 20


def make(scratch=0, nch=896, nr=64, P=600):
    spec = scans.tiny(nch=nch, nr=nr, P=P, rotations=3, nx=128, n_slices=2)
    spec.fov = 200.0
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    ctx = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(backproject_scratch=scratch), device=0)
    ctx.set_views(tube, table)
    rows = torch.randn((spec.V, nr, nch), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    return ctx, rows, ctx.alloc("native")


def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_memory_goes_back():
    small = make(nch=96, nr=8, P=96)  # loads the kernels
    small[0].backproject(small[1], small[2])
    ctx, rows, vol = make()
    assert 4 * rows.numel() > KEEP + (64 << 20)
    before = free()
    for _ in range(3):
        ctx.backproject(rows, vol)
    assert before - free() <= KEEP
    ctx.close()
    assert before - free() <= 0


def test_refused():
    ctx, rows, vol = make(-1)
    ref = torch.empty_like(vol)
    ctx.backproject(rows, vol)
    before = free()
    for _ in range(2):
        ctx.backproject(rows, vol)
        assert free() == before
    other, _, _ = make()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        other.backproject(rows, ref)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(vol.nan_to_num(7.0), ref.nan_to_num(7.0))


def test_first_calls_of_several_threads():
    ctx, rows, vol = make(nch=96, nr=8, P=96)
    ref = torch.empty_like(vol)
    make(nch=96, nr=8, P=96)[0].backproject(rows, ref)
    vols = [torch.empty_like(vol) for _ in range(8)]
    torch.cuda.synchronize()
    start = threading.Barrier(len(vols))

    def call(v):
        s = torch.cuda.Stream()
        start.wait()
        ctx.backproject(rows, v, stream=s)
        s.synchronize()

    threads = [threading.Thread(target=call, args=(v,)) for v in vols]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(torch.equal(v.nan_to_num(7.0), ref.nan_to_num(7.0)) for v in vols)
