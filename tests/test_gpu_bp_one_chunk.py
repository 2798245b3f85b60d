"""One chunk of half-turn angles in the launches that can also run as a cluster
(reference-layout rows, and any launch that counts updates): little shared
memory, down to one view of one slab, where a chunk's sums would not fit. The
volumes and counts are held against k_bp (a captured call) and against the same
launch without the count."""
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


def make(nr, nx, n_slices, layout, precision=T.PRECISION_FP32):
    spec = scans.tiny(nch=288, nr=nr, P=48, rotations=3.3, nx=nx, n_slices=n_slices)
    spec.fov = 200.0
    tube, table = spec.views()
    cg, _ = wfbp.configure_geometry(spec.meta(), table)
    ctx = wfbp.Context(cg, spec.recon_config(), wfbp.make_ext(precision=precision, filtered_layout=layout), device=0)
    ctx.set_views(tube, table)
    return ctx, table


def backproject(ctx, rows, captured=False, count=False):
    v = torch.full((ctx.dims.n_slices_native, ctx.dims.ny, ctx.dims.nx), float("nan"), device=DEV)
    n = torch.zeros(1, dtype=torch.int64, device=DEV) if count else None
    if captured:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            ctx.backproject(rows, v, update_count=n)
        g.replay()
    else:
        ctx.backproject(rows, v, update_count=n)
    torch.cuda.synchronize()
    ctx.check_device_status()
    return v, int(n.item()) if count else 0


@pytest.mark.parametrize("nr", [8, 16])
@pytest.mark.parametrize("where", ["whole", "end", "beyond"])
def test_reference_layout(nr, where):
    ctx, table = make(nr, 512, 40, T.LAYOUT_REFERENCE)
    if where != "whole":  # few or no views reach these slices
        z = float(table.min()) - (200.0 if where == "beyond" else -0.3)
        ctx.set_slices([z, z + 0.5], [z])
    d = ctx.dims
    gen = torch.Generator(device=DEV).manual_seed(nr)
    rows = torch.randn((d.n_views, d.n_rows, d.n_channels), device=DEV, generator=gen)
    a, na = backproject(ctx, rows, count=True)
    b, nb = backproject(ctx, rows, captured=True, count=True)
    c, _ = backproject(ctx, rows)
    assert na == nb and (na > 0) == (where != "beyond")
    assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(a.nan_to_num(7.0), c.nan_to_num(7.0))
    tol = 2 * 24 * 2.0 ** -24 * math.pi * rows.abs().max().item()
    assert (a - b).nan_to_num(0.0).abs().max().item() <= tol


@pytest.mark.parametrize("precision", [T.PRECISION_FP32, T.PRECISION_MIXED])
@pytest.mark.parametrize("nr,n_slices", [(8, 2), (16, 2), (16, 30)])
def test_counted_launches(nr, n_slices, precision):
    ctx, _ = make(nr, 512, n_slices, T.LAYOUT_BACKPROJECTION, precision)
    d = ctx.dims
    gen = torch.Generator(device=DEV).manual_seed(nr)
    raw = torch.randn((d.n_readings, d.raw_rows, d.raw_channels), device=DEV, generator=gen)
    reb, rows = ctx.alloc("rebinned"), ctx.alloc("filtered")
    sc = ctx.alloc("row_scales")
    ctx.rebin(raw, reb)
    ctx.filter(reb, rows, row_scales=sc)
    counts = set()
    for cfg in ctx.bp_configs():
        ctx.set_bp_config(cfg)
        vols = []
        for count in (False, True):
            v = ctx.alloc("native")
            n = torch.zeros(1, dtype=torch.int64, device=DEV) if count else None
            ctx.backproject(rows, v, row_scales=sc, update_count=n)
            torch.cuda.synchronize()
            ctx.check_device_status()
            vols.append(v.cpu().numpy())
        counts.add(int(n.item()))
        assert np.array_equal(vols[0], vols[1], equal_nan=True), cfg.key()
    assert len(counts) == 1 and counts.pop() > 0
