"""Shared memory of the staged backprojection (bp_smem_layout), evaluated on the
host over the launch shapes, detector rows, view slots, record forms and chunk
counts: the region of the chunk sums, which a cluster's CTAs exchange through,
lies inside the allocation whenever the exchange runs (bp_exchanges), apart from
every region that is still in use then, and its words are 16-byte aligned. The
sizes are those of a launch: one view slot is as many channels as a window has,
rounded up to 128 bytes."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "wfbp_internal.h"
#include <stdio.h>
int main() {
  const int shapes[][5] = {{8, 8, 4, 16, 32},  {8, 8, 4, 8, 32},   {8, 16, 8, 8, 16},   {8, 16, 8, 8, 32},
                           {16, 16, 8, 16, 32}, {16, 16, 4, 16, 32}, {16, 20, 8, 20, 16}, {16, 16, 8, 16, 16}};
  const int rows[] = {2, 5, 8, 16, 33, 64, 128};
  long n = 0, bad = 0;
  for (auto& c : shapes)
    for (int nr : rows)
      for (int nv = 1; nv <= 20; nv++)
        for (int W = 4; W <= 64; W *= 2)
          for (int zc = 0; zc < 2; zc++)
            for (int nc = 1; nc <= BP_MAX_CHUNKS; nc *= 2) {
              BPTile b = {};
              b.tx = c[0]; b.ty = c[1]; b.cu = c[2]; b.nw = c[3]; b.slab = c[4];
              b.W = W; b.nrp = (nr + 3) / 4 * 4; b.nv_max = nv; b.zc = zc; b.nc = nc;
              b.slot_bytes = (W * b.nrp * 4 + 127) / 128 * 128;
              const BpSmem L = bp_smem_layout(b, c[0] * c[1] / c[3]);
              const unsigned sums = (unsigned)(b.tx * b.ty * b.slab) * 4u;
              n++;
              if (!bp_exchanges(nc)) continue;
              const bool inside = L.part % 16 == 0 && L.part + sums <= L.total;
              const bool over_ring = L.part == L.slots && sums <= L.vinfo - L.slots;
              const bool behind = L.part >= L.geo + b.nw * (nv + 1) * bp_geo_view(c[0] * c[1] / c[3], b.slab,
                                                                    zc ? BP_GEO_BYTES_ZCULL : BP_GEO_BYTES);
              if (!inside || !(over_ring || behind)) bad++;
            }
  printf("%ld %ld\n", n, bad);
  return 0;
}
"""


def test_chunk_sums_inside_the_allocation(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SOURCE)
    from freect_b200 import build_lib
    cuda = os.path.join(os.path.dirname(os.path.dirname(build_lib.nvcc())), "include")
    if not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    subprocess.run(["g++", "-std=c++17", "-I" + cuda, "-I" + os.path.join(ROOT, "freect_b200", "csrc"),
                    "-I" + os.path.join(ROOT, "include"), str(src), "-o", str(exe)], check=True)
    n, bad = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert n > 10000 and bad == 0

