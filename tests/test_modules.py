"""Each compiled schedule and range length is a translation unit, and so a module, of its own: a process loads
what its plans run and nothing else, and a plan loads it when it is made, so that its first run may be a
stream capture.
"""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

import build as B

ROOT = Path(__file__).resolve().parent.parent


def test_every_schedule_has_its_unit():
    units = B.units()
    names = [u[1] for u in units]
    assert len(set(names)) == len(names)
    blocks, strided = B._cases("params.h", "ASARF_BLOCK_SCHEDULES"), B._cases("params.h", "ASARF_STRIDED_SCHEDULES")
    lengths = B._cases("fft_ct.cuh", "ASARF_CT_LENGTHS")
    assert len(blocks) >= 16 and len(strided) >= 2 and len(lengths) == 8
    for v in ["0, 0, 0"] + blocks:
        assert f"az_rd.cu.{v.replace(', ', '_')}" in names
    for v in strided:
        assert f"az_strided.cu.{v.replace(', ', '_')}_32_1" in names
    for v in ["0"] + lengths:
        assert f"range_compress.cu.{v}" in names
    # the kernels every process uses hold no schedule
    common = (B.CSRC / "kernels.cu").read_text()
    for kernel in ("k_az_rd", "k_az_strided", "k_range_compress", "k_rc_rows"):
        assert f"__global__ void {kernel}" not in common and f"{kernel}<<<" not in common


SCRIPT = """
import sys
sys.path[:0] = [{root!r}, {root!r} + "/asar-focus_b200", {root!r} + "/tests"]
import torch
import asarf
from asarf import scene as S, sim
lib = asarf.load_library()
sc = S.{factory}(range_size={nr}, azimuth_size={na})
sc.prepare(lib)
raw, _ = sim.simulate(sc, device="cuda")
raw = raw if isinstance(raw, torch.Tensor) else torch.from_numpy(raw).cuda()
side = torch.cuda.Stream()
plan = asarf.FocusPlan(sc, lib=lib)
out = [torch.zeros(plan.out_shape, dtype=torch.float32, device="cuda") for _ in range(2)]
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph, stream=side):
    plan.focus(raw, out[0], stream=side.cuda_stream)
graph.replay()
torch.cuda.synchronize()
plan.focus(raw, out[1], stream=side.cuda_stream)
torch.cuda.synchronize()
assert plan.results()["errors"] == 0
assert float(out[1].abs().max()) > 0 and torch.equal(out[0], out[1])
del graph
print("captured first")
"""


@pytest.mark.gpu
@pytest.mark.parametrize("factory,nr,na", [("tiny", 768, 1024), ("tiny_fbaq", 1000, 2010)])
def test_first_run_of_a_process_is_a_capture(gpu_lib, factory, nr, na):
    code = SCRIPT.format(root=str(ROOT), factory=factory, nr=nr, na=na)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "captured first" in r.stdout, r.stdout + r.stderr
