"""The statistics accumulators belong to the plan and each run's finalisation leaves them zero for the next.
A run that ends between its statistics and its finalisation must leave no sums behind: not for the next
direct run, not where a capture that never runs comes between them, and not for a graph that was
captured before it.

Failure and capture are made on the host, in the emulation; a second run of the same bytes is the same
arithmetic, so images and statistics are compared bit for bit.  On the GPU: direct runs around a captured
graph and its replays.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import asarf
from asarf import _lib
from asarf import scene as S
from conftest import scene_and_raw


def _focus(plan, raw):
    out = np.zeros(plan.out_shape, dtype=np.float32)
    plan.focus(raw, out)
    return out, plan.results()


@pytest.mark.parametrize("captured", [0, 1, 2])
def test_sums_of_an_interrupted_run_are_gone(emu_lib, captured):
    sc, raw, _ = scene_and_raw(emu_lib, S.tiny)
    clear = emu_lib.asarf_emu_accumulators_clear
    clear.argtypes = [C.c_void_p]
    plan = asarf.FocusPlan(sc, lib=emu_lib)
    want, stats = _focus(plan, raw)
    assert clear(plan._h) == 1
    emu_lib.asarf_emu_fail_finalize()
    with pytest.raises(_lib.AsarfError, match="made to fail"):
        _focus(plan, raw)
    assert clear(plan._h) == 1  # what a replayed graph would add to
    for _ in range(captured):
        emu_lib.asarf_emu_capture(1)
        try:
            _focus(plan, raw)
        finally:
            emu_lib.asarf_emu_capture(0)
    got, again = _focus(plan, raw)
    assert np.array_equal(got, want) and again == stats
    plan.close()


def test_interrupted_while_captured(emu_lib):
    """The interruption itself under capture: nothing ran, and the next direct run is whole."""
    sc, raw, _ = scene_and_raw(emu_lib, S.tiny)
    plan = asarf.FocusPlan(sc, lib=emu_lib)
    want, stats = _focus(plan, raw)
    emu_lib.asarf_emu_capture(1)
    emu_lib.asarf_emu_fail_finalize()
    try:
        with pytest.raises(_lib.AsarfError):
            _focus(plan, raw)
    finally:
        emu_lib.asarf_emu_capture(0)
    got, again = _focus(plan, raw)
    assert np.array_equal(got, want) and again == stats
    plan.close()


@pytest.mark.gpu
def test_direct_runs_around_a_captured_graph(gpu_lib):
    import torch

    sc, raw, _ = scene_and_raw(gpu_lib, S.tiny)
    plan = asarf.FocusPlan(sc, lib=gpu_lib)
    d = torch.from_numpy(raw).cuda()
    outs = [torch.zeros(plan.out_shape, dtype=torch.float32, device="cuda") for _ in range(4)]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        plan.focus(d, outs[0], stream=side.cuda_stream)
        graph = torch.cuda.CUDAGraph()
        side.synchronize()
        with torch.cuda.graph(graph, stream=side):
            plan.focus(d, outs[1], stream=side.cuda_stream)
        plan.focus(d, outs[2], stream=side.cuda_stream)
        graph.replay()
        graph.replay()
        plan.focus(d, outs[3], stream=side.cuda_stream)
    torch.cuda.synchronize()
    assert plan.results()["errors"] == 0
    for o in outs[1:]:
        assert torch.equal(o, outs[0])
    del graph
    plan.close()
