"""The split-precision form's overall gain: its forward block transform holds the DFT matrix in bf16 hi + lo
parts, whose rounding over the few entries of a short matrix is a gain of up to some 1e-6 that the inverse
scale takes back, as it does for the plain form's transforms.

The gain is the projection of the detected image on the plain form's of the same split, whose own gain is
compensated; an amplitude gain counts twice.  What may stay is the scatter of the tensor cores'
accumulation about the value taken back, at most 0.4e-7 of amplitude for each of the four 16-wide steps of
K, and as much again from the operands' rounding: 4e-7 of intensity.
"""
from __future__ import annotations

import numpy as np
import pytest

import asarf
from asarf import scene as S
from conftest import scene_and_raw


@pytest.mark.gpu
@pytest.mark.parametrize("lines,n2", [(4090, 0), (2010, 0), (2010, 63), (2870, 0), (2870, 60), (1990, 0), (3980, 0),
                                      (3980, 100), (3980, 125)])
def test_gain_against_plain_form(gpu_lib, lines, n2):
    sc, raw, _ = scene_and_raw(gpu_lib, S.tiny, range_size=1500, azimuth_size=lines, seed=31)
    plan = asarf.FocusPlan(sc, lib=gpu_lib, precision=1, az_n2=n2)
    assert plan.dims["precision"] == 1
    got = plan.focus_host(raw).astype(np.float64)
    n2 = plan.dims["n2"]
    plan.close()
    plan = asarf.FocusPlan(sc, lib=gpu_lib, az_n2=n2)
    want = plan.focus_host(raw).astype(np.float64)
    plan.close()
    gain = float((got * want).sum() / (want * want).sum()) - 1.0
    assert abs(gain) < 4e-7, (n2, gain)
