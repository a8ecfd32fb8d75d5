"""Rows of the range-Doppler block that go sample by sample: long wavelengths and steep Vr, where the walk
of every row moves across the tile, with adjacent columns that share the integer walk, that do not, and the
last column of an odd width alone; centroids of either sign and near half the PRF.

The comparison and its tolerance are those of the row decisions' test: the per-stage entry point
against the oracle, 2e-6 relative RMSE for two float32 transforms and the interpolation.
"""
from __future__ import annotations

import pytest

import test_rcmc_rows as rows
from test_rcmc_rows import be  # noqa: F401

CASES = {
    "l_band": dict(wavelength=0.24),
    "l_band_negative": dict(wavelength=0.24, dc=(0.0, 0.0, -700.0)),
    "l_band_half_prf": dict(wavelength=0.24, dc=(0.0, 0.4, 790.0)),
    "l_band_full": dict(wavelength=0.24, az_bw_frac=1.0, dc=(0.0, 0.0, 839.0)),
    # the walk gains or loses a sample every few columns
    "steep_vr": dict(wavelength=0.12, vr=(0.0, -6.0, 7600.0), prf=3200.0),
    "rising_vr": dict(wavelength=0.12, vr=(0.0, 6.0, 6400.0), prf=3200.0, dc=(0.0, 0.0, -900.0)),
    "high_centroid": dict(prf=2080.0, dc=(0.0, 0.0, 1039.0)),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("shape", [(233, 240, 500, 504), (131, 132, 250, 250), (64, 64, 180, 180)])
def test_slow_rows_match_oracle(be, name, shape, monkeypatch):  # noqa: F811
    monkeypatch.setitem(rows.CASES, name, rows._case(**CASES[name]))
    rows.test_range_doppler_matches_oracle(be, name, shape)
