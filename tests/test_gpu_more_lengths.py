"""Compile-time and TMA-fed kernels of the lengths with a factor 7, from 40 to
63, and above 256 (whose line one tensor copy covers as several segments).

Against the FP64 oracle (runs this short meet it at 1e-6; the bar is 1e-5), and the TMA-fed y pass bit for
bit against the plain column kernel (both run the same radix plan)."""
import os

import numpy as np
import pytest

from helpers import case_3d_het, compare, oracle_outputs

pytestmark = pytest.mark.gpu

RECORD = ("p", "p_max", "p_rms", "u", "p_final")

GRIDS = [
    (40, 42, 45), (48, 49, 50), (54, 56, 60), (63, 70, 84), (98, 49, 42), (105, 45, 49), (112, 42, 63),
    (126, 40, 56), (42, 40, 147), (40, 42, 168), (48, 45, 189), (40, 49, 196), (56, 40, 252),
    # last axis in 2, 2, 5, 3 and 7 segments; y axis in 2 and 4
    (40, 42, 288), (42, 40, 540), (40, 40, 625), (40, 40, 729), (40, 40, 343), (40, 432, 45), (40, 1008, 40),
    # enough lines for the large-grid plan variant on every axis
    (112, 98, 126), (84, 105, 140),
]


@pytest.mark.parametrize("n", GRIDS)
def test_against_the_oracle(n):
    from kwave import _lib

    inp, record, start, _ = case_3d_het(n=n, nt=8, record=RECORD)
    gpu = _lib.solve(inp, record=record, start_index=start)
    errs = compare(gpu, oracle_outputs(inp, record, start, dtype=np.float64))
    bad = {k: v for k, v in errs.items() if not v <= 1e-5}
    assert errs and not bad, errs


@pytest.mark.parametrize("ny", [42, 49, 98, 126, 245, 270, 375, 384, 625, 768, 1008, 1024])
def test_tma_y_pass_matches_plain_y_pass(ny, monkeypatch):
    from kwave import _lib

    inp, record, start, _ = case_3d_het(n=(40, ny, 32), nt=4, record=RECORD)
    tma = _lib.solve(inp, record, start_index=start)
    monkeypatch.setenv("KWAVE_B200_NO_TMA", "1")
    plain = _lib.solve(inp, record, start_index=start)
    assert os.environ["KWAVE_B200_NO_TMA"] == "1"
    for k in plain:
        np.testing.assert_array_equal(tma[k], plain[k], err_msg=k)


@pytest.mark.parametrize("n", [(49, 63), (42, 40), (98, 105), (270, 540), (40, 1000), (343, 315)])
def test_2d_against_the_oracle(n):
    from helpers import case_2d_p0
    from kwave import _lib

    inp, record, start, _ = case_2d_p0(n=n, nt=30, record=("p", "p_max", "u", "p_final"))
    gpu = _lib.solve(inp, record=record, start_index=start)
    errs = compare(gpu, oracle_outputs(inp, record, start, dtype=np.float64))
    bad = {k: v for k, v in errs.items() if not v <= 1e-5}
    assert errs and not bad, errs
