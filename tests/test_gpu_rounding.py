"""A result's bits depend on the length of a transform alone, not on the engine
or plan that runs it.

Every plan of the compile-time engine (fft_ct.cuh) does the arithmetic of the
runtime-plan engine's first radix order, whatever passes and threads it spreads
it over, and the TMA-fed last-axis operator of the lengths below 64, above 256
or with a factor 7 evaluates its operators in the operations of the plain
kernel.  So the plan variants of large grids (0) and of small ones (1) must both
agree bit for bit with the runtime-plan engine, at every compile-time length.
KWAVE_B200_TEST_FFT_PLAN makes a session or transform plan run that variant,
or the runtime-plan engine (-1), on every axis.

(Outputs that barely rise above FP32 rounding, such as the velocity component
that a plane wave does not excite in the first ten steps, change by far more
than any tolerance when a transform rounds in another order.)
"""
import os
import sys

import numpy as np
import pytest

from helpers import case_2d_p0, case_3d_het

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "k-wave_b200"))

import build  # noqa: E402  (k-wave_b200/build.py)

pytestmark = pytest.mark.gpu

LENGTHS = sorted(build.ct_sizes() + build._lengths("ct_more_sizes.h"))
BY_EIGHT = [LENGTHS[i:i + 8] for i in range(0, len(LENGTHS), 8)]
OTHER = [n for n in LENGTHS if n < 64 or n > 256 or n % 7 == 0]  # operators from |k|, as the plain kernel's
FROM_K2 = [n for n in LENGTHS if n not in OTHER]
RECORD = ("p", "p_max", "p_rms", "u", "p_final", "u_final")


def _ids(v):
    return f"{v[0]}-{v[-1]}" if isinstance(v, list) else None


HOOK = "KWAVE_B200_TEST_FFT_PLAN"


def _same_in_every_plan(run, what, monkeypatch):
    monkeypatch.setenv(HOOK, "-1")
    want = run()
    for v in ("0", "1"):
        monkeypatch.setenv(HOOK, v)
        got = run()
        for k in want:
            np.testing.assert_array_equal(got[k], want[k], err_msg=f"{k} {what} variant {v}")
    monkeypatch.delenv(HOOK)


def _transform(nx, ny, nz, passes):
    import torch
    from kwave import _lib

    plan = _lib.Fft3d(nx, ny, nz)
    g = torch.Generator(device="cuda").manual_seed(nx + ny + nz)
    real = torch.randn((nz, ny, nx), generator=g, device="cuda")
    spec = torch.randn((nz, ny, plan.nxp, 2), generator=g, device="cuda")
    if passes & 1:
        spec.zero_()
    back = torch.zeros_like(real)
    st = torch.cuda.current_stream().cuda_stream
    plan.exec(real.data_ptr(), spec.data_ptr(), inverse=False, passes=passes, stream=st)
    torch.cuda.synchronize()
    out = {"forward": spec[:, :, : nx // 2 + 1].cpu().numpy()}
    plan.exec(back.data_ptr(), spec.data_ptr(), inverse=True, passes=passes, stream=st)
    torch.cuda.synchronize()
    out["inverse"] = (back if passes & 1 else spec[:, :, : nx // 2 + 1]).cpu().numpy()
    plan.check()
    plan.close()
    return out


# columns of every length, rows of every even one (bare rows always run variant 0)
@pytest.mark.parametrize("ns", BY_EIGHT, ids=_ids)
def test_bare_transforms(ns, monkeypatch):
    for n in ns:
        _same_in_every_plan(lambda: _transform(42, n, 3, 2), f"y {n}", monkeypatch)
        if n % 2 == 0:
            _same_in_every_plan(lambda: _transform(n, 27, 1, 1), f"x {n}", monkeypatch)


def _solve(c):
    from kwave import _lib

    inp, record, start, _ = c
    return _lib.solve(inp, record, start_index=start)


# rows of every length: power-law absorbing (k_x_eos, k_x_rho with and without
# the EOS), corrected additive source; then lossless with a Dirichlet one
@pytest.mark.parametrize("ns", BY_EIGHT, ids=_ids)
def test_rows(ns, monkeypatch):
    for n in ns:
        c = case_3d_het(n=(n, 42, 45), nt=2, record=RECORD)
        _same_in_every_plan(lambda: _solve(c), f"{n} absorbing", monkeypatch)
    for n in ns[::3]:
        c = case_3d_het(n=(n, 40, 42), nt=2, absorbing=False, p_mode="dirichlet", record=RECORD)
        _same_in_every_plan(lambda: _solve(c), f"{n} lossless", monkeypatch)


# the y pass of every length, with the derived y derivative
@pytest.mark.parametrize("ns", BY_EIGHT, ids=_ids)
def test_columns(ns, monkeypatch):
    for n in ns:
        c = case_3d_het(n=(40, n, 45), nt=2, record=RECORD)
        _same_in_every_plan(lambda: _solve(c), n, monkeypatch)


# the last-axis operator of the lengths that evaluate it from |k|: gradient,
# divergence, fractional Laplacian, source correction and shift, in 3D and 2D;
# lines of one to seven segments
@pytest.mark.parametrize("ns", [OTHER[i:i + 8] for i in range(0, len(OTHER), 8)], ids=_ids)
def test_last_axis_operator(ns, monkeypatch):
    for n in ns:
        c = case_3d_het(n=(40, 42, n), nt=3, record=RECORD)
        _same_in_every_plan(lambda: _solve(c), f"3D {n}", monkeypatch)
        c = case_2d_p0(n=(50, n), nt=4, record=("p", "u", "u_non_staggered", "u_final"))
        _same_in_every_plan(lambda: _solve(c), f"2D {n}", monkeypatch)


# the lengths that evaluate it from |k|^2: the same in both variants
@pytest.mark.parametrize("ns", [FROM_K2[i:i + 8] for i in range(0, len(FROM_K2), 8)], ids=_ids)
def test_last_axis_operator_from_k_squared(ns, monkeypatch):
    for n in ns:
        for c in (case_3d_het(n=(40, 42, n), nt=3, record=RECORD), case_2d_p0(n=(50, n), nt=4, record=("p", "u"))):
            monkeypatch.setenv(HOOK, "0")
            want = _solve(c)
            monkeypatch.setenv(HOOK, "1")
            got = _solve(c)
            for k in want:
                np.testing.assert_array_equal(got[k], want[k], err_msg=f"{k} {n}")


# grids whose passes take variant 0 by the session's own choice
@pytest.mark.parametrize("n", [(98, 84, 126), (112, 98, 63), (105, 98, 49), (98, 60, 360), (84, 63, 432), (60, 50, 1008)])
def test_large_grids(n, monkeypatch):
    c = case_3d_het(n=n, nt=2, record=RECORD)
    own = _solve(c)
    monkeypatch.setenv(HOOK, "-1")
    want = _solve(c)
    for k in want:
        np.testing.assert_array_equal(own[k], want[k], err_msg=k)
