"""The compile-time engine's radix plans (fft_ct.cuh) against FP64.

The bare transform (kw_fft3d) is compared with numpy's FP64 FFT at every
compile-time length: a transform of n points in FP32 has a relative L2 error of
about eps sqrt(log2 n) (eps = 6e-8, random roundings), 2e-6 allows ten times
that over three axes.  Runs of a few steps are compared with the FP64 oracle,
in the plan variant of large grids and in that of small ones (a session picks
one per axis from its lines; KWAVE_B200_TEST_FFT_PLAN sets it): FP32 runs this
short meet 1e-6 and are held to 1e-5.
"""
import os
import sys

import numpy as np
import pytest

from helpers import case_3d_het, oracle_outputs

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "k-wave_b200"))

import build  # noqa: E402  (k-wave_b200/build.py)

pytestmark = pytest.mark.gpu

LENGTHS = sorted(build.ct_sizes() + build._lengths("ct_more_sizes.h"))

RECORD = ("p", "p_max", "p_rms", "u", "p_final")

# every length as y or z, each long one beside a short one, and every even one
# as x in turn
EVEN = [n for n in LENGTHS if n % 2 == 0]
GRIDS = [(EVEN[i], LENGTHS[i], LENGTHS[-1 - i]) for i in range(len(LENGTHS) // 2)]
GRIDS += [(n, 49, 40) for n in EVEN[len(LENGTHS) // 2:]]


@pytest.mark.parametrize("n", GRIDS)
def test_bare_transform_matches_numpy(n):
    import torch

    from kwave._lib import Fft3d

    nx, ny, nz = n
    rng = np.random.default_rng(nx + ny + nz)
    f = rng.standard_normal((nz, ny, nx)).astype(np.float32)
    plan = Fft3d(nx, ny, nz)
    x = torch.from_numpy(f).cuda()
    spec = torch.zeros((nz, ny, plan.nxp), device="cuda", dtype=torch.complex64)
    back = torch.empty_like(x)
    st = torch.cuda.current_stream().cuda_stream
    plan.exec(x.data_ptr(), spec.data_ptr(), False, 7, st)
    got = spec.cpu().numpy()[:, :, : nx // 2 + 1]
    plan.exec(back.data_ptr(), spec.data_ptr(), True, 7, st)
    plan.check()
    plan.close()
    ref = np.fft.rfftn(f.astype(np.float64))
    assert np.linalg.norm(got - ref) <= 2e-6 * np.linalg.norm(ref)
    assert np.linalg.norm(back.cpu().numpy() / f.size - f) <= 2e-6 * np.linalg.norm(f)


# rows, columns and last axis in each variant; odd and even-but-not-4 rows
# among them, and long rows (bulk-loaded, several warps a line)
@pytest.mark.parametrize("variant", ["0", "1"])
@pytest.mark.parametrize("n", [(64, 72, 75), (80, 64, 90), (81, 64, 64), (90, 64, 72), (96, 100, 108), (64, 125, 64),
                               (135, 108, 100), (150, 128, 81), (162, 64, 64), (192, 64, 64), (225, 64, 64),
                               (144, 120, 90), (180, 100, 96), (105, 98, 49), (256, 64, 72), (432, 64, 64)])
def test_each_variant_against_the_oracle(n, variant, monkeypatch):
    monkeypatch.setenv("KWAVE_B200_TEST_FFT_PLAN", variant)
    inp, record, start, _ = case_3d_het(n=n, nt=6, record=RECORD)
    _check(inp, record, start)


# long rows on the variant that the session picks, with and without the
# absorbing equation of state
@pytest.mark.parametrize("absorbing", [True, False])
@pytest.mark.parametrize("n", [(256, 72, 80), (540, 64, 45), (1008, 48, 49), (1024, 40, 42)])
def test_long_rows_against_the_oracle(n, absorbing):
    inp, record, start, _ = case_3d_het(n=n, nt=4, absorbing=absorbing, record=RECORD)
    _check(inp, record, start)


def _check(inp, record, start):
    from kwave import _lib

    gpu = _lib.solve(inp, record=record, start_index=start)
    ora = oracle_outputs(inp, record, start, dtype=np.float64)
    # a velocity component against the norm of the whole velocity: its rounding
    # errors are those of the pressure it is a gradient of, and a plane source
    # barely excites uy and uz in these few steps
    errs = {}
    for k in ora:
        parts = [ora[c + k[2:]] for c in ("ux", "uy", "uz")] if k[:2] in ("ux", "uy", "uz") else [ora[k]]
        norm = np.sqrt(sum(np.linalg.norm(np.asarray(p, np.float64).ravel()) ** 2 for p in parts))
        errs[k] = np.linalg.norm((np.asarray(gpu[k], np.float64) - ora[k]).ravel()) / norm
    bad = {k: v for k, v in errs.items() if not v <= 1e-5}
    assert errs and not bad, errs
    print(max(errs.values()))
