"""A step is replayed as one CUDA graph; the steps that cannot be (the first with
an initial pressure, those with a corrected source of their own) are launched
kernel by kernel.  The same kernels run on the same data either way, and the
device clock is advanced by each step's first kernel, so every split of a run
gives the same outputs bit for bit, and the right ones: a clock that is off by
one would move sources and records by a step."""
import numpy as np
import pytest

from helpers import case_2d_p0, case_3d_het, compare, oracle_outputs

pytestmark = pytest.mark.gpu


def _run(inp, record, start, chunks):
    from kwave import _lib

    s = _lib.Session(inp, record, start)
    try:
        for n in chunks:
            s.advance(n)
        assert s.steps_done == sum(chunks)
        return s.read()
    finally:
        s.close()


def _cases():
    yield case_2d_p0(n=(64, 48), nt=150, record=("p", "p_max", "p_rms", "u", "u_final"))  # step 1 is not replayed
    yield case_3d_het(n=(40, 42, 45), nt=150, record=("p", "p_max", "p_rms", "u"))
    yield case_3d_het(n=(40, 42, 45), nt=150, many=True, record=("p", "p_rms"))  # per-step corrected source
    yield case_3d_het(n=(28, 36, 35), nt=150, record=("p", "p_rms"))  # runtime-plan engine


@pytest.mark.parametrize("which", range(4))
def test_every_split_of_a_run_gives_the_same_outputs(which):
    inp, record, start, _ = list(_cases())[which]
    whole = _run(inp, record, start, [150])
    errs = compare(whole, oracle_outputs(inp, record, start, dtype=np.float64))
    assert errs and not {k: v for k, v in errs.items() if not v <= 1e-4}, errs
    for chunks in ([1] * 150, [7, 64, 65, 1, 13], [149, 1], [63, 87]):
        part = _run(inp, record, start, chunks)
        for k in whole:
            np.testing.assert_array_equal(part[k], whole[k], err_msg=f"{k} {chunks[:3]}")


# The operators' series (spec_ops.cuh) run over u = (c_ref dt |k| / 2)^2, up to
# 0.7, 1.0, 1.1 and 2.7 at the highest wavenumbers of these time steps; FP32 runs
# of ten steps meet the FP64 oracle's sine at 1e-6 and are held to 1e-5.
@pytest.mark.parametrize("scale", [1.0, 1.2, 1.3, 2.0])
def test_sinc_series_over_its_range(scale):
    from kwave import _lib

    inp, record, start, _ = case_3d_het(n=(48, 54, 56), nt=10, record=("p", "p_max", "p_rms", "u", "p_final"))
    inp = dict(inp, dt=inp["dt"] * scale)
    gpu = _lib.solve(inp, record=record, start_index=start)
    errs = compare(gpu, oracle_outputs(inp, record, start, dtype=np.float64))
    bad = {k: v for k, v in errs.items() if not v <= 1e-5}
    assert errs and not bad, errs
