"""The trace-pair time kernels (agdeblend_b200/csrc/time_pair.cuh), windows of
128 and 256 samples, against the float64 oracle through the operators (gates
of test_gpu_operators): trace counts around the 16 traces of a block (a lone
trace, odd counts, a block and one trace), odd window sizes, whose bins are
not 16-byte aligned, the fewest time windows, grids that are split over the
windows (small) and grids that are not (many traces), and traces after a
source wavelet, which are read from the window traces instead of the
record."""
import dataclasses

import numpy as np
import pytest

import agdeblend_b200 as A
from agdeblend_b200 import synthetic as S
from test_gpu_operators import _check_operators

pytestmark = pytest.mark.gpu

# shots, samples, space window, time window
CASES = {
    "one_pair": (2, 300, 2, 128),
    "odd_15": (15, 300, 15, 256),
    "odd_17": (17, 700, 17, 256),
    "block_16": (16, 1100, 16, 256),
    "block_and_one_33": (33, 300, 33, 128),
    "fewest_windows": (18, 128, 18, 128),
    "windows_35": (35, 513, 20, 128),
    "many_traces": (900, 300, 36, 128),
}


def _survey(name, seed=6200):
    shots, nt, ws, wt = CASES[name]
    sv = S.gather_2d(seed=seed, n_shots=shots, nt=nt, window=(ws, wt))
    rng = np.random.default_rng(seed)
    tt = rng.choice([S.LIVE] * 8 + [S.BAD, S.MISSING], shots).astype(np.int32)
    tt[0] = S.LIVE
    return dataclasses.replace(sv, trace_types=[tt])


def _uses_pair_kernels(sv, dtype):
    p = A.Problem.from_survey(sv, dtype)
    k = p.kernels()
    p.close()
    return (k["time_fwd"], k["time_adj"]) == ("time_fwd_pair", "time_adj_pair")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("name", sorted(CASES))
def test_time_pair_vs_oracle(name, dtype):
    sv = _survey(name)
    assert _uses_pair_kernels(sv, dtype)
    _check_operators(sv, dtype)


@pytest.mark.parametrize("name", ["odd_17", "windows_35"])
def test_time_pair_with_wavelet(name):
    sv = _survey(name, seed=6300)
    w = np.hanning(24).astype(np.float32)
    n = int(sv.trace_types[0].size)
    sv = dataclasses.replace(sv, trace_types=[np.zeros(n, np.int32)], wavelet_lengths=[24],
                             wavelet_idxs=[np.zeros(n, np.int32)], wavelets=[w])
    assert _uses_pair_kernels(sv, np.float32)
    _check_operators(sv, np.float32)
