"""Every adjoint candidate of the shape-specialised space kernels
(agdeblend_b200/csrc/fast.cuh), float and double, through the ISTA update:
the first threshold of a solve is the largest |x| of the first update, so the
record is that of one model coefficient, placed in turn in every part of a
plane (columns of the last space axis, both parities of the row before it),
and a part that the maximum leaves out changes the whole schedule.  Single
solves and all coefficients together as a batch (one maximum per problem),
against the float64 oracle.

Surveys of one window whose shots do not overlap.  Three iterations of a
forward and an adjoint at the operators' gates (1e-5 and 1e-11 relative L2;
the threshold is a contraction), outputs of 0.8 to 1 of the input's norm:
1e-4 and 1e-10.  A maximum without the coefficient's own four columns is
3e-3 or more off."""
import functools
import os

import numpy as np
import pytest

import agd_oracle as O
import agdeblend_b200 as A
from agdeblend_b200 import synthetic as S
from conftest import rel_l2

pytestmark = pytest.mark.gpu

N_ITS = 4
SHAPES = {"P40": (32,), "P20": (16,), "P20x40": (16, 32), "P20x20": (16, 16),
          "P40x40": (32, 32), "P20x20x20": (16, 16, 16)}


def _survey(space, data=None, nt=128):
    n = int(np.prod(space))
    shape = [*space, nt]
    st = (2 * nt * np.arange(n)).astype(np.int64)
    zero = np.zeros(n, np.int32)
    d = np.zeros(shape) if data is None else data
    return S.Survey("one window", [0], [len(shape)], [shape], [[0] * len(space)], [shape], [st],
                    [zero], [zero], [d], [d], N_ITS)


def _plan(sv):
    return O.make_plan(sv.volumes, sv.n_dims, sv.window_shapes, sv.coords, sv.shapes,
                       sv.shottimes, sv.channels, sv.trace_types, sv.wavelet_lengths,
                       sv.wavelet_idxs, sv.wavelets)


@functools.lru_cache(maxsize=None)
def _cases(name):
    """(survey, oracle solve by the float and by the double schedule) of every
    coefficient."""
    space = SHAPES[name]
    plan = _plan(_survey(space))
    shape = plan.windows[0].model_shape  # time windows, space axes, frequencies
    step = 5 if len(space) < 3 else 9
    out = []
    for c in range(0, shape[-2], step):
        for r in (0, 1) if len(space) > 1 else (0,):
            x = plan.zero_model()
            at = [0, *([7 + r] * (len(space) - 1)), c, 17 + c % 2]
            x[0][tuple(at)] = 1.0
            data = O.set_output(plan, x)[0]
            out.append((_survey(space, data), O.deblend(plan, [data], 1.0, N_ITS)[0],
                        O.deblend(plan, [data], 1.0, N_ITS, double_schedule=True)[0]))
    return out


@pytest.fixture
def variant():
    old = os.environ.get("AGD_GPU_SPACE_VARIANT")

    def force(v):
        os.environ["AGD_GPU_SPACE_VARIANT"] = v

    yield force
    if old is None:
        os.environ.pop("AGD_GPU_SPACE_VARIANT", None)
    else:
        os.environ["AGD_GPU_SPACE_VARIANT"] = old


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_every_candidate_solves_as_the_oracle(name, dtype, variant):
    double = dtype == np.float64
    tol = 1e-10 if double else 1e-4
    cases = _cases(name)
    refs = [d if double else f for _, f, d in cases]
    data = [sv.data[0].astype(dtype) for sv, _, _ in cases]
    variant("0,0")
    probe = A.Problem.from_survey(cases[0][0], dtype)
    n_f, n_a = int(probe.info[12]), int(probe.info[13])
    probe.close()
    assert n_f >= 1 and n_a >= 1
    for v in range(max(n_f, n_a)):
        pick = (min(v, n_f - 1), min(v, n_a - 1))
        variant(f"{pick[0]},{pick[1]}")
        one = A.Problem.from_survey(cases[0][0], dtype)
        assert (one.info[10], one.info[11]) == pick
        for i, (d, ref) in enumerate(zip(data, refs)):
            out = one.solve([d], 1.0, N_ITS)[0]
            assert rel_l2(out, ref) <= tol, (pick, i)
        one.close()
        batch = A.Problem.from_batch([sv for sv, _, _ in cases], dtype)
        for i, (out, ref) in enumerate(zip(batch.solve(data, 1.0, N_ITS), refs)):
            assert rel_l2(out, ref) <= tol, (pick, i, "batch")
        batch.close()
