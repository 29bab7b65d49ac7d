"""The table-DFT space kernels (agdeblend_b200/csrc/plane_dft.cuh) of windows
with two to four space axes: uneven windows (18 x 35 for a nominal 16 x 32),
prime and even padded lengths, the shortest axes, the longest (128) and
planes that fill the shared memory, three and four space axes (one or two
single-axis passes beside the planes), windows on the shape-specialised
kernels beside them.  Against the float64 oracle (operators: the gates of
test_gpu_operators, 1e-5 relative L2 and the dot test in float, 1e-11 in
double) and, for the update and its thresholds, the generic passes
(AGD_GPU_GENERIC=1) over a solve."""
import os

import numpy as np
import pytest

import agd_oracle as O
import agdeblend_b200 as A
from agdeblend_b200 import synthetic as S
from conftest import rel_l2
from test_gpu_operators import _check_operators

pytestmark = pytest.mark.gpu


def _survey(space, windows, nt=70, wt=32, seed=5):
    """One patch with the given space shape and windows, one channel."""
    rng = np.random.default_rng(seed)
    n = int(np.prod(space))
    st = np.cumsum(rng.integers(nt // 3, nt, n)).astype(np.int64)
    tt = rng.choice([S.LIVE] * 8 + [S.BAD, S.MISSING], n).astype(np.int32)
    tt[0] = S.LIVE
    shape = [*space, nt]
    data = rng.standard_normal(shape).astype(np.float32)
    return S.Survey("plane", [0], [len(shape)], [[*windows, wt]], [[0] * len(space)], [shape],
                    [st], [np.zeros(n, np.int32)], [tt], [data], [data.copy()], 12)


# space shape, windows -> window lengths L (padded P) of the axes
CASES = {
    "uneven_18x35": ((37, 101), (16, 32)),      # L 18, 17 x 35, 34; P 23, 22 x 44, 43
    "prime_P43x23": ((88, 28), (32, 16)),       # both windows uneven
    "shortest": ((2, 3), (2, 3)),               # P 3 x 4
    "short_and_long": ((3, 102), (3, 100)),     # P 4 x 128
    "long_and_short": ((101, 5), (101, 5)),     # P 127 x 7
    "largest_plane": ((90, 92), (90, 92)),      # P 113 x 115: one block per SM
    "beside_fast_windows": ((16, 33), (16, 16)),  # 20 x 20 windows and uneven ones
    "three_axes": ((9, 7, 11), (4, 7, 6)),
    "three_axes_uneven_16": ((18, 17, 21), (16, 16, 16)),
    "four_axes": ((5, 4, 6, 5), (4, 4, 6, 5)),
}


def _case(name):
    space, windows = CASES[name]
    return _survey(space, windows)


@pytest.mark.parametrize("name", sorted(CASES))
def test_plane_operators_vs_oracle(name):
    sv = _case(name)
    prob = A.Problem.from_survey(sv)
    assert prob.info[8] in (0, 2)
    if prob.info[8] == 0:
        k = prob.kernels()
        assert k["space_fwd"] == k["space_adj"] and k["space_fwd"] in ("plane_dft", "line_dft")
    prob.close()
    _check_operators(sv, np.float32)


@pytest.mark.parametrize("name", ["uneven_18x35", "shortest", "short_and_long",
                                  "three_axes_uneven_16"])
def test_plane_operators_double(name):
    _check_operators(_case(name), np.float64, 1)


def _solve(sv, generic):
    old = os.environ.get("AGD_GPU_GENERIC")
    os.environ["AGD_GPU_GENERIC"] = "1" if generic else "0"
    try:
        return A.deblend(sv.volumes, sv.window_shapes, sv.coords, sv.shottimes, sv.channels,
                         sv.trace_types, 1.0, sv.n_its, 0, sv.data)
    finally:
        if old is None:
            os.environ.pop("AGD_GPU_GENERIC", None)
        else:
            os.environ["AGD_GPU_GENERIC"] = old


@pytest.mark.parametrize("name", ["uneven_18x35", "beside_fast_windows", "three_axes"])
def test_plane_solve_matches_generic_passes(name):
    sv = _case(name)
    for o, r in zip(_solve(sv, False), _solve(sv, True)):
        assert rel_l2(o, r) <= 1e-4


def test_plane_batch_matches_separate_solves():
    """Per-problem step, threshold and maximum in one launch."""
    svs = [_survey((18, 35), (16, 32), seed=7), _survey((9, 11), (4, 6), seed=8),
           _survey((37,), (16,), seed=9)]
    kw = [dict(volumes=v.volumes, window_shapes=v.window_shapes, coords=v.coords,
               shottimes=v.shottimes, channels=v.channels, trace_types=v.trace_types,
               data=v.data) for v in svs]
    for sv, out in zip(svs, A.deblend_batch(kw, 1.0, svs[0].n_its)):
        for o, r in zip(out, _solve(sv, False)):
            assert rel_l2(o, r) <= 1e-5


# padded 30, 44, 60, 64, 80, 88, 108, 125
@pytest.mark.parametrize("length", [24, 35, 48, 51, 64, 70, 86, 100])
def test_no_less_accurate_than_the_radix_passes(length):
    """Smooth padded lengths: both directions of a square window against the
    double operators, with the table DFTs and with the generic passes (the
    time axis of 100 samples is the generic kernels' in both).  Over 1e5
    values the errors of two draws differ by 0.3 % at most: 1 %."""
    sv = _survey((length, length), (length, length), nt=220, wt=100)

    def problem(dtype, generic):
        old = os.environ.get("AGD_GPU_GENERIC")
        os.environ["AGD_GPU_GENERIC"] = "1" if generic else "0"
        try:
            return A.Problem.from_survey(sv, dtype)
        finally:
            if old is None:
                os.environ.pop("AGD_GPU_GENERIC", None)
            else:
                os.environ["AGD_GPU_GENERIC"] = old

    exact = problem(np.float64, True)
    rng = np.random.default_rng(length)
    rec = rng.standard_normal(exact.record_size).astype(np.float32)
    x = rng.standard_normal(2 * exact.model_size).astype(np.float32)
    adj, fwd = exact.adjoint(rec), exact.forward(x)
    exact.close()
    errors = []
    for generic in (False, True):
        p = problem(np.float32, generic)
        errors.append((rel_l2(p.adjoint(rec), adj), rel_l2(p.forward(x), fwd)))
        p.close()
    for table, radix in zip(*errors):
        assert table <= 1.01 * radix


def _space_ms(sv, dtype, generic):
    """Space phases (forward and adjoint) of an iteration, the fastest of eight."""
    old = os.environ.get("AGD_GPU_GENERIC")
    os.environ["AGD_GPU_GENERIC"] = "1" if generic else "0"
    try:
        p = A.Problem.from_survey(sv, dtype)
    finally:
        if old is None:
            os.environ.pop("AGD_GPU_GENERIC", None)
        else:
            os.environ["AGD_GPU_GENERIC"] = old
    p.time_iterations(sv.data, 1.0, sv.n_its, 2, 4)
    ms = min(t[0] + t[5] for t in (p.profile_iteration(1e-3) for _ in range(8)))
    p.close()
    return ms


# space shape, windows, type: padded 3 x 3, 100 x 100 (a plane fills an SM),
# 128 x 128, 75 x 75, 125 x 10
SPEED = [((60, 60), (2, 2), np.float32), ((60, 60), (2, 2), np.float64),
         ((80, 80), (80, 80), np.float32), ((102, 102), (102, 102), np.float32),
         ((102, 102), (102, 102), np.float64), ((60, 60), (60, 60), np.float64),
         ((100, 40), (100, 8), np.float64)]


@pytest.mark.parametrize("space,windows,dtype", SPEED)
def test_not_slower_than_the_radix_passes(space, windows, dtype):
    """A shape goes to the table DFTs only where they are faster (1.1: the
    spread of the timing where both sides are the same kernels)."""
    sv = _survey(space, windows, nt=600, wt=128)
    assert _space_ms(sv, dtype, False) <= 1.1 * _space_ms(sv, dtype, True)


def test_radix_passes_beside_table_products():
    """In double, 64-trace axes (padded 80) keep the radix passes and 65-trace
    ones (82 = 2 x 41) do not: windows of both kinds in one survey."""
    sv = _survey((64, 129), (64, 64))
    prob = A.Problem.from_survey(sv, np.float64)
    assert prob.kernels()["space_fwd"] in ("plane_dft", "line_dft")
    prob.close()
    _check_operators(sv, np.float64, 1)


def _fk_long(w, x=None, y=None):
    """The oracle's fk_forward of x or fk_adjoint of y in extended precision."""
    real = np.longdouble
    nd = len(w.shape)
    h = w.lt // 2
    scale = ((real(w.scaler) * w.space_taper().astype(real))[None, :, None]
             * w.tapers[-1].astype(real)[None, None, :])
    crop = (slice(None), *(slice(0, n) for n in w.shape), slice(0, w.lt))
    if x is not None:
        u = np.fft.irfftn(x, s=w.padded, axes=tuple(range(1, nd + 2))) * real(np.prod(w.padded))
        u = u[crop].reshape(w.n_tw, w.n_traces, w.lt) * scale
        out = np.zeros((w.n_traces, w.conv), real)
        for t in range(w.n_tw):
            out[:, t * h: t * h + w.lt] += u[t]
        return out
    seg = np.stack([y[:, t * h: t * h + w.lt] for t in range(w.n_tw)]) * scale
    u = np.zeros((w.n_tw, *w.padded), real)
    u[crop] = seg.reshape(w.n_tw, *w.shape, w.lt)
    out = np.fft.rfftn(u, axes=tuple(range(1, nd + 2)))
    out[..., 1: 1 + (w.padded[-1] - 1) // 2] *= 2
    return out


@pytest.mark.skipif(np.finfo(np.longdouble).eps > 1e-18, reason="no extended precision")
@pytest.mark.parametrize("length", [24, 36, 40, 48])  # padded 30, 45, 50, 60
def test_double_no_less_accurate_than_the_radix_passes(length):
    """As in float, against extended precision; shots that do not overlap."""
    n, nt = length * length, 260
    zero = np.zeros(n, np.int32)
    sv = S.Survey("one window", [0], [3], [[length, length, 100]], [[0, 0]],
                  [[length, length, nt]], [(3 * nt * np.arange(n)).astype(np.int64)], [zero],
                  [zero], [np.zeros((length, length, nt))], [np.zeros((length, length, nt))], 4)
    plan = O.make_plan(sv.volumes, sv.n_dims, sv.window_shapes, sv.coords, sv.shapes,
                       sv.shottimes, sv.channels, sv.trace_types, None, None, None)
    (w,) = plan.windows
    rng = np.random.default_rng(length)
    size = int(np.prod(w.model_shape))
    m = rng.standard_normal(2 * size)
    y = _fk_long(w, x=(m[0::2].astype(np.longdouble)
                       + 1j * m[1::2].astype(np.longdouble)).reshape(w.model_shape))
    rec = rng.standard_normal(plan.cfg.total)
    traces = np.zeros((n, w.conv), np.longdouble)
    fwd = np.zeros(plan.cfg.total, np.longdouble)
    for i, (off, ts, k) in enumerate(w.blend):
        traces[i, ts: ts + k] = rec[off: off + k]
        fwd[off: off + k] += y[i, ts: ts + k]
    adj = _fk_long(w, y=traces).reshape(-1)
    errors = []
    for generic in (False, True):
        old = os.environ.get("AGD_GPU_GENERIC")
        os.environ["AGD_GPU_GENERIC"] = "1" if generic else "0"
        try:
            p = A.Problem.from_survey(sv, np.float64)
        finally:
            if old is None:
                os.environ.pop("AGD_GPU_GENERIC", None)
            else:
                os.environ["AGD_GPU_GENERIC"] = old
        g = p.adjoint(rec)
        g = g[0::2].astype(np.longdouble) + 1j * g[1::2].astype(np.longdouble)
        f = p.forward(m).astype(np.longdouble)
        p.close()
        errors.append([float(np.sqrt(np.sum(abs(a - b) ** 2) / np.sum(abs(b) ** 2)))
                       for a, b in ((g, adj), (f, fwd))])
    for table, radix in zip(*errors):
        assert table <= 1.01 * radix
