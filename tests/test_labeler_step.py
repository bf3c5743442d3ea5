"""The labeler's grouped Viterbi step, restated in float32 numpy: a group's
largest log-likelihood and its position from two rounds of pairwise
comparisons, decisions as signs of differences, and the margin test that sends
close frames to the generic rows.  A row either gets the generic row's value
and source or its frame is flagged."""
import numpy as np
import pytest

import oracle
from hw_b200 import workloads
from test_grouped_rows import ROWS, _frames, generic_row

F32 = np.float32
TOL = F32(2.0 ** -21)


def sign(d):
    """The sign bit of a difference; the NaN of two infinities is positive."""
    return 0 if np.isnan(d) else int(np.signbit(d))


def group(v):
    """(largest, position, differences) of a group's four values."""
    with np.errstate(invalid="ignore"):
        e1, e2 = F32(v[1] - v[0]), F32(v[3] - v[2])
        h1, h2 = max(v[0], v[1]), max(v[2], v[3])
        e3 = F32(h2 - h1)
    pos = (1 - sign(e1)) if sign(e3) else 2 + (1 - sign(e2))
    return max(h1, h2), pos, (e1, e2, e3)


def close(es, m, s_max, t_max):
    es = [abs(e) for e in es if not np.isnan(e)]
    if not es or np.isinf(m):
        return bool(es)
    return min(es) <= F32(abs(m) * TOL + F32(s_max * TOL + t_max * TOL))


def grouped_row(T, R, score, ll, A, B):
    with np.errstate(invalid="ignore"):
        c0 = F32(F32(score + T[R, 0]) + ll[0])
        cA, cB = F32(F32(score + T[R, 5]) + A[0]), F32(F32(score + T[R, 9]) + B[0])
        n = max(c0, cA, cB)
        dA, dB = F32(cA - c0), F32(cB - n)
    return n, (9 + B[1]) if not sign(dB) else (5 + A[1]) if not sign(dA) else 0


def test_grouped_step_equals_generic_rows_or_flags_the_frame():
    T = oracle.transition_matrix(workloads.chip_config()).astype(F32)
    t_max = F32(max(abs(T[R, c]) for R in ROWS for c in (0, 5, 9)))
    rng = np.random.default_rng(11)
    flagged = checked = 0
    for ll in _frames(rng, 6000):
        scores = rng.uniform(-40.0, 0.0, 5).astype(F32)
        A, B = group(ll[5:9]), group(ll[9:13])
        s_max = F32(np.abs(scores).max())
        if close(A[2], A[0], s_max, t_max) or close(B[2], B[0], s_max, t_max):
            flagged += 1
            continue
        for R, score in zip(ROWS, scores):
            v0, w0 = generic_row(T, R, score, ll)
            v1, w1 = grouped_row(T, R, score, ll, A, B)
            assert v1.tobytes() == v0.tobytes() and w1 == w0, (R, ll, score)
            checked += 1
    assert flagged > 500 and checked > 10000


@pytest.mark.parametrize("order", [(0, 1, 2, 3), (3, 2, 1, 0), (1, 3, 0, 2), (2, 0, 3, 1)])
def test_group_position_is_the_last_largest(order):
    v = np.array(order, F32)
    assert group(v)[:2] == (v.max(), int(np.argmax(v)))
    assert group(np.full(4, -np.inf, F32))[1] == 3
