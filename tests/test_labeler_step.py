"""The labeler's grouped Viterbi step, restated in float32 numpy: a group's
largest log-likelihood and its position from two rounds of pairwise
comparisons, decisions as signs of differences, and the margin test that sends
close frames to the generic rows.  A row either gets the generic row's value
and source or its frame is flagged.  The traceback word that carries the
decisions gives each state its generic source, and the probabilities that
travel back along it the generic sums.  Log-likelihoods: exact ties, a later
state a few ulps below the group's largest, -inf groups and mixtures.  The
transition constants are the reference's at its defaults, where each 9-way
row's are equal within the source groups 5..8 and 9..12."""
import numpy as np
import pytest

import oracle
from hw_b200 import workloads

F32 = np.float32
NINF = F32(-np.inf)
TOL = F32(2.0 ** -21)
ROWS = (0, 5, 6, 7, 8)
SOURCES = (0, 5, 6, 7, 8, 9, 10, 11, 12)


def generic_row(T, R, score, ll):
    """Candidates (score + T[R][s]) + ll[s] in source order; ties go to the
    later source (the labeler's Pick)."""
    mv, win = None, None
    for s in SOURCES:
        v = F32(F32(score + T[R, s]) + ll[s])
        if mv is None or v >= mv:
            mv, win = v, s
    return mv, win


def _frames(rng, n):
    """log-likelihood vectors with the situations that matter."""
    out = []
    for _ in range(n):
        base = F32(rng.uniform(-3000.0, -10.0))
        ll = (base + rng.normal(0, 5, 13)).astype(F32)
        kind = rng.integers(0, 6)
        if kind == 1:       # exact ties inside the groups
            ll[6] = ll[5]
            ll[11] = ll[9]
        elif kind == 2:     # a later state a few ulps below the group's largest
            for g in (5, 9):
                p = g + rng.integers(0, 3)
                q = p + 1 + rng.integers(0, g + 3 - p)
                ll[q] = np.nextafter(ll[p], NINF, dtype=F32)
                for _ in range(rng.integers(0, 4)):
                    ll[q] = np.nextafter(ll[q], NINF, dtype=F32)
                if ll[q] > max(ll[g:g + 4][ll[g:g + 4] != ll[q]], default=NINF):
                    ll[p] = np.nextafter(ll[q], F32(np.inf), dtype=F32)
        elif kind == 3:     # a group of -inf (non-ROI frames)
            ll[5:9] = NINF
        elif kind == 4:     # every state but the baseline -inf
            ll[1:] = NINF
        elif kind == 5:     # large magnitudes: coarse ulps, many rounding ties
            ll = (F32(-2.0e6) + rng.integers(-3, 4, 13).astype(F32)).astype(F32)
        out.append(ll)
    return out


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
    for R in ROWS:
        assert (T[R, 5:9] == T[R, 5]).all() and (T[R, 9:13] == T[R, 9]).all()
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


# ---- the traceback word -----------------------------------------------------------
# Bit 2 s + 1 of state s: the sign of its last decision (1: not the last
# source, or not group B), bit 2 s of a 9-way state the sign of the one before
# (1: state 0); bits 31..29 and 28..26 the signs of groups A's and B's three
# differences.  A two-way state's bit 2 s is not defined.

POSITIONS = 0x2367


def pack(last, before, e_a, e_b, junk):
    w = int(junk) & sum(1 << (2 * s) for s in range(13) if s not in ROWS)
    for s in range(13):
        w |= int(last[s]) << (2 * s + 1)
        if s in ROWS:
            w |= int(before[s]) << (2 * s)
    for i in range(3):
        w |= int(e_a[i]) << (31 - i) | int(e_b[i]) << (28 - i)
    return w


def trace_source(w, state):
    v = w >> (2 * state)
    first, nine = (v >> 1) & 1, state in ROWS
    if nine and first and v & 1:
        return 0
    pos = (POSITIONS >> ((w >> (25 + 3 * first)) & 14)) & 3
    return 5 + 4 * nine - 4 * first + (pos if nine else (state + 3) & 3)


def back_step(w, p):
    """The labeler's sums of the probabilities at each source."""
    bit = lambda i: (w >> i) & 1      # noqa: E731
    z, a, b = [], [], []
    for s in ROWS:
        last_b, via_a = not bit(2 * s + 1), not bit(2 * s)
        b.append(p[s] if last_b else F32(0))
        rest = F32(0) if last_b else p[s]
        a.append(rest if via_a else F32(0))
        z.append(F32(0) if via_a else rest)
    out = np.zeros(13, F32)
    out[0] = F32(F32(F32(F32(z[0] + z[1]) + z[2]) + z[3]) + z[4])
    pos_a, pos_b = (POSITIONS >> ((w >> 28) & 14)) & 3, (POSITIONS >> ((w >> 25) & 14)) & 3
    for u in range(4):
        full, down = bit(2 * (1 + u) + 1), bit(2 * (9 + u) + 1)
        out[1 + u] = F32((p[1 + u] if full else F32(0)) + (p[9 + u] if down else F32(0)))
        in_a, in_b = pos_a == u, pos_b == u
        t = F32((a[0] if in_a else F32(0)) + (F32(0) if full else p[1 + u]))
        v = b[0] if in_b else F32(0)
        for i in range(1, 5):
            t = F32(t + a[i]) if in_a else t
            v = F32(v + b[i]) if in_b else v
        out[5 + u] = F32(t + (F32(0) if down else p[9 + u]))
        out[9 + u] = v
    return out


def test_word_gives_the_generic_sources():
    T = oracle.transition_matrix(workloads.chip_config()).astype(F32)
    t_max = F32(max(abs(T[R, c]) for R in ROWS for c in (0, 5, 9)))
    rng = np.random.default_rng(29)
    checked = 0
    for ll in _frames(rng, 3000):
        score = rng.uniform(-40.0, 0.0, 9).astype(F32)
        sco = np.concatenate([score, score[5:9]])          # the down states score as the up states
        A, B = group(ll[5:9]), group(ll[9:13])
        s_max = F32(np.abs(sco[list(ROWS)]).max())
        if close(A[2], A[0], s_max, t_max) or close(B[2], B[0], s_max, t_max):
            continue
        last, before, want = np.zeros(13, int), np.zeros(13, int), np.zeros(13, int)
        with np.errstate(invalid="ignore"):
            for s in range(13):
                if s in ROWS:
                    want[s] = generic_row(T, s, sco[s], ll)[1]
                    c0 = F32(F32(sco[s] + T[s, 0]) + ll[0])
                    cA, cB = F32(F32(sco[s] + T[s, 5]) + A[0]), F32(F32(sco[s] + T[s, 9]) + B[0])
                    before[s], last[s] = sign(F32(cA - c0)), sign(F32(cB - max(c0, cA, cB)))
                else:
                    one, two = (s, s + 4) if s < 5 else (s - 8, s - 4)
                    c1, c2 = F32(F32(sco[s] + T[s, one]) + ll[one]), F32(F32(sco[s] + T[s, two]) + ll[two])
                    want[s] = two if c2 >= c1 else one
                    last[s] = sign(F32(c2 - c1))
        w = pack(last, before, [sign(e) for e in A[2]], [sign(e) for e in B[2]], rng.integers(0, 1 << 26))
        assert [trace_source(w, s) for s in range(13)] == want.tolist(), ll
        checked += 1
    assert checked > 1000


def test_probabilities_travel_back_as_the_generic_scatter_sums_them():
    rng = np.random.default_rng(31)
    for _ in range(4000):
        w = int(rng.integers(0, 1 << 32))
        p = np.where(rng.random(13) < 0.2, 0, rng.random(13)).astype(F32)
        want = np.zeros(13, F32)
        for s in range(13):
            to = trace_source(w, s)
            want[to] = F32(want[to] + p[s])
        assert back_step(w, p).tobytes() == want.tobytes(), hex(w)


def test_position_table_is_the_pairwise_rule():
    """All eight sign combinations of a group's three differences."""
    for e1 in (0, 1):
        for e2 in (0, 1):
            for e3 in (0, 1):
                w = pack(np.zeros(13), np.zeros(13), (e1, e2, e3), (e1, e2, e3), 0)
                want = (1 - e1) if e3 else 2 + (1 - e2)
                assert trace_source(w, 0) == 9 + want
                assert trace_source(w | 2, 0) == 5 + want
