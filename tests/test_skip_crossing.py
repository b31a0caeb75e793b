"""The empty-box crossing of the skipping traversal (vt_device.cuh: skip_cross), restated in binary32
and checked against iterating the DDA step it replaces (trace.frag:83-86) until some axis takes its
last move to the box face: side distances, moves per axis and the axes stepped on the last iteration
are identical, or the restatement says that the lane iterates.  Step counts come from an approximate
quotient in the kernel: they are perturbed here, so that every check that sends a lane to the
iteration is met, and boxes one move deep and exact ties are frequent."""
import math
import random

import pytest

from test_crossing import INF, add_chain, f32, fadd, fma, fminf, literal, random_case


def crossing(s, d, n, errs):
    """(sides, moves, mask), or None where a check fails and the lane iterates."""
    a = [fma(f32(n[i] - 1), d[i], s[i]) if not math.isinf(s[i]) else f32(INF) for i in range(3)]
    amin = fminf(fminf(a[0], a[1]), a[2])
    first = next(i for i in range(3) if a[i] == amin)
    cnt = []
    for i in range(3):
        if i == first:
            cnt.append(n[i])
        elif math.isinf(s[i]):
            cnt.append(0)
        else:
            q = math.floor(float(f32(amin - s[i])) / float(d[i])) + 1
            cnt.append(min(max(q, 0) + errs[i] if q > 0 else max(errs[i], 0), n[i] - 1))
            cnt[i] = max(cnt[i], 0)
    h = [add_chain(s[i], d[i], cnt[i] - 1) for i in range(3)]
    ts = h[first]
    u = [fadd(h[i], d[i]) if cnt[i] else s[i] for i in range(3)]
    if min(u) <= ts or any(cnt[i] and h[i] > ts for i in range(3)):
        return None
    return u, cnt, [bool(cnt[i] and h[i] == ts) for i in range(3)]


@pytest.mark.parametrize("far", [False, True])
def test_crossing_equals_the_iterated_step(far):
    rng = random.Random(3 + far)
    iterated = 0
    for case in range(2500):
        s, d, st, n = random_case(rng)
        if far:
            s = [x if math.isinf(x) else f32(float(x) * 32.0 + 32768.0) for x in s]
        if case % 3 == 0:
            n = [min(x, rng.randint(1, 2)) for x in n]
        if case % 5 == 0:  # another axis's exit in the neighbourhood of the first one's
            i, j = rng.sample(range(3), 2)
            if st[i] and st[j]:
                t = add_chain(s[i], d[i], n[i] - 1)
                s[j] = f32(max(0.0, float(t) - (n[j] - 1) * float(d[j])) * (1.0 + rng.randint(-2, 2) * 2.0 ** -24))
        errs = [0, 0, 0] if case % 2 else [rng.choice((-1, 0, 0, 1)) for _ in range(3)]
        want = literal(s, d, st, n)
        got = crossing(s, d, n, errs)
        if got is None:
            iterated += 1
            continue
        assert list(got[1]) == list(want[1]) and got[2] == want[2], (case, s, d, st, n, errs, got, want)
        assert all(g == w for g, w in zip(got[0], want[0])), (case, s, d, st, n, errs, got, want)
    assert 0 < iterated < 2500
