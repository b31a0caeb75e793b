"""The empty-box crossing of the skipping traversal (vt_device.cuh: skip_cross), restated in binary32
and checked against iterating the DDA step it replaces (trace.frag:83-86) until some axis takes its
last move to the box face: side distances, moves per axis and the axes stepped on the last iteration
are identical (at the event where a corrected crossing stops), or the restatement says that the lane
iterates.  Step counts come from an approximate quotient in the kernel: they are perturbed here, so that
every correction is met, and boxes one move deep and exact ties are frequent."""
import math
import random

import pytest

from test_crossing import INF, add_chain, f32, fadd, fma, fminf, literal, random_case


def crossing(s, d, n, errs):
    """(sides, moves, mask, corrected) at the first event left out or at the box's exit, or None where
    one correction is not enough and the lane iterates."""
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
            cnt.append(max(min(max(q, 0) + errs[i], n[i] - 1), 0))
    h = [add_chain(s[i], d[i], cnt[i] - 1) for i in range(3)]
    ts = h[first]
    u = [fadd(h[i], d[i]) if cnt[i] else s[i] for i in range(3)]
    over = [bool(cnt[i] and h[i] > ts) for i in range(3)]
    corrected = min(u) <= ts or any(over)
    if corrected:
        ts = min(ts, min(u))
        over = [bool(cnt[i] and h[i] > ts) for i in range(3)]
        if any(over[i] and fma(f32(-0.5), d[i], h[i]) > ts for i in range(3)):
            return None
        more = [u[i] == ts for i in range(3)]
        w = [h[i] if over[i] else (fadd(u[i], d[i]) if more[i] else u[i]) for i in range(3)]
        h = [u[i] if more[i] else h[i] for i in range(3)]
        cnt = [cnt[i] + more[i] - over[i] for i in range(3)]
        u = w
        if min(u) <= ts:
            return None
    return u, cnt, [bool(cnt[i] and h[i] == ts) for i in range(3)], corrected


def stop_at(s, d, st, moves):
    """The DDA step iterated until the axes have taken `moves` steps."""
    s, got = list(s), [0, 0, 0]
    while got != list(moves):
        mn = fminf(fminf(s[0], s[1]), s[2])
        m = [s[i] == mn for i in range(3)]
        for i in range(3):
            if m[i]:
                s[i] = fadd(s[i], d[i])
                got[i] += 1
        if any(got[i] > moves[i] for i in range(3)):
            return None
    return s, got, m


@pytest.mark.parametrize("far", [False, True])
def test_crossing_equals_the_iterated_step(far):
    rng = random.Random(3 + far)
    iterated = corrected = 0
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
        got = crossing(s, d, n, errs)
        if got is None:
            iterated += 1
            continue
        # a correction may stop at an event before the exit: the state is then the iteration's there,
        # with no axis past the box
        corrected += got[3]
        want = stop_at(s, d, st, got[1]) if got[3] else literal(s, d, st, n)
        assert want is not None and all(got[1][i] <= n[i] for i in range(3) if st[i]), (case, s, d, st, n, errs, got)
        assert list(got[1]) == list(want[1]) and got[2] == want[2], (case, s, d, st, n, errs, got, want)
        assert all(g == w for g, w in zip(got[0], want[0])), (case, s, d, st, n, errs, got, want)
    assert corrected > 20 and iterated < 2500  # both kinds are met, and not everything iterates
