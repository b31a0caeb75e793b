"""How often the empty-box crossing (vt_device.cuh: skip_cross, restated in test_skip_crossing.py) needs its
correction and its fallback, and what the fallback does.  With the kernel's own estimates a box is crossed
without either in nearly every case; rays whose axes step in lock-step are corrected, not iterated; where the
lane iterates, it stops at the first event that leaves the brick it started in, with the state of the
literal DDA there (trace.frag:83-86), and never past the box."""
import random

from test_crossing import fadd, fminf, random_case
from test_skip_crossing import crossing, stop_at


def iterate(s, d, st, v):
    """The kernel's fallback: the step until a coordinate leaves its 8-voxel brick."""
    s, moves = list(s), [0, 0, 0]
    while True:
        mn = fminf(fminf(s[0], s[1]), s[2])
        m = [bool(s[a] == mn) for a in range(3)]
        for a in range(3):
            if m[a]:
                s[a] = fadd(s[a], d[a])
                moves[a] += 1
        if any(((v[a] + st[a] * moves[a]) ^ v[a]) & ~7 for a in range(3)):
            return s, moves, m


def box(rng, st):
    """A start voxel and the moves to the faces of a box of 1 to 4 bricks forward (axis_moves)."""
    v = [rng.randint(64, 127) for _ in range(3)]
    n = [8 * rng.randint(1, 4) - ((v[a] & 7) if st[a] >= 0 else 7 - (v[a] & 7)) for a in range(3)]
    return v, n


def test_near_rays_hardly_ever_need_the_correction():
    rng = random.Random(11)
    cases = corrected = iterated = 0
    while cases < 1500:
        s, d, st, _ = random_case(rng)
        stepping = [a for a in range(3) if st[a]]
        # a camera or bounce ray: no two axes in lock-step, no further than the starts of random_case
        if len({float(d[a]) for a in stepping}) < len(stepping):
            continue
        s = [s[a] if not st[a] else type(s[a])(float(d[a]) * rng.random() * rng.choice((1, 20, 200))) for a in range(3)]
        _, n = box(rng, st)
        got = crossing(s, d, n, [0, 0, 0])
        cases += 1
        iterated += got is None
        corrected += got is not None and got[3]
    # 1%; on the GPU 6e-5 to 3e-3 of a cave's and a terrain's crossings are corrected
    assert corrected <= 15 and iterated == 0, (corrected, iterated)


def test_lock_step_rays_are_corrected_not_iterated():
    rng = random.Random(12)
    cases = iterated = 0
    while cases < 1500:
        s, d, st, _ = random_case(rng)
        if 0 in st:
            continue
        i, j = rng.sample(range(3), 2)
        s[i] = type(s[i])(float(d[i]) * rng.random())
        s[j], d[j] = s[i], d[i]  # the same event times on two axes
        k = 3 - i - j
        s[k] = type(s[k])(float(d[k]) * rng.random())
        _, n = box(rng, st)
        cases += 1
        iterated += crossing(s, d, n, [0, 0, 0]) is None
    assert iterated <= 15, iterated


def test_the_fallback_stops_inside_the_box_with_the_literal_state():
    rng = random.Random(13)
    met = 0
    for _ in range(6000):
        s, d, st, _ = random_case(rng)
        s = [x if not st[a] else type(x)(float(x) * 32.0 + 32768.0) for a, x in enumerate(s)]  # far-travelled
        v, n = box(rng, st)
        if crossing(s, d, n, [rng.choice((-2, -1, 1, 2)) for _ in range(3)]) is not None:
            continue
        met += 1
        got = iterate(s, d, st, v)
        assert all(got[1][a] <= n[a] for a in range(3) if st[a]), (s, d, st, v, n, got)
        want = stop_at(s, d, st, got[1])
        assert want is not None
        assert list(want[1]) == got[1] and [bool(x) for x in want[2]] == got[2], (s, d, st, v, n, got, want)
        assert all(g == w for g, w in zip(got[0], want[0]))
    assert met > 200, met
