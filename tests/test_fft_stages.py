"""The transforms' generic radix restated lane by lane: every index inside its buffer, every input pair combined by one
lane, every output written by one lane, and the result against numpy's transform, for a warp and a block per row pair."""
import numpy as np
import pytest


def plan(n):
    """The radices of the transform: odd ones first, any prime by the generic stage, then fours and a two."""
    radices, odd = [], n
    while odd % 2 == 0:
        odd //= 2
    even = n // odd
    for r in (5, 3):
        while odd % r == 0:
            radices.append(r)
            odd //= r
    r = 7
    while r * r <= odd:
        while odd % r == 0:
            radices.append(r)
            odd //= r
        r += 2
    if odd > 1:
        radices.append(odd)
    while even % 4 == 0:
        radices.append(4)
        even //= 4
    return radices + ([2] if even == 2 else [])


def lanes_walk(lane, step, items, count):
    """(u, e) of a lane's work items, as the kernel advances them without divisions."""
    du, u = step // items, lane // items
    de, e = step - du * items, lane - u * items
    for _ in range(lane, count * items, step):
        assert 0 <= u < count and 0 <= e < items
        yield u, e
        u, e = u + du, e + de
        if e >= items:
            e, u = e - items, u + 1


def stage_any(x, n, R, s, step, tw):
    items, h = n // R, R // 2
    seen = set()
    for lane in range(step):
        for u, e in lanes_walk(lane, step, items, h):
            i, j = e + (u + 1) * items, e + (R - 1 - u) * items
            assert i != j and not {i, j} & seen and 0 <= min(i, j) and max(i, j) < n
            seen |= {i, j}
            x[i], x[j] = x[i] + x[j], x[i] - x[j]
    assert len(seen) == n - items
    y, written = np.zeros(n, complex), set()

    def put(o, v):
        assert 0 <= o < n and o not in written
        written.add(o)
        y[o] = v

    t = np.arange(1, h + 1)
    for lane in range(step):
        for u, e in lanes_walk(lane, step, items, h + 1):
            p, q = e // s, e % s
            w = tw[t * u * items % n]
            c = x[e] + np.sum(w.real * x[e + t * items])
            d = np.sum(w.imag * x[e + (R - t) * items])
            assert p * s * (R - u) < n or u == 0
            put(q + s * (R * p + u), (c - 1j * d) * np.conj(tw[p * s * u]))
            if u:
                put(q + s * (R * p + R - u), (c + 1j * d) * np.conj(tw[p * s * (R - u)]))
    assert len(written) == n
    return y


def transform(x, step):
    n, s = len(x), 1
    tw = np.exp(2j * np.pi * np.arange(n) / n)
    for R in plan(n):
        if R > 5:
            x = stage_any(x.copy(), n, R, s, step, tw)
        else:
            e = np.arange(n // R)
            p, q = e // s, e % s
            b = np.fft.fft(x.reshape(R, n // R), axis=0)
            y = np.zeros(n, complex)
            for u in range(R):
                y[q + s * (R * p + u)] = b[u] * np.conj(tw[p * u * s])
            x = y
        s *= R
    return x


@pytest.mark.parametrize("step", [32, 128])
@pytest.mark.parametrize("n", [7, 8, 11, 14, 21, 35, 37, 49, 66, 67, 77, 98, 119, 121, 134, 143, 179, 242, 359, 362])
def test_generic_radix(n, step):
    assert np.prod(plan(n)) == n
    rng = np.random.default_rng(n)
    x = rng.normal(size=n) + 1j * rng.normal(size=n)
    want = np.fft.fft(x)
    # sums of at most n terms of size one
    assert np.max(np.abs(transform(x, step) - want)) <= 8 * n * np.finfo(float).eps * np.sqrt(n)
