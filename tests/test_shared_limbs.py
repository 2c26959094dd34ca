"""The carry rules of the shared-memory accumulators (smem_fix_add,
smem_add_s64 and smem_count_add in gr_internal.cuh), restated on 32-bit words
and compared with plain integers at the values where a carry runs through
one, two or three words."""
import itertools

M = 0xFFFFFFFF
EDGES = [0, 1, M - 1, M, M + 1, (M << 32) | M, (M - 1) << 32, 1 << 62, (1 << 63) - 1]
VALUES = sorted({s * e for e in EDGES for s in (1, -1) if -(1 << 63) <= s * e < 1 << 63})


def _atomic_add(w, i, v):
    old = w[i]
    w[i] = (old + v) & M
    return old


def _fix_add(w, v):
    v0, v1 = v & M, (v >> 32) & M
    o0 = _atomic_add(w, 0, v0)
    c0 = 1 if (o0 + v0) & M < o0 else 0
    h = (v1 + c0) & M
    o1 = _atomic_add(w, 1, h)
    up = (-1 if v < 0 else 0) + (1 if (o1 + h) & M < o1 or h < c0 else 0)
    if up:
        o2 = _atomic_add(w, 2, up & M)
        if o2 == (0 if up < 0 else M):
            _atomic_add(w, 3, up & M)


def _add_s64(w, v):
    v0 = v & M
    old = _atomic_add(w, 0, v0)
    h = ((v >> 32) & M) + (1 if (old + v0) & M < old else 0) & M
    if h:
        _atomic_add(w, 1, h)


def _count_add(w, n):
    old = _atomic_add(w, 0, n)
    if (old + n) & M < old:
        _atomic_add(w, 1, 1)


def _value(w):
    return sum(x << (32 * i) for i, x in enumerate(w))


def test_fix_add_equals_128_bit_integers():
    for start in itertools.product((0, 1, M), repeat=4):
        for v in VALUES:
            w = list(start)
            _fix_add(w, v)
            assert _value(w) == (_value(start) + v) % (1 << 128), (start, v)


def test_partials_equal_64_bit_integers():
    for start in itertools.product((0, 1, M), repeat=2):
        for v in VALUES:
            w = list(start)
            _add_s64(w, v)
            assert _value(w) == (_value(start) + v) % (1 << 64), (start, v)


def test_counts_equal_64_bit_integers():
    for start in itertools.product((0, 1, M - 1, M), (0, 1)):
        for n in (1, 2, 3):
            w = list(start)
            _count_add(w, n)
            assert _value(w) == _value(start) + n
