"""Outer BCH decoding where a locator loses a coefficient on the way: once the
first root has been divided out, coefficient j of what is left, of degree d, is
zero.  Every degree and coefficient the masked scan runs, both fields: the sent
message comes back and every error is counted."""
import numpy as np
import pytest

import gf2_b200 as g

pytestmark = pytest.mark.gpu


def field(m, prim):
    exp, log, x = np.zeros(2 << m, np.int64), np.zeros(1 << m, np.int64), 1
    N = (1 << m) - 1
    for e in range(N):
        exp[e], log[x] = x, e
        x <<= 1
        if x >> m:
            x ^= prim
    exp[N:2 * N] = exp[:N]
    return exp, log, N


@pytest.mark.parametrize("frame,rate", [(1, 0), (1, 5), (0, 0), (0, 2)])
def test_zero_coefficient_after_the_first_root(gpu, frame, rate):
    code = g.BchCode.dvb_t2(frame, rate)
    n, k, t = code.n(), code.k(), code.t()
    exp, log, N = field(14, 0b100000000101011) if frame == 1 else field(16, 0b10000000000101101)
    mul = lambda a, b: int(exp[log[a] + log[b]]) if a and b else 0
    rng = np.random.default_rng(10 * frame + rate)
    roots = []
    for d in range(3, t):
        for j in range(1, d):
            while True:  # d - 1 roots, and the one that makes coefficient j of the product zero
                pos = rng.choice(np.arange(600, n), d - 1, replace=False)
                e = [1] + [0] * d
                for p in pos:
                    for i in range(d, 0, -1):
                        e[i] ^= mul(e[i - 1], int(exp[p]))
                if not e[j] or not e[j - 1]:
                    continue
                last = (log[e[j]] - log[e[j - 1]]) % N
                if 600 <= last < n and last not in pos:
                    roots.append([int(rng.integers(0, 200)), *map(int, pos), int(last)])
                    break
    msg = rng.integers(0, 2, (len(roots), k)).astype(np.uint8)
    cw = g.unpack_bits(g.BchEncoder(code).encode_words(g.pack_bits(msg)), n)
    for f, r in enumerate(roots):
        for i in r:
            cw[f, n - 1 - i] ^= 1
    out = g.BchDecoder(code).decode_words(g.pack_bits(cw))
    assert (out["corrected"] == [len(r) for r in roots]).all()
    assert (g.unpack_bits(out["msg"], k) == msg).all()
