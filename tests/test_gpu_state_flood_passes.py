"""Flooding min-sum by every kind of kernel the check-state decoder has: the frame's
state on chip or in the workspace, with structured tables, without (Z above the
descriptors' range), or by each frame's code in a mixed batch, one CTA per frame
and teams; bit for bit what the oracle gives."""
import numpy as np
import pytest

import gf2_b200 as g

pytestmark = pytest.mark.gpu


def base(rows, cols, z, seed):
    rng = np.random.default_rng(seed)
    b = [[int(rng.integers(0, z)) if rng.random() < 0.35 else -1 for _ in range(cols)] for _ in range(rows)]
    for r in range(rows):
        b[r][cols - rows + r] = 0
    return b


CODES = {"on chip": (6, 12, 100), "in the workspace": (12, 24, 1000), "without tables": (3, 6, 2500)}


def make(oracle, name):
    rows, cols, z = CODES[name]
    b = base(rows, cols, z, z)
    return g.LdpcCode.from_quasi_cyclic(g.QuasiCyclicLdpc(b, z)), oracle.Code.qc(b, z)


@pytest.mark.parametrize("frames", [1, 40, 200])
@pytest.mark.parametrize("name", CODES)
def test_one_code(gpu, oracle, name, frames):
    code, ocode = make(oracle, name)
    x = np.random.default_rng(frames).normal(1.2, 1.3, (2, code.n())).astype(np.float32)
    o = ocode.decode(x, 4)
    at = np.arange(frames) % 2
    r = g.LdpcDecoder(code).decode_arrays(x[at], 4, beliefs=True)
    assert (r["iters"] == o["iters"][at]).all() and (r["conv"] == o["conv"][at]).all()
    assert (g.unpack_bits(r["msg"], code.k()) == o["msg"][at]).all()
    assert np.array_equal(r["beliefs"], o["beliefs"][at])


@pytest.mark.parametrize("frames", [3, 300])
@pytest.mark.parametrize("names", [("on chip", "in the workspace"), ("in the workspace", "without tables"),
                                   ("on chip", "without tables")])
def test_mixed(gpu, oracle, names, frames):
    codes, ocodes = zip(*(make(oracle, n) for n in names))
    rng = np.random.default_rng(frames)
    xs = [rng.normal(1.2, 1.3, c.n()).astype(np.float32) for c in codes]
    os_ = [o.decode(x[None], 4) for o, x in zip(ocodes, xs)]
    cid = np.arange(frames) % 2
    off = np.cumsum([0] + [codes[c].n() for c in cid])[:-1]
    w = [g.words(c.k()) for c in codes]
    moff = np.cumsum([0] + [w[c] for c in cid])[:-1]
    m = g.LdpcDecoder(codes[0], codes=list(codes)).decode_mixed_arrays(
        np.concatenate([xs[c] for c in cid]), off, cid, np.full(frames, 4), moff)
    for c in (0, 1):
        k = codes[c].k()
        assert (m["iters"][cid == c] == os_[c]["iters"][0]).all() and (m["conv"][cid == c] == os_[c]["conv"][0]).all()
        got = np.stack([m["msg"][moff[f]:moff[f] + w[c]] for f in np.nonzero(cid == c)[0]])
        assert (g.unpack_bits(got, k) == os_[c]["msg"][0]).all()
