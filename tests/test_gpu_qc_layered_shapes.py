"""Layered decoding of QC codes with several checks per thread, every slot count
that has a kernel: the launch shape changes nothing in the results."""
import numpy as np
import pytest

import gf2_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", [g.ALGO_SPA_FAST, g.ALGO_MINSUM])
@pytest.mark.parametrize("slots", [7, 9, 10, 11, 13, 14, 18, 19, 22])
def test_shapes_agree(gpu, slots, algo):
    rng = np.random.default_rng(slots)
    base = [[int(rng.integers(0, 360)) if (c - r) % 24 < slots - (r == 2) else -1 for c in range(24)] for r in range(4)]
    code = g.LdpcCode.from_quasi_cyclic(g.QuasiCyclicLdpc(base, 360))
    x = rng.normal(2.0, 1.5, (3, code.n())).astype(np.float32)
    kw = dict(algorithm=algo, schedule=g.SCHED_LAYERED, msg_dtype=g.MSG_F16)
    r = g.LdpcDecoder(code, **kw).decode_arrays(x, 5, beliefs=True)
    for threads, ctas in ((192, 0), (192, 5), (128, 0)):
        s = g.LdpcDecoder(code, threads_per_block=threads, blocks_per_sm=ctas, **kw).decode_arrays(x, 5, beliefs=True)
        assert all(np.array_equal(r[k], s[k]) for k in r)
