"""GPU test: a decoder stays usable after others of smaller codes were made.

A kernel's limit of dynamic shared memory belongs to the kernel, and one kernel
serves codes whose tables and frame states differ in size: making a decoder for
the smaller code must not lower the limit under the larger one's launches.  Each
result equals, bit for bit, the one from before the smaller decoder existed."""
import ctypes

import numpy as np
import pytest

import gf2_b200 as g
from gf2_b200 import _capi as C

pytestmark = pytest.mark.gpu

LAYERED16 = dict(schedule=g.SCHED_LAYERED, msg_dtype=g.MSG_F16)
N, S = g.LdpcCode.dvb_t2_normal, g.LdpcCode.dvb_t2_short


def qc(z):
    base = [[(7 * r + 3 * c) % z if (r + c) % 3 else -1 for c in range(12)] for r in range(6)]
    return g.LdpcCode.from_quasi_cyclic(g.QuasiCyclicLdpc(base, z))


PAIRS = {
    "min-sum, normal 2/3 and short 2/3": (lambda: N(2), lambda: S(2), {}),
    "min-sum, normal 1/2 and short 1/2": (lambda: N(0), lambda: S(0), {}),
    "min-sum, state on chip": (lambda: qc(360), lambda: qc(40), {}),
    "sum-product, normal 2/3 and short 2/3": (lambda: N(2), lambda: S(2), dict(algorithm=g.ALGO_SPA)),
    "layered min-sum, short 4/5 and short 3/4": (lambda: S(4), lambda: S(3), LAYERED16),
    "layered sum-product, short 4/5 and short 3/4": (lambda: S(4), lambda: S(3), dict(algorithm=g.ALGO_SPA_FAST, **LAYERED16)),
    "layered min-sum, quasi-cyclic": (lambda: qc(384), lambda: qc(360), LAYERED16),
}


def llrs(gpu, code, frames):
    import torch
    gen = torch.Generator(device=gpu).manual_seed(5)
    return torch.randn((frames, code.n()), generator=gen, device=gpu) * 2.0 + 2.0


def equal(a, b):
    import torch
    return all(torch.equal(a[k], b[k]) for k in b)


@pytest.mark.parametrize("pair", PAIRS)
def test_a_smaller_code_leaves_the_larger_one_its_shared_memory(gpu, pair):
    large, small, kw = PAIRS[pair]
    code = large()
    # frame counts: a team of CTAs per frame, and more frames than SMs
    xs = [llrs(gpu, code, f) for f in (1, 700)]
    dec = g.LdpcDecoder(code, **kw)
    ref = [dec.decode_tensors(x, 3) for x in xs]
    other = small()
    for _ in range(2):
        g.LdpcDecoder(other, **kw).decode_tensors(llrs(gpu, other, 1), 3)
        assert all(equal(dec.decode_tensors(x, 3), r) for x, r in zip(xs, ref))


def test_noalloc_decode_after_a_smaller_decoder(gpu):
    import torch
    code = N(2)
    x = llrs(gpu, code, 2)

    def noalloc():
        out = dict(msg=torch.zeros((2, g.words(code.k())), dtype=torch.int64, device=gpu),
                   iters=torch.zeros(2, dtype=torch.int32, device=gpu),
                   conv=torch.zeros(2, dtype=torch.uint8, device=gpu), synd_ok=torch.zeros(2, dtype=torch.uint8, device=gpu))
        C.check(C.lib.gf2c_decode_batch_noalloc(code.handle, ctypes.c_void_p(x.data_ptr()), 2, 3,
                                                *(ctypes.c_void_p(out[k].data_ptr()) for k in ("msg", "iters", "conv", "synd_ok")),
                                                None))
        torch.cuda.synchronize()
        return out

    ref = noalloc()
    g.LdpcDecoder(S(2))
    assert equal(noalloc(), ref)


def test_encoders_and_syndromes_of_two_sizes_in_turn(gpu):
    import torch
    codes = [N(5), S(0), N(5), S(0)]
    words = [torch.from_numpy(np.arange(f * g.words(c.k()), dtype=np.int64).reshape(f, -1)).to(gpu)
             for c, f in zip(codes, (3, 3, 2000, 2000))]
    for c, w in zip(codes, words):
        if c.k() % 64:
            w[:, -1] &= (1 << (c.k() % 64)) - 1
        cw = g.LdpcEncoder(c).encode_packed(w)
        _, weight = c.syndrome_batch(cw)
        assert int(weight.abs().sum()) == 0
