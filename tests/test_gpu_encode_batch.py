"""GPU tests of the DVB-T2 encoder's batch sizes: one frame per CTA, four frames
per CTA, a last group of one to three frames, and every task width (the codes'
row-group counts), against the oracle's encoder; bits are equal."""
import numpy as np
import pytest

import gf2_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("idx", range(12))
@pytest.mark.parametrize("frames", [1, 1185, 2371])
def test_encode_batches(gpu, oracle, idx, frames):
    import torch
    code = g.LdpcCode.dvb_t2_normal(idx) if idx < 6 else g.LdpcCode.dvb_t2_short(idx - 6)
    ocode = oracle.Code.dvbt2(idx // 6, idx % 6)
    rng = np.random.default_rng(idx)
    some = rng.integers(0, 2, (5, code.k()), dtype=np.uint8)
    ref = ocode.encode(some)
    at = rng.integers(0, 5, frames)
    at[-3:] = (0, 3, 4)[-min(3, frames):]
    packed = g.pack_bits(some, code.k())[at]
    packed[:, -1] |= np.uint64(0) if code.k() % 64 == 0 else np.uint64(1) << np.uint64(63)  # bits beyond k are ignored
    cw = g.LdpcEncoder(code).encode_packed(torch.from_numpy(packed.view(np.int64)).to(gpu))
    want = g.pack_bits(ref, code.n())[at]
    assert (cw.cpu().numpy().view(np.uint64) == want).all()
    _, w = code.syndrome_batch(cw)
    assert int(w.abs().sum()) == 0
