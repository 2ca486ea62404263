"""GPU tests of the layered training kernels of the DVB-T2 codes: loss and
gradients against the FP64 oracle for every slot bucket, with the tolerance of
the existing gradient checks (max abs error 2e-3 of the largest component), and
the final soft output equal to the inference decoder's posteriors bit for bit."""
import ctypes

import numpy as np
import pytest

import gf2_b200 as g
from gf2_b200 import _capi as C
from gf2_b200.learned import NmsTrainer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("idx,frames", [(0, 2), (1, 1), (2, 3), (5, 1), (6, 3), (7, 2), (9, 3), (11, 2), (6, 150)])
def test_layered_gradients_and_soft_output(gpu, oracle, idx, frames):
    import torch
    code = g.LdpcCode.dvb_t2_normal(idx) if idx < 6 else g.LdpcCode.dvb_t2_short(idx - 6)
    ocode = oracle.Code.dvbt2(idx // 6, idx % 6)
    T = 3
    tr = NmsTrainer(code, iterations=T, batch=frames, schedule=g.SCHED_LAYERED, device=gpu)
    rng = np.random.default_rng(idx)
    P = np.stack([0.6 + 0.4 * rng.random((T, tr.L)), 0.3 * rng.random((T, tr.L))]).astype(np.float32)
    tr.P.copy_(torch.from_numpy(P))
    distinct = min(frames, 3)
    _, ocw, ollr = ocode.channel(21, 0, distinct, 2.0)
    at = np.arange(frames) % distinct
    llr = torch.from_numpy(np.ascontiguousarray(ollr[at])).to(gpu)
    cw = torch.from_numpy(g.pack_bits(ocw[at], code.n()).view(np.int64)).to(gpu)
    soft = torch.zeros((frames, code.n()), dtype=torch.float32, device=gpu)
    vp = lambda t: ctypes.c_void_p(t.data_ptr())
    C.check(C.lib.gf2c_nms_loss_grad(tr._h, vp(llr), vp(cw), frames, vp(tr.P[0]), vp(tr.P[1]), vp(tr.G[0]),
                                     vp(tr.G[1]), vp(tr.loss_buf), vp(soft), None))
    torch.cuda.synchronize()
    dec = g.LdpcDecoder(code, algorithm=g.ALGO_NMS, schedule=g.SCHED_LAYERED, nms_alpha=P[0], nms_beta=P[1],
                        early_stop=False)
    assert torch.equal(soft, dec.decode_tensors(llr, T, beliefs=True)["beliefs"])
    if frames > 8:  # repeated frames: the mean over the batch, not a new oracle run
        return
    loss, ga, gb, _ = ocode.nms_loss_grad(ollr[at], ocw[at], T, P[0], P[1], layered=True)
    assert abs(float(tr.loss_buf.item()) - loss) <= 2e-3 * abs(loss)
    for got, want in ((tr.G[0].cpu().numpy(), ga), (tr.G[1].cpu().numpy(), gb)):
        assert np.abs(got - want).max() <= 2e-3 * np.abs(want).max()
