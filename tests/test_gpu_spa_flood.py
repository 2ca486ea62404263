"""GPU parity tests of the DVB-T2 flooding sum-product kernel: every slot
bucket (regular and irregular row groups), FP32 and FP16 messages, teams of 16
to 2 CTAs per frame, batches of several waves, special channel values.  The
general flooding kernel (an explicit launch shape selects it) runs the same
operations in the same order, so results are equal bit for bit; the exact
numerics also equal the oracle's."""
import numpy as np
import pytest

import gf2_b200 as g

pytestmark = pytest.mark.gpu


def dvb(i):
    return g.LdpcCode.dvb_t2_normal(i) if i < 6 else g.LdpcCode.dvb_t2_short(i - 6)


def special(llr):
    rng = np.random.default_rng(4)
    llr = llr.copy()
    for f in range(llr.shape[0]):
        at = rng.choice(llr.shape[1], 60, replace=False)
        llr[f, at[:10]] = np.inf
        llr[f, at[10:20]] = -np.inf
        llr[f, at[20:30]] = -0.0
        llr[f, at[30:40]] = rng.normal(0, 1, 10) * 1e-30
        llr[f, at[40:50]] = rng.normal(0, 1, 10) * 1e-41
        if f == 0:
            llr[f, at[50:]] = np.nan
    return llr


def equal(a, b, at=None):
    at = slice(None) if at is None else at
    return all(np.array_equal(a[k], b[k][at], equal_nan=k == "beliefs") for k in a)


@pytest.mark.parametrize("msg16", [False, True])
@pytest.mark.parametrize("algo", ["spa", "fast"])
@pytest.mark.parametrize("idx", range(12))
def test_structured_sum_product_equals_general_kernel(gpu, idx, algo, msg16):
    code = dvb(idx)
    _, _, llr = g.awgn_frames(code, 11, 0, 3, g.sigma2_from_ebn0(1.0 + 0.4 * (idx % 6), code.rate()))
    kw = dict(algorithm=g.ALGO_SPA if algo == "spa" else g.ALGO_SPA_FAST, msg_dtype=g.MSG_F16 if msg16 else g.MSG_F32)
    for x in (llr, special(llr)):
        r = g.LdpcDecoder(code, **kw).decode_arrays(x, 7, beliefs=True)
        assert equal(r, g.LdpcDecoder(code, threads_per_block=256, **kw).decode_arrays(x, 7, beliefs=True))


@pytest.mark.parametrize("frames", [1, 12, 40, 100, 301])
def test_team_sizes_equal_oracle(gpu, oracle, frames):
    code, ocode = dvb(6), oracle.Code.dvbt2(1, 0)
    _, _, llr = ocode.channel(5, 0, 3, 1.1)
    o = ocode.decode(llr, 12, algo=1)
    at = np.arange(frames) % 3
    r = g.LdpcDecoder(code, algorithm=g.ALGO_SPA).decode_arrays(llr[at], 12, beliefs=True)
    assert (r["iters"] == o["iters"][at]).all() and (r["conv"] == o["conv"][at]).all()
    assert (r["synd_ok"] == o["synd_ok"][at]).all()
    assert (g.unpack_bits(r["msg"], code.k()) == o["msg"][at]).all()
    assert np.array_equal(r["beliefs"], o["beliefs"][at])
