"""GPU parity tests of the DVB-T2 layered kernels: every slot bucket and
placement (regular and irregular row groups, runs of repeated variables, the
staircase's corner), messages in FP16 and FP32, and each launch shape.  The
min-sum family equals the oracle's layered schedule operation for operation;
the SFU sum-product has one arithmetic whatever the shape or the batch, so its
kernels must agree with one another bit for bit (its error against the FP64
judge is tested elsewhere)."""
import numpy as np
import pytest

import gf2_b200 as g

pytestmark = pytest.mark.gpu

THR = [1.2, 1.6, 2.0, 2.5, 3.0, 3.3, 1.0, 1.6, 2.0, 2.4, 2.8, 3.1]


def dvb(i):
    return g.LdpcCode.dvb_t2_normal(i) if i < 6 else g.LdpcCode.dvb_t2_short(i - 6)


def same(a, b):
    return all(np.array_equal(a[k], b[k], equal_nan=k == "beliefs") for k in a)


def special(llr, seed):
    rng = np.random.default_rng(seed)
    llr = llr.copy()
    for f in range(llr.shape[0]):
        at = rng.choice(llr.shape[1], 40, replace=False)
        llr[f, at[:10]] = np.inf
        llr[f, at[10:20]] = -np.inf
        llr[f, at[20:30]] = -0.0
        if f == 0:
            llr[f, at[30:]] = np.nan
    return llr


@pytest.mark.parametrize("msg16", [True, False])
@pytest.mark.parametrize("idx", range(12))
def test_layered_nms_equals_oracle(gpu, oracle, idx, msg16):
    code, ocode = dvb(idx), oracle.Code.dvbt2(idx // 6, idx % 6)
    _, _, llr = ocode.channel(3, 0, 3, THR[idx])
    llr = special(llr, idx)
    rng = np.random.default_rng(idx)
    a = (0.6 + 0.4 * rng.random((2, code.layers()))).astype(np.float32)
    b = (0.3 * rng.random((2, code.layers()))).astype(np.float32)
    o = ocode.decode(llr, 4, algo=3, sched=1, msg16=msg16, alpha=a, beta=b)
    for threads in ((0, 192, 128) if msg16 else (0,)):
        r = g.LdpcDecoder(code, algorithm=g.ALGO_NMS, schedule=g.SCHED_LAYERED, nms_alpha=a, nms_beta=b,
                          msg_dtype=g.MSG_F16 if msg16 else g.MSG_F32,
                          threads_per_block=threads).decode_arrays(llr, 4, beliefs=True)
        assert (r["iters"] == o["iters"]).all() and (r["conv"] == o["conv"]).all()
        assert (r["synd_ok"] == o["synd_ok"]).all()
        assert (g.unpack_bits(r["msg"], code.k()) == o["msg"]).all()
        assert np.array_equal(r["beliefs"], o["beliefs"], equal_nan=True)


@pytest.mark.parametrize("idx", range(12))
def test_layered_sfu_shapes_and_mixed_batches_agree(gpu, idx):
    """One thread per check, two, three; alone and in a mixed batch (with the
    short frames' posteriors on chip, and in the workspace)."""
    code = dvb(idx)
    _, _, llr = g.awgn_frames(code, 5, 0, 5, g.sigma2_from_ebn0(THR[idx], code.rate()))
    kw = dict(algorithm=g.ALGO_SPA_FAST, schedule=g.SCHED_LAYERED, msg_dtype=g.MSG_F16)
    r = g.LdpcDecoder(code, **kw).decode_arrays(llr, 30, beliefs=True)
    assert r["iters"].max() > 2 and r["conv"].any()
    for threads in (192, 128):
        assert same(r, g.LdpcDecoder(code, threads_per_block=threads, **kw).decode_arrays(llr, 30, beliefs=True))
    codes = [dvb(i) for i in (0, idx, 11, 6)]
    for threads in (0, 192):
        dec = g.LdpcDecoder(codes[0], codes=codes, threads_per_block=threads, **kw)
        w = g.words(code.k())
        m = dec.decode_mixed_arrays(llr.reshape(-1), np.arange(5) * code.n(), np.full(5, 1), np.full(5, 30),
                                    np.arange(5) * w)
        assert np.array_equal(m["msg"].reshape(5, w), r["msg"])
        assert all(np.array_equal(m[k], r[k]) for k in ("iters", "conv", "synd_ok"))


def test_layered_min_sum_batch_of_many_waves(gpu, oracle):
    """More frames than the one-check-per-thread launch holds at once."""
    code, ocode = dvb(2), oracle.Code.dvbt2(0, 2)
    _, _, llr = ocode.channel(3, 0, 3, 2.4)
    o = ocode.decode(llr, 3, sched=1, msg16=True)
    r = g.LdpcDecoder(code, schedule=g.SCHED_LAYERED, msg_dtype=g.MSG_F16).decode_arrays(np.tile(llr, (310, 1)), 3)
    at = np.arange(930) % 3
    assert (r["iters"] == o["iters"][at]).all() and (r["conv"] == o["conv"][at]).all()
    assert (g.unpack_bits(r["msg"], code.k()) == o["msg"][at]).all()


def test_layered_mixed_with_a_qc_code(gpu, oracle):
    rng = np.random.default_rng(2)
    base = [[int(s) if rng.random() < 0.5 else -1 for s in rng.integers(0, 360, 12)] for _ in range(5)]
    qc = g.LdpcCode.from_quasi_cyclic(g.QuasiCyclicLdpc(base, 360))
    codes = [dvb(6), qc]
    kw = dict(algorithm=g.ALGO_SPA_FAST, schedule=g.SCHED_LAYERED, msg_dtype=g.MSG_F16)
    xs = [rng.normal(1.5, 1.5, (2, c.n())).astype(np.float32) for c in codes]
    one = [g.LdpcDecoder(c, **kw).decode_arrays(x, 6) for c, x in zip(codes, xs)]
    offs = np.cumsum([0] + [c.n() for c in codes for _ in range(2)])[:4]
    moffs = np.cumsum([0] + [g.words(c.k()) for c in codes for _ in range(2)])[:4]
    for threads in (0, 192):
        m = g.LdpcDecoder(codes[0], codes=codes, threads_per_block=threads, **kw).decode_mixed_arrays(
            np.concatenate([x.reshape(-1) for x in xs]), offs, np.array([0, 0, 1, 1]), np.full(4, 6), moffs)
        assert np.array_equal(m["iters"], np.concatenate([r["iters"] for r in one]))
        assert np.array_equal(m["msg"], np.concatenate([r["msg"].reshape(-1) for r in one]))
