"""Mixed batches of the sum-product decoders against single-code decodes of the
same frames, bit for bit (one arithmetic, whatever the kernel): layered SFU with
FP32 and FP16 messages, DVB-T2 codes alone and with QC codes of other slot
counts, and flooding in both numerics, where a single DVB-T2 code has a kernel of
its own."""
import numpy as np
import pytest

import gf2_b200 as g

pytestmark = pytest.mark.gpu


def dvb(i):
    return g.LdpcCode.dvb_t2_normal(i) if i < 6 else g.LdpcCode.dvb_t2_short(i - 6)


def qc(rows, cols, z, fill):
    rng = np.random.default_rng([rows, cols, z])
    base = [[int(s) if rng.random() < fill else -1 for s in rng.integers(0, z, cols)] for _ in range(rows)]
    return g.LdpcCode.from_quasi_cyclic(g.QuasiCyclicLdpc(base, z))


SETS = {"all DVB-T2": lambda: [dvb(i) for i in range(12)],
        "DVB-T2 and QC": lambda: [dvb(6), dvb(0), dvb(10), qc(5, 24, 360, 0.6)],
        "QC": lambda: [qc(5, 12, 360, 0.5), qc(4, 22, 360, 0.8), qc(6, 30, 384, 0.5)]}


def check(codes, threads, **kw):
    rng = np.random.default_rng(len(codes))
    cid = np.tile(np.arange(len(codes)), 2)
    xs = [rng.normal(1.8, 1.8, codes[c].n()).astype(np.float32) for c in cid]
    off = np.cumsum([0] + [len(x) for x in xs])[:-1]
    moff = np.cumsum([0] + [g.words(codes[c].k()) for c in cid])[:-1]
    m = g.LdpcDecoder(codes[0], codes=codes, threads_per_block=threads, **kw).decode_mixed_arrays(
        np.concatenate(xs), off, cid, np.full(len(cid), 6), moff)
    for f, c in enumerate(cid):
        r = g.LdpcDecoder(codes[c], **kw).decode_arrays(xs[f][None], 6)
        assert m["iters"][f] == r["iters"][0] and m["conv"][f] == r["conv"][0] and m["synd_ok"][f] == r["synd_ok"][0]
        assert np.array_equal(m["msg"][moff[f]:moff[f] + g.words(codes[c].k())], r["msg"][0])


@pytest.mark.parametrize("threads,msg", [(0, g.MSG_F32), (0, g.MSG_F16), (192, g.MSG_F16)])
@pytest.mark.parametrize("codes", SETS)
def test_layered(gpu, codes, threads, msg):
    check(SETS[codes](), threads, algorithm=g.ALGO_SPA_FAST, schedule=g.SCHED_LAYERED, msg_dtype=msg)


@pytest.mark.parametrize("algo", [g.ALGO_SPA, g.ALGO_SPA_FAST])
def test_flooding(gpu, algo):
    check(SETS["all DVB-T2"](), 0, algorithm=algo)
