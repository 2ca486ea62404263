"""GPU parity tests of the check-state flooding kernel's structured passes: the
unrolled slot counts (regular and irregular codes, a code with more distinct
slot counts than unrolled bodies), odd circulant sizes, clusters of CTAs per
frame (few frames), one CTA per frame and small CTAs (many frames of a small
code).  The arithmetic is the oracle's operation for operation, so iterations,
flags, decisions and posteriors are equal (posteriors as numbers: the sign of a
zero is free)."""
import numpy as np
import pytest

import gf2_b200 as g

pytestmark = pytest.mark.gpu


def qc_base(rows, cols, z, keep, seed):
    rng = np.random.default_rng(seed)
    return [[int(s) if rng.random() < k else -1 for s in rng.integers(0, z, cols)]
            for k in np.linspace(keep[0], keep[1], rows)]


def make(oracle, spec):
    if spec[0] == "qc":
        base = qc_base(*spec[1:])
        z = spec[3]
        return g.LdpcCode.from_quasi_cyclic(g.QuasiCyclicLdpc(base, z)), oracle.Code.qc(base, z)
    fs, r = spec
    return (g.LdpcCode.dvb_t2_short(r) if fs else g.LdpcCode.dvb_t2_normal(r)), oracle.Code.dvbt2(fs, r)


def llrs(n, frames, seed, special):
    rng = np.random.default_rng(seed)
    x = rng.normal(1.6, 1.6, (frames, n)).astype(np.float32)
    if special:
        for f in range(frames):
            at = rng.choice(n, 30, replace=False)
            x[f, at[:6]] = np.inf
            x[f, at[6:12]] = -np.inf
            x[f, at[12:18]] = 0.0
            x[f, at[18:24]] = -0.0
            if f % 2:
                x[f, at[24:]] = np.nan
    return x


@pytest.mark.parametrize("spec,frames", [
    ((1, 0), 1), ((1, 0), 40), ((1, 0), 150),           # irregular 4..7 slots; teams of 16 and 2, one CTA
    ((1, 3), 9), ((1, 5), 3), ((0, 5), 2), ((0, 0), 18),  # 9..13, 16..19, 22 and 7 slots; teams of 8 and 16
    (("qc", 6, 40, 33, (0.2, 0.95), 3), 5),             # odd circulants, more slot counts than bodies
    (("qc", 4, 12, 1, (0.6, 0.9), 4), 3),               # circulants of one bit
    (("qc", 12, 24, 96, (0.3, 0.45), 5), 700),          # 256-thread CTAs, several frames per SM
    (("qc", 12, 24, 31, (0.3, 0.45), 6), 301),          # 512-thread CTAs
])
@pytest.mark.parametrize("special", [False, True])
def test_structured_flooding_minsum_equals_oracle(gpu, oracle, spec, frames, special):
    code, ocode = make(oracle, spec)
    distinct = min(frames, 4)
    x = llrs(code.n(), distinct, 7, special and code.n() >= 100)
    r = g.LdpcDecoder(code).decode_arrays(np.tile(x, (-(-frames // distinct), 1))[:frames], 6, beliefs=True)
    o = ocode.decode(x, 6)
    for f in range(frames):
        i = f % distinct
        assert r["iters"][f] == o["iters"][i] and r["conv"][f] == o["conv"][i] and r["synd_ok"][f] == o["synd_ok"][i]
    assert (g.unpack_bits(r["msg"], code.k()) == o["msg"][np.arange(frames) % distinct]).all()
    assert np.array_equal(r["beliefs"], o["beliefs"][np.arange(frames) % distinct], equal_nan=True)


@pytest.mark.parametrize("frames", [1, 160])
def test_structured_flooding_nms_fp16_equals_oracle(gpu, oracle, frames):
    code, ocode = make(oracle, (1, 4))
    rng = np.random.default_rng(3)
    a = (0.6 + 0.4 * rng.random((3, code.layers()))).astype(np.float32)
    b = (0.3 * rng.random((3, code.layers()))).astype(np.float32)
    x = llrs(code.n(), 1, 9, True)
    r = g.LdpcDecoder(code, algorithm=g.ALGO_NMS, nms_alpha=a, nms_beta=b,
                      msg_dtype=g.MSG_F16).decode_arrays(np.repeat(x, frames, 0), 5, beliefs=True)
    o = ocode.decode(x, 5, algo=3, msg16=True, alpha=a, beta=b)
    assert (r["iters"] == o["iters"][0]).all() and (r["conv"] == o["conv"][0]).all()
    assert (g.unpack_bits(r["msg"], code.k()) == o["msg"]).all()
    assert np.array_equal(r["beliefs"], np.repeat(o["beliefs"], frames, 0), equal_nan=True)


def test_noalloc_takes_a_code_just_inside_its_scratch(gpu):
    """A QC code whose structured tables (43 KB and more) are too large for shared
    memory and would exceed the 64 MiB scratch, of which the rest of it leaves 30 KB:
    it is decoded without them, bit for bit like the allocating entry point."""
    import ctypes

    import torch
    from gf2_b200 import _capi as C
    mb, nb, Z, dc = 500, 1000, 914, 10
    base = np.full((mb, nb), -1, np.int32)
    for r in range(mb):
        for i in range(dc):
            c = r if i == 0 else mb + r if i == 1 else (r * 5 + i * 3) % nb
            base[r, c] = (r * 37 + c * 11) % Z
    code = g.LdpcCode._create(C.lib.gf2c_code_create_qc, base.ctypes.data_as(ctypes.c_void_p), mb, nb, Z)
    gen = torch.Generator(device=gpu).manual_seed(3)
    llr = torch.randn((1, code.n()), generator=gen, device=gpu) + 1.0
    ref = g.LdpcDecoder(code).decode_tensors(llr, 2)
    msg = torch.zeros((1, g.words(code.k())), dtype=torch.int64, device=gpu)
    it = torch.zeros(1, dtype=torch.int32, device=gpu)
    cv, so = (torch.zeros(1, dtype=torch.uint8, device=gpu) for _ in range(2))
    C.check(C.lib.gf2c_decode_batch_noalloc(code.handle, ctypes.c_void_p(llr.data_ptr()), 1, 2,
                                            *(ctypes.c_void_p(t.data_ptr()) for t in (msg, it, cv, so)), None))
    torch.cuda.synchronize()
    assert torch.equal(msg, ref["msg"]) and torch.equal(it, ref["iters"]) and torch.equal(cv, ref["conv"])
