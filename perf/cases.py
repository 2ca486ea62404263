"""The work that a user of this framework has it do, as cases that can be timed.

Each case is one call (or, for a Monte Carlo point, one whole point) through
the package's public entry points, with the library's default launch shapes.
The codes are the twelve DVB-T2 LDPC codes and their outer BCH codes, plus one
generic quasi-cyclic code; frames are seeded BPSK / AWGN frames near the codes'
waterfalls, where receivers run.  Eb/N0 of frame f steps through `points`
equally spaced values from `ebn0` to `ebn0 + span` dB.
"""
import math
import os

import numpy as np
import torch

import gf2_b200 as g
from gf2_b200.learned import NmsTrainer
from gf2_b200.montecarlo import simulate_point

RATES = ("1/2", "3/5", "2/3", "3/4", "4/5", "5/6")
# BPSK Shannon limits (dB Eb/N0) near the codes' actual rates, normal and short frames
LIMITS = {"normal": (0.2, 0.7, 1.1, 1.6, 2.0, 2.4), "short": (-0.1, 0.7, 1.1, 1.5, 1.9, 2.2)}
ALGOS = {"minsum": g.ALGO_MINSUM, "spa": g.ALGO_SPA, "spa_fast": g.ALGO_SPA_FAST}
SCHEDULES = {"flooding": g.SCHED_FLOODING, "layered": g.SCHED_LAYERED}
MESSAGES = {"f32": g.MSG_F32, "f16": g.MSG_F16}
WEIGHTS = os.path.join(os.path.dirname(g.__file__), "weights", "nms_layered_normal_%s_T10.npz")


def listed():
    return [
        # A receiver decodes one frame as it arrives: one host frame in, bits out.
        dict(name="one_frame", kind="one", frame="short", rate="1/2", ebn0=2.0, max_iter=50, iters=15),
        # A generic quasi-cyclic code in an iterative receiver: an odd, small
        # batch whose posteriors are read too (soft output).
        dict(name="qc_soft", kind="qc", z=96, cols=24, rows=12, frames=301, ebn0=2.4, max_iter=30, iters=9),
        # Short frames, the reference's decoder and plain sum-product, at low
        # Eb/N0 where nearly every iteration of the budget runs.
        dict(name="short_minsum", kind="decode", frame="short", rate="1/2", algo="minsum", schedule="flooding",
             msg="f32", frames=256, ebn0=1.0, span=0.0, points=1, max_iter=50, iters=49),
        dict(name="short_sumproduct", kind="decode", frame="short", rate="1/2", algo="spa", schedule="flooding",
             msg="f32", frames=256, ebn0=1.0, span=0.0, points=1, max_iter=50, iters=30),
        # Normal frames, the reference's decoder over its waterfall.
        dict(name="normal_minsum", kind="decode", frame="normal", rate="3/5", algo="minsum", schedule="flooding",
             msg="f32", frames=1000, ebn0=1.5, span=0.8, points=9, max_iter=50, iters=30),
        # Layered sum-product with FP16 messages over a sweep from failing to decoding.
        dict(name="normal_sumproduct", kind="decode", frame="normal", rate="3/5", algo="spa_fast", schedule="layered",
             msg="f16", frames=2048, ebn0=0.6, span=0.8, points=9, max_iter=50, iters=39),
        # Serving: the learned decoder, sum-product on the frames that it fails.
        dict(name="learned_fallback", kind="fallback", rate="2/3", frames=16384, ebn0=2.2, span=0.4, points=5,
             iters=8),
        # All twelve codes in one batch, a budget for each frame, one launch.
        dict(name="mixed_codes", kind="mixed", frames=8192, iters=8),
        # A transmitter: systematic encoding of a large batch.
        dict(name="encode", kind="encode", frame="normal", rate="3/5", frames=65536),
        # The step after LDPC decoding: the outer code, 0..t errors per frame.
        dict(name="outer_bch", kind="bch", frame="normal", rate="3/5", frames=65536),
        # Training of the learned decoder: loss and gradients of one batch.
        dict(name="train_gradients", kind="train", rate="2/3", frames=256, ebn0=2.0, span=0.8, points=5),
        # Simulation: frames, channel, decoder and error counters of one point.
        dict(name="monte_carlo", kind="monte_carlo", frame="short", rate="3/4", frames=4096, ebn0=2.6, max_iter=50,
             iters=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another code, batch size and noise level of the ranges above."""
    kind = rng.choice(("one", "qc", "decode", "decode", "decode", "decode", "decode", "fallback", "mixed", "encode",
                       "bch", "train", "monte_carlo"))
    frame, r = rng.choice(("short", "normal")), rng.randrange(6)
    thr, rate = LIMITS[frame][r], RATES[r]
    if kind == "one":
        return dict(kind=kind, frame=frame, rate=rate, ebn0=round(thr + rng.uniform(1.4, 2.2), 2), max_iter=50, iters=15)
    if kind == "qc":
        return dict(kind=kind, z=rng.randrange(24, 129), cols=24, rows=rng.choice((6, 8, 12)),
                    frames=_log_int(rng, 1, 2000), ebn0=round(rng.uniform(2.4, 4.5), 2), max_iter=30, iters=9)
    if kind == "decode":
        algo, schedule, msg = rng.choice((("minsum", "flooding", "f32"), ("minsum", "flooding", "f32"),
                                          ("spa", "flooding", "f32"), ("spa_fast", "layered", "f16"),
                                          ("spa_fast", "layered", "f16"), ("spa_fast", "layered", "f32"),
                                          ("minsum", "layered", "f16"), ("minsum", "layered", "f32")))
        top = 1000 if frame == "normal" and algo != "spa_fast" else 2048
        if algo == "spa":
            top = 256 if frame == "normal" else 1000
        return dict(kind=kind, frame=frame, rate=rate, algo=algo, schedule=schedule, msg=msg,
                    frames=_log_int(rng, 1, top), ebn0=round(thr + rng.uniform(0.6, 1.2), 2),
                    span=round(rng.uniform(0.2, 0.8), 2), points=rng.randrange(1, 10), max_iter=rng.choice((20, 30, 50)),
                    iters=20)
    if kind == "fallback":
        rate = rng.choice(("1/2", "2/3"))
        return dict(kind=kind, rate=rate, frames=_log_int(rng, 16, 12000),
                    ebn0=round((2.2 if rate == "2/3" else 1.9) + rng.uniform(0.0, 0.3), 2), span=0.4, points=5, iters=8)
    if kind == "mixed":
        return dict(kind=kind, frames=_log_int(rng, 24, 8192), iters=8)
    if kind in ("encode", "bch"):
        return dict(kind=kind, frame=frame, rate=rate, frames=_log_int(rng, 1, 65536))
    if kind == "train":
        rate = rng.choice(("1/2", "2/3"))
        return dict(kind=kind, rate=rate, frames=_log_int(rng, 16, 256), ebn0=2.0 if rate == "2/3" else 1.2, span=0.8,
                    points=5)
    return dict(kind=kind, frame=frame, rate=rate, frames=_log_int(rng, 64, 4096 if frame == "short" else 1024),
                ebn0=round(thr + rng.uniform(0.8, 1.4), 2), max_iter=50, iters=12)


def _code(case):
    r = RATES.index(case["rate"])
    return g.LdpcCode.dvb_t2_short(r) if case.get("frame", "normal") == "short" else g.LdpcCode.dvb_t2_normal(r)


def _sigma2(case, rate):
    pts = max(1, case.get("points", 1))
    eb = [case["ebn0"] + (case.get("span", 0.0) * p / (pts - 1) if pts > 1 else 0.0) for p in range(pts)]
    s2 = np.array([g.sigma2_from_ebn0(e, rate) for e in eb])
    return s2[np.arange(case.get("frames", 1)) % pts]


def _frames(case, code, seed, want_cw=False):
    """Seeded frames of the case on the GPU: (codewords, LLRs)."""
    _, cw, llr = g.awgn_frames(code, seed, 0, case.get("frames", 1), _sigma2(case, code.rate()),
                               device=torch.device("cuda"), want_info=False, want_cw=want_cw)
    return cw, llr


def _weights(rate):
    z = np.load(WEIGHTS % rate.replace("/", "_"))
    return z["P"][0].copy(), z["P"][1].copy()


# ---- the generic quasi-cyclic code: three circulants per information block,
# a block staircase for the parity, so that it encodes by accumulation ----
def _qc_base(case):
    rows, cols, z = case["rows"], case["cols"], case["z"]
    rng = np.random.default_rng([rows, cols, z])
    base = [[-1] * cols for _ in range(rows)]
    for c in range(cols - rows):
        for r in rng.permutation(rows)[:3]:
            base[r][c] = int(rng.integers(0, z))
    for r in range(rows):
        base[r][cols - rows + r] = 0
        if r:
            base[r][cols - rows + r - 1] = 0
    return base


def _qc_llr(case, seed):
    """Seeded LLRs of random codewords of the code of _qc_base."""
    rows, cols, z, F = case["rows"], case["cols"], case["z"], case["frames"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kb = cols - rows
    u = torch.randint(0, 2, (F, kb, z), generator=gen, device="cuda")
    base = _qc_base(case)
    par, prev = [], None
    for r in range(rows):
        s = torch.zeros_like(u[:, 0])
        for c in range(kb):
            if base[r][c] >= 0:
                s = s ^ torch.roll(u[:, c], -base[r][c], 1)
        prev = s if prev is None else prev ^ s
        par.append(prev)
    cw = torch.cat([u.reshape(F, -1)] + par, 1)
    s2 = 1.0 / (2.0 * (kb / cols) * 10.0 ** (case["ebn0"] / 10.0))
    y = 1.0 - 2.0 * cw.double() + math.sqrt(s2) * torch.randn(cw.shape, generator=gen, device="cuda", dtype=torch.float64)
    return (2.0 * y / s2).float()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "one":
        code = _code(case)
        _, llr = _frames(case, code, seed)
        return dict(kind=kind, dec=g.LdpcDecoder(code), llr=llr[0].cpu().numpy(), max_iter=case["max_iter"])
    if kind == "qc":
        code = g.LdpcCode.from_quasi_cyclic(g.QuasiCyclicLdpc(_qc_base(case), case["z"]))
        return dict(kind=kind, dec=g.LdpcDecoder(code), llr=_qc_llr(case, seed), max_iter=case["max_iter"])
    if kind == "decode":
        code = _code(case)
        dec = g.LdpcDecoder(code, algorithm=ALGOS[case["algo"]], schedule=SCHEDULES[case["schedule"]],
                            msg_dtype=MESSAGES[case["msg"]])
        _, llr = _frames(case, code, seed)
        return dict(kind=kind, dec=dec, llr=llr, max_iter=case["max_iter"])
    if kind == "fallback":
        code = _code(case)
        a, b = _weights(case["rate"])
        nms = g.LdpcDecoder(code, algorithm=g.ALGO_NMS, schedule=g.SCHED_LAYERED, nms_alpha=a, nms_beta=b,
                            msg_dtype=g.MSG_F16)
        spa = g.LdpcDecoder(code, algorithm=g.ALGO_SPA_FAST, schedule=g.SCHED_LAYERED, msg_dtype=g.MSG_F16)
        _, llr = _frames(case, code, seed)
        return dict(kind=kind, nms=nms, spa=spa, llr=llr)
    if kind == "mixed":
        return _prepare_mixed(case, seed)
    if kind == "encode":
        code = _code(case)
        return dict(kind=kind, enc=g.LdpcEncoder(code), msg=_random_words(case["frames"], code.k(), seed))
    if kind == "bch":
        return _prepare_bch(case, seed)
    if kind == "train":
        code = _code(case)
        a, b = _weights(case["rate"])
        tr = NmsTrainer(code, iterations=a.shape[0], batch=case["frames"], schedule=g.SCHED_LAYERED)
        tr.P[0].copy_(torch.from_numpy(a))
        tr.P[1].copy_(torch.from_numpy(b))
        cw, llr = _frames(case, code, seed, want_cw=True)
        return dict(kind=kind, tr=tr, cw=cw, llr=llr)
    code = _code(case)
    dec = g.LdpcDecoder(code, algorithm=g.ALGO_SPA_FAST, schedule=g.SCHED_LAYERED, msg_dtype=g.MSG_F16)
    return dict(kind=kind, code=code, dec=dec, ebn0=case["ebn0"], max_iter=case["max_iter"], frames=case["frames"],
                seed=seed)


def _random_words(frames, bits, seed):
    """Seeded packed random vectors [frames, ceil(bits / 64)], tail bits zero."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    w = g.words(bits)
    lo = torch.randint(0, 1 << 32, (frames, w), generator=gen, device="cuda")
    hi = torch.randint(0, 1 << 32, (frames, w), generator=gen, device="cuda")
    x = lo | (hi << 32)
    if bits % 64:
        x[:, -1] &= (1 << (bits % 64)) - 1
    return x


def _prepare_bch(case, seed):
    code = g.BchCode.dvb_t2(g.FrameSize.Short if case["frame"] == "short" else g.FrameSize.Normal,
                            RATES.index(case["rate"]))
    F, n, t = case["frames"], code.n(), code.t()
    cw = g.BchEncoder(code).encode_words(_random_words(F, code.k(), seed))
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    f = torch.arange(F, device="cuda")
    for e in range(t):  # frame f carries f mod (t + 1) random bit errors
        at = torch.randint(0, n, (F,), generator=gen, device="cuda")
        bit = torch.where(f % (t + 1) > e, torch.ones_like(at) << (at % 64), torch.zeros_like(at))
        cw[f, at // 64] ^= bit
    return dict(kind="bch", dec=g.BchDecoder(code), cw=cw)


def _prepare_mixed(case, seed):
    codes = [g.LdpcCode.dvb_t2_normal(r) for r in range(6)] + [g.LdpcCode.dvb_t2_short(r) for r in range(6)]
    F, rng, dev = case["frames"], np.random.default_rng(seed), torch.device("cuda")
    thr = LIMITS["normal"] + LIMITS["short"]
    cid = rng.permutation(np.arange(F) % 12)
    budget = rng.integers(10, 51, F).astype(np.int32)
    up = rng.random(F)
    n, wk = np.array([c.n() for c in codes]), np.array([g.words(c.k()) for c in codes])
    off = np.cumsum(n[cid]) - n[cid]
    msg_off = np.cumsum(wk[cid]) - wk[cid]
    llr = torch.empty(int(n[cid].sum()), dtype=torch.float32, device=dev)
    for c, code in enumerate(codes):
        idx = np.nonzero(cid == c)[0]
        if len(idx):
            s2 = np.array([g.sigma2_from_ebn0(thr[c] + 0.8 + up[i], code.rate()) for i in idx])
            _, _, x = g.awgn_frames(code, seed, c << 24, len(idx), s2, device=dev, want_info=False, want_cw=False)
            for j, f in enumerate(idx):
                llr[int(off[f]):int(off[f]) + code.n()] = x[j]
    t = lambda a: torch.from_numpy(a).to(dev)
    dec = g.LdpcDecoder(codes[0], codes=codes, algorithm=g.ALGO_SPA_FAST, schedule=g.SCHED_LAYERED, msg_dtype=g.MSG_F16)
    return dict(kind="mixed", dec=dec, llr=llr, off=t(off.astype(np.int64)), cid=t(cid.astype(np.int32)),
                budget=t(budget), msg_off=t(msg_off.astype(np.int64)),
                out=dict(msg=torch.zeros(int(wk[cid].sum()), dtype=torch.int64, device=dev),
                         iters=torch.zeros(F, dtype=torch.int32, device=dev),
                         conv=torch.zeros(F, dtype=torch.uint8, device=dev),
                         synd_ok=torch.zeros(F, dtype=torch.uint8, device=dev)))


def run(s):
    kind = s["kind"]
    if kind == "one":
        r = s["dec"].decode_iterative(s["llr"], s["max_iter"])
        return dict(bits=r.decoded_bits, iterations=r.iterations, converged=r.converged, synd_ok=r.syndrome_check_passed)
    if kind == "qc":
        return s["dec"].decode_tensors(s["llr"], s["max_iter"], beliefs=True)
    if kind == "decode":
        return s["dec"].decode_tensors(s["llr"], s["max_iter"])
    if kind == "fallback":
        return s["nms"].decode_with_fallback(s["spa"], s["llr"], 10, 50)
    if kind == "mixed":
        o = s["out"]
        s["dec"].decode_mixed_tensors(s["llr"], s["off"], s["cid"], s["budget"], o["msg"], s["msg_off"], o["iters"],
                                      o["conv"], o["synd_ok"])
        return o
    if kind == "encode":
        return s["enc"].encode_packed(s["msg"])
    if kind == "bch":
        return s["dec"].decode_words(s["cw"])
    if kind == "train":
        loss, grads = s["tr"].loss_grad(s["llr"], s["cw"])
        return dict(loss=loss, grads=grads)
    r = simulate_point(s["dec"], s["code"], s["ebn0"], s["max_iter"], batch=s["frames"], max_frames=s["frames"],
                       seed=s["seed"])
    return {k: (np.array(v) if k == "iter_hist" else v) for k, v in r.items() if k not in ("fer_ci", "fer_ref_rule_ci")}


def work(case):
    """Inputs read once, outputs written once; per edge and iteration about ten
    operations for a min-sum message (subtract, compare, select, add) and thirty
    for a sum-product one.  `iters` is the case's usual mean iteration count."""
    kind, F = case["kind"], case.get("frames", 1)
    if kind == "mixed":
        ops = by = 0.0
        for c in [g.LdpcCode.dvb_t2_normal(r) for r in range(6)] + [g.LdpcCode.dvb_t2_short(r) for r in range(6)]:
            by += F / 12 * (4 * c.n() + c.k() / 8 + 30)
            ops += F / 12 * 30 * c.nnz() * case["iters"]
        return {"bytes": by, "flops": ops}
    if kind == "qc":
        n, rows, z = case["cols"] * case["z"], case["rows"], case["z"]
        edges = z * (3 * (case["cols"] - rows) + 2 * rows - 1)
        return {"bytes": F * (8 * n + (n - rows * z) / 8 + 6), "flops": 10.0 * F * edges * case["iters"]}
    if kind == "bch":
        code = g.BchCode.dvb_t2(g.FrameSize.Short if case["frame"] == "short" else g.FrameSize.Normal,
                                RATES.index(case["rate"]))
        return {"bytes": F * ((code.n() + code.k()) / 8 + 4), "flops": F * code.n() * code.t() * 2.0}
    code = _code(case)
    n, k, edges = code.n(), code.k(), code.nnz()
    if kind == "encode":
        return {"bytes": F * (k + n) / 8, "flops": float(F * edges)}
    if kind == "train":
        return {"bytes": F * (4 * n + n / 8) + 16.0 * 10 * code.layers(), "flops": 30.0 * F * edges * 10}
    per = 10.0 if kind in ("one", "fallback") or case.get("algo") == "minsum" else 30.0
    by = k / 8 + 6 + (0 if kind == "monte_carlo" else 4 * n)
    return {"bytes": F * by, "flops": per * F * edges * case["iters"]}


def exact(case, seed):
    """The soft outputs of the generic code's decoder: flooding min-sum in 64
    bits.  Every other case returns bits and counts, or works on the DVB-T2
    tables, which only the package holds."""
    if case["kind"] != "qc":
        return None
    rows, cols, z, F = case["rows"], case["cols"], case["z"], case["frames"]
    base = _qc_base(case)
    deg = max(sum(s >= 0 for s in row) for row in base)
    var = torch.full((rows * z, deg), -1, dtype=torch.long)
    i = torch.arange(z)
    for r in range(rows):
        for d, c in enumerate(c for c in range(cols) if base[r][c] >= 0):
            var[r * z:(r + 1) * z, d] = c * z + (i + base[r][c]) % z
    var = var.cuda()
    real = var >= 0
    at = var.clamp(min=0)
    llr = _qc_llr(case, seed).double()
    belief, msg = llr.clone(), torch.zeros((F,) + var.shape, dtype=torch.float64, device="cuda")
    out, todo = torch.empty_like(llr), torch.arange(F, device="cuda")
    for it in range(case["max_iter"]):
        x = belief[:, at] - msg
        mag = torch.where(real, x.abs(), torch.full_like(x, math.inf))
        neg = real & (x < 0)
        two, where = mag.topk(2, dim=2, largest=False)
        first = torch.zeros_like(real).unsqueeze(0).expand(x.shape).clone().scatter_(2, where[:, :, :1], True)
        m = torch.where(first, two[:, :, 1:], two[:, :, :1])
        sign = neg.sum(2, keepdim=True) % 2 == 1
        msg = torch.where(real, torch.where(sign ^ neg, -m, m), torch.zeros_like(m))
        belief = llr[todo].index_add(1, at.reshape(-1), msg.reshape(len(todo), -1))
        bad = ((real & (belief[:, at] < 0)).sum(2) % 2).any(1)
        done = ~bad if it + 1 < case["max_iter"] else torch.ones_like(bad)
        out[todo[done]] = belief[done]
        todo, belief, msg = todo[~done], belief[~done], msg[~done]
        if not len(todo):
            break
    return dict(beliefs=out, msg=None, iters=None, conv=None, synd_ok=None)
