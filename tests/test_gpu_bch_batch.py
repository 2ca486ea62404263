"""Outer BCH decoding of large batches (bit-sliced syndromes, 32 frames per CTA)
against small batches of the same frames, whose kernel the oracle tests pin:
messages, corrected counts and syndromes are equal bit for bit.  Every code
(14- and 16-bit fields, 12 and 10 factors, lengths that end inside a block of
1024 bits) with a ragged last group, 0..t+3 errors, all-zero and all-one words."""
import pytest

import gf2_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frame,rate", [(f, r) for f in (1, 0) for r in range(6)])
def test_large_batch_equals_small_batches(gpu, frame, rate):
    import torch
    code = g.BchCode.dvb_t2(frame, rate)
    n, k, t = code.n(), code.k(), code.t()
    sms = torch.cuda.get_device_properties(gpu).multi_processor_count
    frames = 2 * 32 * sms * 4 + (1, 17, 31)[rate % 3]  # more groups than CTAs fit at once
    gen = torch.Generator(device=gpu).manual_seed(1000 * frame + rate)
    msg = torch.randint(-2**63, 2**63 - 1, (frames, g.words(k)), generator=gen, device=gpu, dtype=torch.int64)
    if k % 64:
        msg[:, -1] &= (1 << (k % 64)) - 1
    cw = g.BchEncoder(code).encode_words(msg)
    every = torch.arange(frames, device=gpu)
    for e in range(t + 3):
        pos = torch.randint(0, n, (frames,), generator=gen, device=gpu)
        if e == 0:
            pos[: t + 4] = 0
        if e == 1:
            pos[: t + 4] = n - 1
        cw[every, pos // 64] ^= (torch.ones_like(pos) << (pos % 64)) * (every % (t + 4) > e)
    cw[40] = 0
    cw[41] = -1
    cw[frames - 1] = -1
    dec = g.BchDecoder(code)
    big = dec.decode_words(cw, syndromes=True)
    step = 16 * sms
    for a in range(0, frames, step):
        small = dec.decode_words(cw[a:a + step], syndromes=True)
        for key in ("msg", "corrected", "syndromes"):
            assert torch.equal(big[key][a:a + step], small[key]), (key, a)
