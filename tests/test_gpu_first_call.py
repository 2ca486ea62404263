"""A decoder's first call: what it sets up then must not disturb a stream capture,
and gives what later calls give."""
import pytest

import gf2_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames", [1, 100, 700])
@pytest.mark.parametrize("algo", [g.ALGO_MINSUM, g.ALGO_SPA])
def test_first_call_under_capture(gpu, algo, frames):
    import torch
    code = g.LdpcCode.dvb_t2_short(0)
    gen = torch.Generator(device=gpu).manual_seed(frames)
    x = torch.randn((frames, code.n()), generator=gen, device=gpu) * 2.0 + 2.0
    ref = g.LdpcDecoder(code, algorithm=algo).decode_tensors(x, 4)
    dec = g.LdpcDecoder(code, algorithm=algo)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = dec.decode_tensors(x, 4)
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(out[k], ref[k]) for k in ref)


def test_small_host_batches_with_and_without_a_pinned_buffer(gpu):
    """More calls than a new decoder waits for its buffer, sizes of both classes in
    turn, decoders that come and go in several threads: always the device call's
    results."""
    import threading

    import numpy as np
    import torch
    code = g.LdpcCode.dvb_t2_short(0)
    rng = np.random.default_rng(1)
    xs = [rng.normal(2.0, 2.0, (f, code.n())).astype(np.float32) for f in (1, 3, 14)]
    dev = g.LdpcDecoder(code)
    ref = [{k: v.cpu().numpy() for k, v in dev.decode_tensors(torch.from_numpy(x).to(gpu), 4).items()} for x in xs]
    wrong = []

    def work(turn):
        for life in range(3):
            dec = g.LdpcDecoder(code)
            for call in range(12):
                i = (turn + life + call // 2) % len(xs)
                r = dec.decode_arrays(xs[i], 4)
                if not all((np.asarray(r[k]).astype(np.int64) == ref[i][k].astype(np.int64)).all() for k in ref[i]):
                    wrong.append((turn, life, call))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
