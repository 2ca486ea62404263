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
