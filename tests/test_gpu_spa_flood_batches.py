"""Flooding sum-product of the short codes with more than 11 slots per check at the
batch size where one CTA per frame takes over from teams: the frames decode as they
do a few at a time."""
import numpy as np
import pytest

import gf2_b200 as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", [g.ALGO_SPA, g.ALGO_SPA_FAST])
@pytest.mark.parametrize("rate", [3, 4, 5])
def test_one_cta_per_frame_equals_teams(gpu, rate, algo):
    import torch
    code = g.LdpcCode.dvb_t2_short(rate)
    sms = torch.cuda.get_device_properties(gpu).multi_processor_count
    _, _, llr = g.awgn_frames(code, 9, 0, 3, g.sigma2_from_ebn0(2.4 + 0.3 * (rate - 3), code.rate()))
    dec = g.LdpcDecoder(code, algorithm=algo)
    few = dec.decode_arrays(llr, 8, beliefs=True)
    for frames in (sms - 1, sms, 2 * sms + 5):
        at = np.arange(frames) % 3
        many = dec.decode_arrays(llr[at], 8, beliefs=True)
        assert all(np.array_equal(many[k], few[k][at]) for k in few)
