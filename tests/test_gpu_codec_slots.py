"""Encoder and decoder at slot counts on both sides of what one CTA of the
special transforms holds (1024), bit for bit against the oracle, whose
transforms run one stage after another."""
import numpy as np
import pytest
import torch

from gpu_common import pair

pytestmark = pytest.mark.gpu
KS = "keyswitch_l24_a8.json"


@pytest.mark.parametrize("slots", [1, 2, 8, 512, 1024, 2048, 4096, 16384, 32768])
def test_encode_decode(cuda_ok, slots):
    o, g = pair(KS)
    rng = np.random.default_rng(slots)
    msg = rng.normal(size=slots) + 1j * rng.normal(size=slots)
    level, scale = 3, 2.0 ** 40
    pt = g.encode(level, scale, msg)
    torch.cuda.synchronize()
    ref = o.encode(level, scale, msg)
    assert np.array_equal(pt.cpu().numpy().view(np.uint32), ref)
    got, want = g.decode(level, scale, pt, slots), o.decode(level, scale, ref, slots)
    assert np.array_equal(got, want)
