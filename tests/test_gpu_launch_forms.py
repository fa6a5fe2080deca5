"""The forms that a launch takes by its size at N = 2^16 give the same words:
raw transforms on both sides of one or two limbs per CTA and of 64 limbs
(the smaller launch descriptor), ModDown on both sides of 8 and of 64
column-pass jobs, against the same calls on one polynomial at a time, which
the oracle tests cover."""
import pytest
import torch

import cheddar_b200 as chd
from gpu_common import pair

pytestmark = pytest.mark.gpu
KS = "keyswitch_l24_a8.json"


def uniform(g, shape, gidx, seed):
    primes = torch.tensor(all_primes(), device="cuda")[torch.tensor(list(gidx), device="cuda")][:, None]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.randint(0, 2 ** 62, (*shape, len(gidx), g.n), generator=gen, device="cuda") % primes
    torch.cuda.synchronize()
    return r.to(torch.int32)


def all_primes():
    o, _ = pair(KS)
    return [int(q) for q in o.all_primes()]


@pytest.mark.parametrize("primes,count", [(1, 2), (24, 4), (24, 5), (24, 6), (24, 7), (24, 17), (1, 63), (1, 64), (1, 65),
                                          (1, 120), (1, 121), (2, 61)])
def test_raw_transforms(cuda_ok, primes, count):
    _, g = pair(KS)
    x = uniform(g, (count,), g.gidx(primes, 0, 0), 100 * primes + count)
    for call in (g.ntt_raw, g.intt_raw):
        batch, single = x.clone(), x.clone()
        torch.cuda.synchronize()
        call(primes, 0, 0, batch, mont=True, count=count)
        for i in range(count):
            call(primes, 0, 0, single[i], mont=True)
        g.synchronize()
        torch.cuda.synchronize()
        assert torch.equal(batch, single)


@pytest.mark.parametrize("level,npoly", [(3, 7), (3, 8), (3, 9), (3, 16), (3, 17), (3, 18), (1, 127), (1, 128), (1, 130)])
def test_moddown(cuda_ok, level, npoly):
    _, g = pair(KS)
    x = uniform(g, (npoly,), g.gidx(*g.level_np(level), g.alpha), npoly)
    batch = torch.zeros((npoly, g.num_q(level), g.n), dtype=torch.int32, device="cuda")
    single = torch.zeros_like(batch)
    torch.cuda.synchronize()
    g.moddown_raw(level, chd.CHD_MODDOWN, x, batch, npoly=npoly)
    for i in range(npoly):
        g.moddown_raw(level, chd.CHD_MODDOWN, x[i], single[i])
    g.synchronize()
    assert torch.equal(batch, single)
