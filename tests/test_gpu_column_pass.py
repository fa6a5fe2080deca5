"""The fused column pass (modswitch.cu) at every source count 1 .. 16 and at
target counts around the groups of four that a warp converts together: raw
ModUp (digits of alpha sources, a ragged last one) and ModDown (alpha
sources), bit for bit against the oracle, on residues at the edges of the
centred range as well as uniform ones.

The parameter sets are the 31-bit auxiliary and ~30-bit main primes of the
12-auxiliary bootstrapping set, regrouped: alpha auxiliary primes (main ones
past the twelfth) and L = alpha + extra main primes at N = 2^16."""
import json

import numpy as np
import pytest
import torch

import cheddar_b200 as chd
import pyoracle as po
from gpu_common import param_json

pytestmark = pytest.mark.gpu


def regrouped(alpha, L):
    p = param_json("boot_l34_a12.json")
    main = [q for q in p["main_primes"] if q > 1 << 28]
    pool = p["auxiliary_primes"] + main[L:]
    return dict(log_degree=16, log_default_scale=p["log_default_scale"], default_encryption_level=0,
                level_config=[[i, 0] for i in range(1, L + 1)], main_primes=main[:L], auxiliary_primes=pool[:alpha],
                terminal_primes=[], additional_base=[1, 0])


def edges(o, level, seed, num_aux=0):
    """Uniform residues with 0, 1, (q - 1) / 2, (q + 1) / 2 and q - 1 sprinkled in."""
    x = o.uniform(seed, level, num_aux=num_aux)
    primes = o.all_primes()
    rows = list(range(o.num_q(level))) + [o.L + i for i in range(num_aux)]
    rng = np.random.default_rng(seed)
    for r, g in enumerate(rows):
        q = int(primes[g])
        at = rng.integers(0, o.n, 500)
        x[r, at] = rng.choice([0, 1, (q - 1) // 2, (q + 1) // 2, q - 1], 500)
    return x


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()


def _host(t):
    torch.cuda.synchronize()
    return t.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("alpha,extra", [(1, 1), (2, 3), (3, 2), (4, 5), (5, 1), (6, 7), (7, 4), (8, 0), (9, 3), (10, 9),
                                         (11, 2), (12, 13), (13, 5), (14, 1), (15, 6), (16, 4)])
def test_every_source_count(cuda_ok, alpha, extra):
    p = regrouped(alpha, alpha + extra)
    o, g = po.Oracle(p), chd.Context(json.dumps(p))
    level = o.max_level
    x = edges(o, level, 10 * alpha)
    mu = torch.zeros((o.beta(level), o.num_q(level) + alpha, o.n), dtype=torch.int32, device="cuda")
    g.modup_raw(level, _dev(x), mu)
    g.synchronize()
    ref = o.modup(level, x)
    assert np.array_equal(_host(mu).reshape(ref.shape), ref)
    xa = edges(o, level, 10 * alpha + 1, num_aux=alpha)
    out = torch.zeros((o.num_q(level), o.n), dtype=torch.int32, device="cuda")
    g.moddown_raw(level, chd.CHD_MODDOWN, _dev(xa), out)
    g.synchronize()
    assert np.array_equal(_host(out), o.moddown(level, xa))
