"""Fused key switches at N = 2^16 for every digit count 1 .. 8 (k_ks_rows,
keyswitch.cu: the digits' rows together in shared memory up to four, in groups
above), against the oracle: multiplication with and without rescale,
relinearisation of a three-part product, a rotation, and one batch over
levels of different digit counts.

The parameter sets are ~30-bit main primes of the 12-auxiliary bootstrapping
set, regrouped: alpha auxiliary primes (main ones past the twelfth) and L main
primes, in ceil(L / alpha) digits, the last one ragged where alpha does not
divide L."""
import json

import numpy as np
import pytest

import cheddar_b200 as chd
import pyoracle as po
from boot_oracle import lt_evaluate
from test_gpu_column_pass import regrouped

pytestmark = pytest.mark.gpu


def _setup(alpha, L):
    p = regrouped(alpha, L)
    o, g = po.Oracle(p), chd.Context(json.dumps(p))
    return o, g, o.gen_secret(5, 192)


def _eq(ct, ref):
    for x, y in zip(ct.numpy(), ref):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("alpha,L", [(4, 4), (4, 7), (3, 9), (4, 15), (3, 14), (3, 18), (2, 14), (2, 15), (1, 8)])
def test_every_digit_count(cuda_ok, alpha, L):
    o, g, s = _setup(alpha, L)
    mk, rk = o.gen_mult_key(1, s), o.gen_rot_key(2, s, 5)
    gmk, grk = g.evk(*mk), g.evk(*rk)
    ct = lambda seed, lvl: [o.uniform(seed + i, lvl) for i in range(2)]  # noqa: E731
    top = o.max_level
    a, b = ct(10, top), ct(20, top)
    ga, gb = g.import_ct(top, a), g.import_ct(top, b)
    ref = o.hmult(top, a, b, mk, rescale=False)
    _eq(g.HMult(ga, gb, gmk, rescale=False), ref)
    _eq(g.Relinearize(g.Mult(ga, gb), gmk), ref)
    if top > 0:
        _eq(g.HMult(ga, gb, gmk, rescale=True), o.hmult(top, a, b, mk, rescale=True))
    _eq(g.HRot(ga, grk, 5), o.hrot(top, a, rk, 5))
    levels = sorted({top, top // 2, 1, max(1, top - alpha)}) * 2
    pairs = [(ct(100 + 10 * i, x), ct(500 + 10 * i, x)) for i, x in enumerate(levels)]
    out = g.HMultBatch([g.import_ct(x, p[0]) for x, p in zip(levels, pairs)],
                       [g.import_ct(x, p[1]) for x, p in zip(levels, pairs)], gmk, rescale=True)
    for x, p, r in zip(levels, pairs, out):
        _eq(r, o.hmult(x, p[0], p[1], mk, rescale=True))


def test_giant_steps_of_five_digits(cuda_ok):
    # the giant steps' key switches keep every prime and have no P (d0, d1) term
    o, g, s = _setup(3, 14)
    level, scale = o.max_level, o.rescale_prime_prod(o.max_level)
    rng = np.random.default_rng(3)
    diags = {i: 0.3 * (rng.random(o.n // 2) + 0j) for i in range(4)}
    lt = chd.LinearTransform(g, diags, level, scale, 2, 2)
    keys, host = chd.EvkMap(g), {}
    for r in lt.rotations():
        host[r] = o.gen_rot_key(30 + r, s, r)
        keys.set_rotation(r, g.evk(*host[r]))
    a = [o.uniform(40 + i, level) for i in range(2)]
    res = lt.evaluate(g.import_ct(level, a, scale=scale), keys)
    rb, ra = lt_evaluate(o, level, a, scale, lt.plaintexts(), scale, host)[0]
    _eq(res, [rb, ra])
