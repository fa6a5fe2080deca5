"""The stages of a bootstrap at its full size (N = 2^16, alpha = 12, four
digits), where every key switch takes the fused pipeline, bit for bit against
the oracle running the same compiled program: EvalMod (every level of its
multiplications, rescales and constant accumulations) and a linear transform
from the top level (hoisted baby steps, giant steps, plaintext accumulation,
merged ModDown and rescale), with uniform random ciphertexts and keys.  The
whole program is compared with the oracle at N = 2^12
(tests/test_gpu_bootstrap.py); at N = 2^16 that takes the oracle minutes."""
import functools

import numpy as np
import pytest

import cheddar_b200 as chd
from boot_oracle import Ct, lt_evaluate, run_program
from gpu_common import pair

pytestmark = pytest.mark.gpu
BOOT = "boot_l34_a12.json"


@functools.lru_cache(maxsize=None)
def _key():
    o, g = pair(BOOT)
    rng = np.random.default_rng(8)
    one = lambda: np.stack([np.stack([rng.integers(0, int(q), o.n, dtype=np.uint32) for q in o.all_primes()])  # noqa: E731
                            for _ in range(-(-o.L // o.alpha))])
    host = (one(), one())
    return host, g.evk(*host)


def _eq(ct, ref):
    for x, y in zip(ct.numpy(), ref):
        assert np.array_equal(x, y)


def test_evalmod(cuda_ok):
    o, g = pair(BOOT)
    host, key = _key()
    level = 30
    prog = chd.Program.evalmod(g, level, chd.boot_mod_coefficients(), num_double_angle=3, initial_K=2)
    keys = chd.EvkMap(g)
    keys.set_mult(key)
    a = [o.uniform(50 + i, level) for i in range(2)]
    res = prog.run(g.import_ct(level, a, prog.start_scale), keys)
    ref = run_program(o, prog.json(), Ct(level, a, prog.start_scale), mult_key=host)
    assert ref.level == level - 8
    _eq(res, ref.parts)


def test_linear_transform(cuda_ok):
    o, g = pair(BOOT)
    host, key = _key()
    level = o.max_level
    scale = o.rescale_prime_prod(level)
    rng = np.random.default_rng(9)
    diags = {i: 0.3 * (rng.random(o.n // 2) + 1j * rng.random(o.n // 2)) for i in range(8)}
    lt = chd.LinearTransform(g, diags, level, scale, 4, 2)
    keys = chd.EvkMap(g)
    for r in lt.rotations():
        keys.set_rotation(r, key)
    a = [o.uniform(60 + i, level) for i in range(2)]
    res = lt.evaluate(g.import_ct(level, a, scale), keys)
    _eq(res, lt_evaluate(o, level, a, scale, lt.plaintexts(), scale, {r: host for r in lt.rotations()})[0])
