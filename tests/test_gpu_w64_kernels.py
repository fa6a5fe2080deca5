"""The 64-bit transforms and base conversion (w64_kernels.cu) against their
definitions in Python integers: the forward transform of X and its order,
round trips, and ModUp / ModDown at sampled coefficients, for source counts 1
to 16 on both sides of the conversion's size rule (every prime below 2^58, or
not), with primes just below the line and edge residues.
"""
import json

import numpy as np
import pytest
import torch

import cheddar_b200 as chd

pytestmark = pytest.mark.gpu
N = 1 << 16


def is_prime(n):
    if any(n % p == 0 for p in (3, 5, 7, 11, 13)):
        return False
    d, s = n - 1, 0
    while d % 2 == 0:
        d, s = d // 2, s + 1
    for a in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37):
        x = pow(a, d, n)
        if x in (1, n - 1):
            continue
        for _ in range(s - 1):
            x = x * x % n
            if x == n - 1:
                break
        else:
            return False
    return True


def primes_below(top, count):
    """The `count` largest primes below `top` that are 1 mod 2^17."""
    out, p = [], ((top - 1) >> 17 << 17) + 1
    while len(out) < count:
        if p < top and is_prime(p):
            out.append(p)
        p -= 1 << 17
    return out


def make(alpha, L, main_top, aux_top):
    main = primes_below(main_top, L)
    aux = [p for p in primes_below(aux_top, alpha + L) if p not in main][:alpha]
    p = dict(log_degree=16, log_default_scale=40, default_encryption_level=0,
             level_config=[[i, 0] for i in range(1, L + 1)], main_primes=main, auxiliary_primes=aux,
             terminal_primes=[], additional_base=[1, 0])
    return chd.Context64(json.dumps(p)), main, aux


def residues(primes, seed):
    rng = np.random.default_rng(seed)
    x = np.stack([rng.integers(0, q, N, dtype=np.uint64) for q in primes])
    for row, q in zip(x, primes):
        row[rng.integers(0, N, 300)] = rng.choice(np.array([0, 1, (q - 1) // 2, (q + 1) // 2, q - 1], dtype=np.uint64), 300)
    return x


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()


def host(t):
    torch.cuda.synchronize()
    return t.cpu().numpy().view(np.uint64)


def to_coefficients(g, np_, t, count=1):
    """Plain coefficients of Montgomery-form transforms."""
    t = t.clone()
    torch.cuda.synchronize()
    g.ntt(np_, t, count=count, inverse=True, mont=True)
    g.synchronize()
    return host(t)


def lift(coeffs, primes):
    """sum_k centred(a_k qhat_k^-1 mod q_k) qhat_k for one coefficient: the value the base conversion reduces."""
    Q, y = 1, 0
    for q in primes:
        Q *= q
    for a, q in zip(coeffs, primes):
        v = int(a) * pow(Q // q, -1, q) % q
        y += (v - q if v > q // 2 else v) * (Q // q)
    return y


def test_forward_order_and_round_trip(cuda_ok):
    g, main, aux = make(2, 3, 1 << 50, 1 << 60)
    primes = main + aux
    x = np.zeros((len(primes), N), dtype=np.uint64)
    x[:, 1] = 1  # the polynomial X
    t = dev(x)
    torch.cuda.synchronize()
    g.ntt((3, 0, 2), t)
    g.synchronize()
    y = host(t)
    brev = lambda k: int(f"{k:016b}"[::-1], 2)  # noqa: E731
    for row, q in zip(y, primes):
        psi = int(row[0])
        assert pow(psi, N, q) == q - 1
        for k in [1, 2, 3, 255, 256, 4095, 4096, 30000, N - 1]:
            assert int(row[k]) == pow(psi, 2 * brev(k) + 1, q)
    z = residues(primes, 5)
    t = dev(z)
    torch.cuda.synchronize()
    g.ntt((3, 0, 2), t, mont=True)
    g.ntt((3, 0, 2), t, inverse=True, mont=True)
    g.synchronize()
    assert np.array_equal(host(t), z)


@pytest.mark.parametrize("alpha,L,main_top,aux_top",
                         [(1, 2, 1 << 40, 1 << 41), (3, 5, 1 << 60, 1 << 61), (7, 9, 1 << 50, 1 << 57),
                          (8, 8, 1 << 58, 1 << 58), (9, 10, 1 << 55, 1 << 58), (16, 17, 1 << 45, 1 << 58),
                          (10, 11, 1 << 52, 1 << 59)])
def test_modup_moddown(cuda_ok, alpha, L, main_top, aux_top):
    g, main, aux = make(alpha, L, main_top, aux_top)
    level, all_p = L - 1, main + aux
    beta = -(-L // alpha)
    at = np.unique(np.concatenate([[0, 1, N - 1], np.random.default_rng(alpha).integers(0, N, 150)]))
    x = residues(main, 10 + alpha)
    out = torch.zeros((beta, L + alpha, N), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    g.modup_raw(level, dev(x), out)
    g.synchronize()
    a = to_coefficients(g, (L, 0, 0), dev(x))
    got = to_coefficients(g, (L, 0, alpha), out, count=beta)
    for i in range(beta):
        s, e = i * alpha, min((i + 1) * alpha, L)
        assert np.array_equal(host(out)[i, s:e], x[s:e])
        for n in at:
            y = lift(a[s:e, n], main[s:e])
            for r, p in enumerate(all_p):
                if not s <= r < e:
                    assert int(got[i, r, n]) == y % p
    xa = residues(all_p, 30 + alpha)
    low = torch.zeros((L, N), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    g.moddown_raw(level, chd.CHD_MODDOWN, dev(xa), low)
    g.synchronize()
    a = to_coefficients(g, (L, 0, alpha), dev(xa))
    got = to_coefficients(g, (L, 0, 0), low)
    P = 1
    for p in aux:
        P *= p
    for n in at:
        y = lift(a[L:, n], aux)
        for r, q in enumerate(main):
            assert int(got[r, n]) == (int(a[r, n]) - y) * pow(P, -1, q) % q
