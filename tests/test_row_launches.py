"""Which launches of raw transforms take two limbs of one prime per CTA, read
from the row kernels' grids (one row of 16 per x, a limb or a pair per y) on
the stand-in for the CUDA runtime, for a GPU of 148 SMs.  Pairs are taken
where the launches that share the GPU fill two waves of them, 888 CTAs."""
import pytest

from cudart_stand_in import runtime  # noqa: F401


@pytest.mark.parametrize("primes,count,groups", [
    (24, 1, [24]),               # one polynomial: nothing to pair
    (24, 4, [96]),               # 48 pairs, 768 CTAs of one launch
    (20, 5, [60]),               # 40 pairs and 20 single limbs, 960 CTAs
    (24, 5, [72]),
    (24, 6, [36] * 2),           # launches that alternate between two streams, 1152 CTAs of two of them
    (24, 16, [48] * 4),
    (24, 32, [55] * 6 + [54]),
    (1, 121, [31, 30]),          # 62 and 59 limbs
])
def test_pairs_of_limbs(runtime, primes, count, groups):  # noqa: F811
    runtime(f"""
        ctx = chd.Context(chd.load_params("ntt_bootparam30_p24.json"))
        buf = np.zeros(1, np.uint32)
        for call in (ctx.ntt_raw, ctx.intt_raw):
            rt.fake_reset(-1)
            call({primes}, 0, 0, buf.ctypes.data, count={count})
            grids = [[rt.fake_grid(i, k) for k in range(3)] for i in range(rt.fake_launches())]
            rows = [y for x, y, threads in grids if (x, threads) == (16, 256)]
            assert rows == {groups}, rows
    """)
