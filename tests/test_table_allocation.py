"""Device memory that runs out while a context builds its constant tables.

Runs without a GPU, on the stand-in for the CUDA runtime, which refuses the
n-th allocation.  A context must be refused whichever allocation fails, never
come up with a table missing, and give back what it had taken; whatever is
refused must also leave the next call, with memory again, intact.
"""
from cudart_stand_in import runtime  # noqa: F401


def test_context_is_refused_whichever_allocation_fails(runtime):  # noqa: F811
    # three primes of digits 1 wide: every table kind of N = 2^16 and of a
    # smaller degree, over three levels and a rescale
    runtime("""
        p = json.load(open(os.path.join(chd.PARAM_DIR, "keyswitch_l8_a3.json")))
        p.update(main_primes=p["main_primes"][:3], auxiliary_primes=p["auxiliary_primes"][:1],
                 level_config=[[i, 0] for i in range(1, 4)], default_encryption_level=0)
        for log_n in (16, 12):
            text = json.dumps(dict(p, log_degree=log_n))
            rt.fake_reset(-1)
            ctx = chd.Context(text)
            total = rt.fake_mallocs()
            assert total >= 15 and rt.fake_live() == total
            ctx.close()
            assert rt.fake_live() == 0
            for n in range(total):
                rt.fake_reset(n)
                err, ctx = refused(lambda: chd.Context(text))
                assert err and "allocation" in err, (log_n, n, err)
                assert rt.fake_live() == 0 and rt.fake_last() == 0, (log_n, n)
    """)


def test_level_constants_of_the_64_bit_path(runtime):  # noqa: F811
    # built on first use: ModUp and ModDown + Rescale fail with the
    # allocation, launch nothing, and work once there is memory
    runtime("""
        p = json.load(open(os.path.join(chd.PARAM_DIR, "bootparam_40_64bit.json")))
        p.update(main_primes=p["main_primes"][:3], auxiliary_primes=p["auxiliary_primes"][:2],
                 level_config=[[i, 0] for i in range(1, 4)], default_encryption_level=0)
        src, ext = np.zeros((5, 65536), np.uint64), np.zeros((2, 5, 65536), np.uint64)
        calls = [lambda c: c.modup_raw(2, src.ctypes.data, ext.ctypes.data),
                 lambda c: c.moddown_raw(2, chd.CHD_MODDOWN_RESCALE, src.ctypes.data, ext.ctypes.data)]
        for call in calls:
            total = 1
            n = -1
            while n < total:
                rt.fake_reset(-1)
                ctx = chd.Context64(json.dumps(p))
                rt.fake_reset(n)
                err, _ = refused(lambda: call(ctx))
                if n < 0:
                    total = rt.fake_mallocs()
                    assert total >= 5 and err is None
                elif n < total:
                    assert err and "failed" in err and rt.fake_launches() == 0, (n, err)
                    rt.fake_reset(-1)
                    call(ctx)
                assert rt.fake_launches() > 0 and rt.fake_early() == 0
                del ctx
                n += 1
    """)


def test_level_constants_of_the_64_bit_path_during_a_capture(runtime):  # noqa: F811
    # a level's first use may be recorded into a graph: its tables are
    # uploaded then and there, not by the graph
    runtime("""
        p = json.load(open(os.path.join(chd.PARAM_DIR, "bootparam_40_64bit.json")))
        p.update(main_primes=p["main_primes"][:3], auxiliary_primes=p["auxiliary_primes"][:2],
                 level_config=[[i, 0] for i in range(1, 4)], default_encryption_level=0)
        src, ext = np.zeros((5, 65536), np.uint64), np.zeros((2, 5, 65536), np.uint64)
        ctx = chd.Context64(json.dumps(p))
        stream = C.create_string_buffer(8)
        ctx.set_stream(C.addressof(stream))
        rt.fake_reset(-1)
        rt.fake_capture(C.addressof(stream))
        ctx.modup_raw(2, src.ctypes.data, ext.ctypes.data)
        assert rt.fake_launches() > 0 and rt.fake_early() == 0
        rt.fake_capture(None)
    """)


def test_tables_of_the_encoder(runtime):  # noqa: F811
    # built on first use; a call that had memory for one of the two tables
    # only must not leave the next one without the other
    runtime("""
        p = json.load(open(os.path.join(chd.PARAM_DIR, "keyswitch_l8_a3.json")))
        p.update(log_degree=12)
        re, im, pt, slots = np.ones(4), np.zeros(4), np.zeros((8, 4096), np.uint32), C.c_int()

        def encode(ctx):
            chd._check(chd.lib().chd_encode(ctx.ptr, 2, 2.0 ** 30, re.ctypes.data, im.ctypes.data, 4, 0, pt.ctypes.data,
                                            C.byref(slots)))

        total, n = 1, -1
        while n < total:
            rt.fake_reset(-1)
            ctx = chd.Context(json.dumps(p))
            rt.fake_reset(n)
            err, _ = refused(lambda: encode(ctx))
            if n < 0:
                total, held = rt.fake_mallocs(), rt.fake_live()
                assert total >= 3 and err is None
            elif n < total:
                assert err and "failed" in err and rt.fake_launches() == 0, (n, err)
                rt.fake_reset(-1)
                encode(ctx)
            assert rt.fake_launches() > 0 and rt.fake_early() == 0 and rt.fake_live() == held, n
            ctx.close()
            n += 1
    """)


def test_64_bit_modup_refuses_digits_of_more_than_16_primes(runtime):  # noqa: F811
    # as the 32-bit path does; the conversion holds 16 sources
    runtime("""
        p = json.load(open(os.path.join(chd.PARAM_DIR, "bootparam_40.json")))
        q = p["main_primes"]
        buf = np.zeros((2, 40, 65536), np.uint64)
        for alpha, fits in ((16, True), (17, False)):
            spec = dict(p, log_degree=16, main_primes=q[:alpha + 1], auxiliary_primes=q[20:20 + alpha], terminal_primes=[],
                        level_config=[[alpha, 0], [alpha + 1, 0]], default_encryption_level=0, additional_base=[1, 0])
            ctx = chd.Context64(json.dumps(spec))
            rt.fake_reset(-1)
            err, _ = refused(lambda: ctx.modup_raw(1, buf[0].ctypes.data, buf.ctypes.data))
            assert (err is None) == fits and (rt.fake_launches() > 0) == fits, (alpha, err)
    """)
