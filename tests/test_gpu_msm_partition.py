"""The partitioned sort of large passes, asked for at small sizes: every form of digits it has a loop
for (and the general one), chunks cut short and shared by several MSMs, key ranges of many parts
(repeated scalars, a narrow top window), split top digits and bases without an entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(ctx, ocpu, pts, sizes, offs, sc, **opts):
    first = np.concatenate([[0], np.cumsum(sizes)])
    out = ctx.mult_uneven(sizes, offs, sc, **opts)
    for j, (s, o) in enumerate(zip(sizes, offs)):
        assert np.array_equal(out[j], ocpu.msm(pts[o:o + s], sc[first[j]:first[j] + s])), (opts, j)


@pytest.mark.parametrize("table", [11, 16, 20, 21, 22, 23, 24])
def test_partition_tables(engine, ocpu, monkeypatch, table):
    n = 5003
    pts = ocpu.gen_bases(61 + table, n)
    monkeypatch.setenv("MSM_FIXED_BASE", str(table))
    ctx = engine.multi_scalar_mult_init(pts)
    monkeypatch.setenv("MSM_SORT_PARTITION", "1")
    try:
        sc = engine.generate_scalars(62, n)
        sc[:40] = 255  # 253 bits set: digits above the top window's buckets
        check(ctx, ocpu, pts, [n], [0], sc, fixed_base=1)
        check(ctx, ocpu, pts, [n], [0], engine.generate_scalars(63, n, kind=1), fixed_base=1, use_graph=1)
    finally:
        ctx.close()


@pytest.mark.parametrize("signed", [1, 2])
@pytest.mark.parametrize("bits", [4, 9, 14, 15, 17, 18, 19, 21])
def test_partition_windows(engine, ocpu, monkeypatch, bits, signed):
    n = 3001
    pts = ocpu.gen_bases(71, n)
    monkeypatch.setenv("MSM_SORT_PARTITION", "1")
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        sc = engine.generate_scalars(72, n, kind=1)
        sc[:40] = 255
        check(ctx, ocpu, pts, [n], [0], sc, window_bits=bits, signed_digits=signed, fixed_base=2)
    finally:
        ctx.close()


@pytest.mark.parametrize("mode", [1, 2])
def test_partition_several_msms(engine, ocpu, monkeypatch, mode):
    """Chunks of 1024 points that hold the ends of several MSMs, an empty one among them; mode 1 uploads
    in pieces of whole chunks."""
    nb = 1 << 13
    pts = ocpu.gen_bases(81, nb)
    sizes, offs = [1, 1023, 0, 1025, 5000, 2, nb], [5, 0, 3, 17, 3000, 100, 0]
    monkeypatch.setenv("MSM_SORT_PARTITION", "1")
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        for opts in (dict(), dict(use_graph=1), dict(fixed_base=2), dict(window_bits=12)):
            check(ctx, ocpu, pts, sizes, offs, engine.generate_scalars(82, sum(sizes), kind=1), mode=mode, **opts)
    finally:
        ctx.close()


@pytest.mark.parametrize("n", [1, 1024, 16385, 1 << 18])
def test_partition_equal_scalars(engine, ocpu, monkeypatch, n):
    """Every window's entries in one bucket: the warp's shared atomic, and a key range of 16 parts."""
    pts = ocpu.gen_bases(91, n)
    monkeypatch.setenv("MSM_SORT_PARTITION", "1")
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        check(ctx, ocpu, pts, [n], [0], np.repeat(engine.generate_scalars(92, 1), n, axis=0))
    finally:
        ctx.close()


def test_partition_by_size(engine, ocpu):
    """The default rule on a pass above its line (2^17 + 3 points on tables of width 16)."""
    n = (1 << 17) + 3
    pts = ocpu.gen_bases(95, n)
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        check(ctx, ocpu, pts, [n, n], [0, 0], engine.generate_scalars(96, 2 * n), mode=1)
    finally:
        ctx.close()


def test_partition_two_threads(engine, ocpu, monkeypatch):
    """Two contexts whose partitions need different amounts of shared memory, from two threads at once."""
    import threading
    monkeypatch.setenv("MSM_SORT_PARTITION", "1")
    n, res = 4000, {}
    pts, sc = ocpu.gen_bases(97, n), engine.generate_scalars(98, n)
    want = ocpu.msm(pts, sc)
    ctxs = [engine.multi_scalar_mult_init(pts) for _ in range(2)]

    def work(j):
        opts = dict(window_bits=4, fixed_base=2) if j else dict(fixed_base=1)
        res[j] = all(np.array_equal(ctxs[j].mult(sc, **opts)[0], want) for _ in range(200 if j == 0 else 40))

    try:
        threads = [threading.Thread(target=work, args=(j,)) for j in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert res == {0: True, 1: True}
    finally:
        for c in ctxs:
            c.close()
