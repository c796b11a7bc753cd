"""The bucket reduction by rows, columns and bits, on both sides of its rule: windows of 8 to 2^19
buckets (odd and even numbers of bits, short top windows, rows cut off by the top window's cap), single
and many windows, mostly empty buckets, and bucket sums that are all equal (additions of equal points at
every step), against the CPU oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scalars(engine, n, kind, seed):
    sc = engine.generate_scalars(seed, n, kind=kind)
    sc[:min(n, 5)] = 255  # above r: the top window's last buckets
    return sc


@pytest.mark.parametrize("n,kind", [(1, 0), (40, 0), (3000, 0), (3000, 1)])
@pytest.mark.parametrize("table", [11, 12, 13, 16, 17, 19, 20, 21])
def test_lines_tables(engine, ocpu, monkeypatch, table, n, kind):
    pts = ocpu.gen_bases(300 + table, n)
    monkeypatch.setenv("MSM_FIXED_BASE", str(table))
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        sc = scalars(engine, n, kind, 301)
        want = ocpu.msm(pts, sc)
        assert np.array_equal(ctx.mult(sc, fixed_base=1)[0], want)
        assert np.array_equal(ctx.mult(sc, fixed_base=1, red_len_log2=3)[0], want), "by runs"
    finally:
        ctx.close()


@pytest.mark.parametrize("signed", [1, 2])
@pytest.mark.parametrize("bits", [4, 5, 9, 12, 13, 14, 16])
def test_lines_windows(engine, ocpu, bits, signed):
    n = 2500
    pts = ocpu.gen_bases(311, n)
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        for kind in (0, 1):
            sc = scalars(engine, n, kind, 312)
            out = ctx.mult(sc, window_bits=bits, signed_digits=signed, fixed_base=2)
            assert np.array_equal(out[0], ocpu.msm(pts, sc)), kind
    finally:
        ctx.close()


@pytest.mark.parametrize("table", [11, 12, 16])
def test_lines_equal_sums(engine, ref, ocpu, monkeypatch, table):
    """One base throughout and scalars 1..n below half a window: every bucket sum is that base."""
    n = (1 << (table - 1)) - 1
    pts = np.repeat(ocpu.gen_bases(321, 1), n, axis=0)
    sc = np.zeros((n, 32), dtype=np.uint8)
    sc[:, :4] = np.arange(1, n + 1, dtype=np.uint32).view(np.uint8).reshape(n, 4)
    sc = sc.view(engine.generate_scalars(1, 1).dtype).reshape((n,) + engine.generate_scalars(1, 1).shape[1:])
    monkeypatch.setenv("MSM_FIXED_BASE", str(table))
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        assert np.array_equal(ctx.mult(sc, fixed_base=1)[0], ocpu.msm(pts, sc))
    finally:
        ctx.close()


def test_lines_several_msms(engine, ocpu):
    """One pass of MSMs on shared bucket arrays and on windows, an empty one among them."""
    pts = ocpu.gen_bases(331, 4000)
    sizes, offs = [4000, 0, 1, 700, 2222], [0, 5, 17, 100, 1000]
    first = np.concatenate([[0], np.cumsum(sizes)])
    sc = scalars(engine, sum(sizes), 1, 332)
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        want = [ocpu.msm(pts[o:o + s], sc[first[j]:first[j] + s]) for j, (s, o) in enumerate(zip(sizes, offs))]
        for opts in (dict(), dict(use_graph=1), dict(window_bits=8, fixed_base=2), dict(window_bits=13, fixed_base=2)):
            out = ctx.mult_uneven(sizes, offs, sc, mode=2, **opts)
            for j in range(len(sizes)):
                assert np.array_equal(out[j], want[j]), (opts, j)
    finally:
        ctx.close()
