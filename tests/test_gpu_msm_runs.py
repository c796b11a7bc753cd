"""The runs that a pass of few entries is split into: enough of them where a few buckets hold most of the
entries (narrow tables, narrow windows), against the CPU oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("table,bits,n", [(11, 0, 20011), (12, 0, 39000), (13, 0, 9001), (0, 4, 8192), (0, 6, 13001)])
def test_runs_of_few_buckets(engine, ocpu, monkeypatch, table, bits, n, kind):
    pts = ocpu.gen_bases(500 + table + bits, n)
    sc = engine.generate_scalars(501, n, kind=kind, msm_index=2)
    monkeypatch.setenv("MSM_FIXED_BASE", str(table))
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        opts = dict(fixed_base=1) if table else dict(fixed_base=2, window_bits=bits)
        assert np.array_equal(ctx.mult(sc, **opts)[0], ocpu.msm(pts, sc))
        st = ctx.last_pass_stats()
    finally:
        ctx.close()
    assert st["entries"] <= 7 << 17  # four lanes a run
    assert st["tasks"] >= min(st["entries"] // 64, 7000)


@pytest.mark.parametrize("bits", [6, 13])
def test_windowed_against_the_oracle(engine, ocpu, bits):
    """A windowed pass on quads, with scalars of zero and at or above r, of which 253 bits are used."""
    n = 4099
    pts = ocpu.gen_bases(511, n)
    sc = engine.generate_scalars(512, n, kind=1, msm_index=1)
    sc[5] = 0
    sc[7] = np.uint64(2**64 - 1)
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        out = ctx.mult(sc, window_bits=bits, fixed_base=2)
    finally:
        ctx.close()
    masked = sc.copy()
    masked[:, 3] &= np.uint64(2**61 - 1)
    assert np.array_equal(out[0], ocpu.msm(pts, masked))


@pytest.mark.parametrize("bits,msms", [(4, 18), (5, 17), (6, 13), (6, 14), (7, 16), (8, 9), (8, 10)])
def test_reduction_of_many_small_windows(engine, ocpu, bits, msms):
    """Passes of up to 2^16 buckets on both sides of the limit on pieces of lines."""
    n = 60
    pts = ocpu.gen_bases(521, n)
    sc = engine.generate_scalars(522, n * msms, kind=1)
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        out = ctx.mult(sc, window_bits=bits, fixed_base=2, mode=2)
    finally:
        ctx.close()
    for j in range(0, msms, 4):
        assert np.array_equal(out[j], ocpu.msm(pts, sc[j * n:(j + 1) * n])), j
