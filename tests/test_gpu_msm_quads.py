"""MSMs whose runs, split buckets and level-1 reduction are summed by four lanes each, and their
neighbours on the other side of each rule, against the CPU oracle, byte for byte: the smallest sizes,
both sides of the entry limit (7 * 2^17 entries at 17 per point on width-16 tables), both sides of the
limit on level-1 runs (tables of width 18 and 19), mostly empty buckets, and the mix with repeated
scalars, whose heavy buckets are split and merged."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(engine, ocpu, n, kind, seed):
    pts = engine.generate_bases(seed, n)
    sc = engine.generate_scalars(seed + 1, n, kind=kind, msm_index=3)
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        out = engine.multi_scalar_mult(ctx, pts, sc)
    finally:
        ctx.close()
    assert np.array_equal(out[0], ocpu.msm(pts, sc))


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 257, 5000, 53970, 53971])
def test_entry_limit(engine, ocpu, n, kind):
    run(engine, ocpu, n, kind, 40 + n % 97)


@pytest.mark.parametrize("bits", [15, 18, 19])
@pytest.mark.parametrize("n", [9, 3000])
def test_level_one_limit(engine, ocpu, monkeypatch, n, bits):
    monkeypatch.setenv("MSM_FIXED_BASE", str(bits))
    run(engine, ocpu, n, 1, 7 * bits + n)


@pytest.mark.parametrize("bits", [6, 13])
def test_windowed(engine, ocpu, bits):
    n = 4099
    pts = engine.generate_bases(91, n)
    sc = engine.generate_scalars(92, n, kind=1, msm_index=1)
    sc[5] = 0
    sc[7] = np.uint64(2**64 - 1)  # at or above r: 253 bits are used
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        out = ctx.mult(sc, window_bits=bits, fixed_base=2)
    finally:
        ctx.close()
    ref = engine.multi_scalar_mult_init(pts)
    try:
        want = engine.multi_scalar_mult(ref, pts, sc)
    finally:
        ref.close()
    assert np.array_equal(out, want)


@pytest.mark.parametrize("tables", ["0", "11", "16", "17"])
@pytest.mark.parametrize("n", [1, 300, 20011, 65536])
def test_noalloc_layouts(engine, ocpu, monkeypatch, n, tables):
    """msm_mult_noalloc on tables of at most 16 bits and on windows where the context has none."""
    import torch

    monkeypatch.setenv("MSM_FIXED_BASE", tables)
    pts = engine.generate_bases(71, n + 3)
    sc = engine.generate_scalars(72, n, kind=1, msm_index=2)
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        d_sc = torch.from_numpy(sc.view(np.uint8).reshape(-1)).cuda()
        d_out = torch.zeros(144, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        for _ in range(2):
            ctx.mult_noalloc(n, 3, d_sc.data_ptr(), d_out.data_ptr())
        torch.cuda.synchronize()
    finally:
        ctx.close()
    assert np.array_equal(d_out.cpu().numpy(), ocpu.msm(pts[3:], sc))


def test_groups_of_an_open_mode(engine, ocpu):
    """Without a mode, consecutive MSMs share passes up to 2^22 points; MSMs around that limit, empty
    ones and small ones on either side, host and device scalars, as one pass each."""
    import torch

    nbase = (1 << 22) + 5
    pts = engine.generate_bases(61, 1 << 12)
    pts = np.concatenate([pts] * ((nbase >> 12) + 1))[:nbase]
    sizes = [10, 0, 3000, 1 << 22, (1 << 22) - 3, 4, 7, nbase, 0, 1]
    offs = [5, 9, 100, 2, 0, nbase - 4, 1, 0, nbase, 77]
    sc = engine.generate_scalars(62, 1 << 16)
    sc = np.concatenate([sc] * ((sum(sizes) >> 16) + 1))[:sum(sizes)]
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        want = ctx.mult_uneven(sizes, offs, sc, mode=1)
        assert np.array_equal(ctx.mult_uneven(sizes, offs, sc), want)
        d_sc = torch.from_numpy(np.ascontiguousarray(sc).view(np.uint8).reshape(-1)).cuda()
        torch.cuda.synchronize()
        assert np.array_equal(ctx.mult_device(sizes, offs, d_sc.data_ptr()), want)
        at = sum(sizes[:2])
        assert np.array_equal(want[2], ocpu.msm(pts[100:3100], sc[at:at + 3000]))
    finally:
        ctx.close()
