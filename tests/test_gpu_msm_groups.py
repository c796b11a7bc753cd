"""Calls of many MSMs without a mode: the passes that consecutive MSMs share are bounded by the memory of
their buckets as well as by their points, and a pass that finds no memory is split, down to one MSM."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sample(ocpu, pts, sizes, offs, sc, out, step):
    first = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    for j in list(range(0, len(sizes), step)) + [len(sizes) - 1]:
        want = ocpu.msm(pts[offs[j]:offs[j] + sizes[j]], sc[first[j]:first[j + 1]])
        assert np.array_equal(out[j], want), j


@pytest.mark.parametrize("host", [True, False])
def test_one_point_msms(engine, ocpu, host):
    """65536 MSMs of one point on tables of width 16: 2^31 buckets in all."""
    import torch

    m = 1 << 16
    pts = engine.generate_bases(401, 64)
    sc = engine.generate_scalars(402, m)
    sizes, offs = [1] * m, [j % 64 for j in range(m)]
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        if host:
            out = ctx.mult_uneven(sizes, offs, sc)
        else:
            d_sc = torch.from_numpy(sc.view(np.uint8).reshape(-1)).cuda()
            torch.cuda.synchronize()
            out = ctx.mult_device(sizes, offs, d_sc.data_ptr())
    finally:
        ctx.close()
    sample(ocpu, pts, sizes, offs, sc, out, 4099)


def test_workspace_of_many_small_msms(engine, ocpu):
    """3000 MSMs of 0 to 100 points: 22 GB as one pass, the workspace stays below 4 GB."""
    import torch

    rng = np.random.default_rng(403)
    sizes = [int(x) for x in rng.integers(0, 101, 3000)]
    offs = [int(rng.integers(0, 128 - s + 1)) for s in sizes]
    pts = engine.generate_bases(404, 128)
    sc = engine.generate_scalars(405, sum(sizes), kind=1)
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        out = ctx.mult_uneven(sizes, offs, sc)
        used = free - torch.cuda.mem_get_info()[0]
    finally:
        ctx.close()
    sample(ocpu, pts, sizes, offs, sc, out, 251)
    assert used < 4 << 30


@pytest.mark.parametrize("mb", [64, 8])
def test_no_room(engine, ocpu, monkeypatch, mb):
    """Buffers refused above 64 MB (passes of a few MSMs fit) or 8 MB (one MSM fits), with a graph captured
    before and replayed after; a pass that was asked for as one still reports the failure."""
    import torch

    m, n = 40, 1000
    pts = engine.generate_bases(406, n)
    sc = engine.generate_scalars(407, m * n)
    sizes, offs = [n] * m, [0] * m
    d_sc = torch.from_numpy(sc.view(np.uint8).reshape(-1)).cuda()
    torch.cuda.synchronize()
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        one = ctx.mult_device([n], [0], d_sc.data_ptr())
        monkeypatch.setenv("MSM_ALLOC_FAIL_MB", str(mb))
        out = ctx.mult_device(sizes, offs, d_sc.data_ptr())
        sample(ocpu, pts, sizes, offs, sc, out, 13)
        assert np.array_equal(ctx.mult(sc), out)
        with pytest.raises(engine.MsmError):
            ctx.mult_device(sizes, offs, d_sc.data_ptr(), mode=2)
        assert np.array_equal(ctx.mult_device([n], [0], d_sc.data_ptr()), one)
        monkeypatch.delenv("MSM_ALLOC_FAIL_MB")
        assert np.array_equal(ctx.mult_device(sizes, offs, d_sc.data_ptr()), out)
        assert np.array_equal(ctx.mult_device(sizes, offs, d_sc.data_ptr(), mode=2), out)
    finally:
        ctx.close()


@pytest.mark.parametrize("pull", ["0", "1"])
def test_large_and_small_msms_from_host(engine, ocpu, monkeypatch, pull):
    """Around the size up to which scalars that are copied first share a pass, both ways of uploading."""
    big = (1 << 20) + 1
    pts = np.concatenate([engine.generate_bases(408, 1 << 12)] * 257)[:big]
    sizes = [7, big, 1 << 20, 5, 0, big, big, 100]
    offs = [3, 0, 1, 0, 0, 0, 0, 50]
    sc = np.concatenate([engine.generate_scalars(409, 1 << 16)] * 65)[:sum(sizes)]
    monkeypatch.setenv("MSM_HOST_PULL", pull)
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        out = ctx.mult_uneven(sizes, offs, sc)
        assert np.array_equal(ctx.mult_uneven(sizes, offs, sc, mode=1), out)
    finally:
        ctx.close()
    first = np.concatenate([[0], np.cumsum(sizes)])
    for j in (0, 3, 4, 7):
        assert np.array_equal(out[j], ocpu.msm(pts[offs[j]:offs[j] + sizes[j]], sc[first[j]:first[j + 1]])), j


def test_graphs_when_the_results_move(engine, ocpu):
    """One pass per MSM from device scalars, in calls of more and more MSMs: each replays graphs of the calls
    before it, unless the pinned results that those write to have moved."""
    import torch

    n, sizes = 200, [1, 16, 256, 512, 700, 256]
    pts = engine.generate_bases(411, n)
    sc = engine.generate_scalars(412, 4 * n)
    want = [ocpu.msm(pts, sc[k * n:(k + 1) * n]) for k in range(4)]
    d_sc = torch.from_numpy(np.tile(sc.view(np.uint8).reshape(-1), max(sizes) // 4)).cuda()
    torch.cuda.synchronize()
    ctx = engine.multi_scalar_mult_init(pts)
    try:
        for m in sizes:
            out = ctx.mult_device([n] * m, [0] * m, d_sc.data_ptr(), mode=1)
            assert all(np.array_equal(out[j], want[j % 4]) for j in range(m)), m
    finally:
        ctx.close()
