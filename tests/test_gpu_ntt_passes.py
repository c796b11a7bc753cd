"""Every split of a transform into passes (1, 2 or 3 of 2^4 to 2^8 points) on the GPU against the
oracle, bit-exact, both directions: all sizes, with edge values and values at or above p, device
buffers that start 8 bytes off a 16-byte boundary, and in place where the entry point takes it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0xFFFFFFFF00000001


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("log_n", list(range(0, 24)))
def test_every_size(engine, ocpu, log_n, inverse):
    import torch

    from hardcaml_zprize_gb300.ntt import NttContext
    n = 1 << log_n
    rng = np.random.default_rng(1000 + 2 * log_n + inverse)
    x = rng.integers(0, 2**64, n, dtype=np.uint64)
    edge = np.array([2**64 - 1, P - 1, P, 0, 1, 2**32 - 1, 2**32, 2**63], dtype=np.uint64)
    at = rng.random(n) < 0.3
    x[at] = edge[rng.integers(0, len(edge), int(at.sum()))]
    want = ocpu.ntt(x % np.uint64(P), inverse=inverse)
    ctx = NttContext(log_n, inverse=inverse)
    try:
        d = torch.zeros(2 * n + 2, dtype=torch.int64, device="cuda")
        src, dst = d[1:n + 1], d[n + 1:2 * n + 1]
        src.copy_(torch.from_numpy(x.view(np.int64)))
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        ctx.evaluate_device(dst.data_ptr(), src.data_ptr(), stream.cuda_stream)
        torch.cuda.synchronize()
        assert np.array_equal(dst.cpu().numpy().view(np.uint64), want)
        assert int(d[0]) == 0 and int(d[-1]) == 0
        if log_n > 12:
            ctx.evaluate_device(src.data_ptr(), src.data_ptr(), stream.cuda_stream)
            torch.cuda.synchronize()
            assert np.array_equal(src.cpu().numpy().view(np.uint64), want)
    finally:
        ctx.close()


@pytest.mark.parametrize("log_n,count", [(0, 1), (1, 4), (12, 1), (12, 4), (12, 5), (18, 4), (19, 3), (19, 4), (21, 1), (21, 2)])
def test_batch_sizes(engine, ocpu, log_n, count):
    """Host batches on both sides of the rule that runs a few vectors on one stream, from a buffer on a
    16-byte boundary (read by the copy kernel) and one 8 bytes off it (copied by the driver)."""
    from hardcaml_zprize_gb300.ntt import NttContext
    n = 1 << log_n
    buf = np.random.default_rng(5 * log_n + count).integers(0, 2**64, count * n + 3, dtype=np.uint64)
    off = (buf.ctypes.data >> 3) & 1
    ctx = NttContext(log_n)
    try:
        for start in (off, 1 + off):
            xs = buf[start:start + count * n].reshape(count, n)
            got = ctx.evaluate_batch(xs)
            for i in range(count):
                assert np.array_equal(got[i], ocpu.ntt(xs[i] % np.uint64(P))), (start, i)
    finally:
        ctx.close()
