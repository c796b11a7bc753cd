"""Every split of a transform into passes (1, 2 or 3 of 2^4 to 2^8 points) on the GPU against the
oracle, bit-exact, both directions: all sizes, with edge values and values at or above p, device
buffers that start 8 bytes off a 16-byte boundary, and in place where the entry point takes it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P = 0xFFFFFFFF00000001


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("log_n", list(range(0, 22)) + [23])
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
