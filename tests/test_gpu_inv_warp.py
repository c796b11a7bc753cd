"""The inversion by a whole warp that every MSM result's map to affine form uses (fq_inv_warp: signed 30-bit
digits over the lanes), element by element against Python's modular inverse: edge values, digits that are
all zeros or all ones, values in [q, 2q) and random ones."""
import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_inverse_by_a_warp(engine, ref):
    q = ref.Q
    rng = random.Random(23)
    vals = [1, 2, 3, q - 1, q - 2, (q - 1) // 2, (q + 1) // 2, ref.MONT_R % q, q + 1, 2 * q - 1, 2 * q - 2]
    vals += [1 << k for k in range(377)] + [(1 << k) - 1 for k in range(2, 377)] + [q - (1 << k) for k in range(376)]
    vals += [sum(((1 << 30) - 1) << (30 * k) for k in range(s, 12, 2)) for s in (0, 1)]
    vals += [rng.randrange(1, q) for _ in range(3000)] + [rng.randrange(q + 1, 2 * q) for _ in range(1000)]
    vals += [rng.randrange(1, 1 << b) for b in range(1, 376)]
    assert all(v % q and v < 2 * q for v in vals)
    a = np.array([[(v >> (32 * k)) & 0xFFFFFFFF for k in range(12)] for v in vals], dtype=np.uint32)
    out = engine.field_selftest(7, a, a)
    for v, r in zip(vals, out):
        inv = sum(int(w) << (32 * k) for k, w in enumerate(r))
        assert inv < 1 << 383 and inv * v % q == 1, hex(v)
