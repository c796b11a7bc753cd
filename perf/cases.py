"""The calls whose speed this repository is measured by: MSMs over BLS12-377 G1 and Goldilocks NTTs,
through the public entry points of `hardcaml_zprize_gb300`, over the range of sizes that the
library's own tests, configurations and benchmark cover.

A case is a dict: `op` names the entry point, the other keys its sizes and options.
  harness  multi_scalar_mult: `batch` MSMs of `n` points, scalars in pageable host memory, as the
           reference's Rust harness calls it
  device   MultiScalarMultContext.mult_device: one MSM of `n` points, scalars already in HBM;
           `tables` False asks for the plain resident records (what a base set too large for
           fixed-base tables gets)
  uneven   MultiScalarMultContext.mult_device, `count` MSMs of log-uniform sizes in one pass over
           slices of `n` shared bases, mixed scalars; the sizes follow from `mix`
  noalloc  MultiScalarMultContext.mult_noalloc: one MSM of `n` points on a stream, no allocation
  ntt      NttContext.evaluate_device: one transform of 2^`log_n` points between device buffers
  ntt_host NttContext.evaluate_batch: `batch` transforms of 2^`log_n` points, host to host

Every output is a whole number (curve points as canonical bytes, field elements), so results are
compared for equality; there is no rounding to compare with.
"""
import numpy as np
import torch

import hardcaml_zprize_gb300 as eng
from hardcaml_zprize_gb300.ntt import NttContext

_streams = []


def _stream():
    """The stream that all transforms of this program are enqueued on, one after another."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def listed():
    return [
        # the smallest proofs: one MSM of a few thousand points, where launches and the serial
        # tail of the reduction are the time
        {"name": "msm_4k_host", "op": "harness", "n": 4096, "batch": 1},
        # the harness's batch call: several scalar vectors over one base set, ragged size
        {"name": "msm_50k_host_x4", "op": "harness", "n": 50000, "batch": 4},
        # an ordinary circuit: 2^20 points, scalars left in HBM by the previous step
        {"name": "msm_1m_device", "op": "device", "n": 1 << 20, "tables": True},
        # a large ragged circuit with its scalars on the host
        {"name": "msm_3m_host", "op": "harness", "n": 3000001, "batch": 1},
        # the headline size
        {"name": "msm_16m_device", "op": "device", "n": 1 << 24, "tables": True},
        # plain records instead of tables, as for a base set that leaves no room for tables
        {"name": "msm_2m_plain", "op": "device", "n": 1 << 21, "tables": False},
        # many MSMs of very different sizes in one pass (the benchmark's uneven mix: repeated,
        # short and extreme scalars among uniform ones)
        {"name": "msm_uneven_x64", "op": "uneven", "n": 1 << 20, "count": 64, "mix": 7},
        # inside another runtime's memory pool: no allocation, stream-ordered
        {"name": "msm_noalloc_20k", "op": "noalloc", "n": 20011},
        # the smallest transform of one block
        {"name": "ntt_4k", "op": "ntt", "log_n": 12, "inverse": False},
        # an ordinary transform, the inverse direction, odd log2
        {"name": "intt_512k", "op": "ntt", "log_n": 19, "inverse": True},
        # the NTT track's size
        {"name": "ntt_16m", "op": "ntt", "log_n": 24, "inverse": False},
        # host to host, transfers overlapping the transforms
        {"name": "ntt_4m_host_x4", "op": "ntt_host", "log_n": 22, "batch": 4, "inverse": False},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    op = rng.choice(["harness", "harness", "device", "device", "uneven", "noalloc", "ntt", "ntt", "ntt_host"])
    if op == "harness":
        n = _log_uniform(rng, 1000, 1 << 22)
        return {"op": op, "n": n, "batch": 1 + int(rng.random() * min(6, (1 << 23) / n))}
    if op == "device":
        return {"op": op, "n": _log_uniform(rng, 1000, 1 << 23), "tables": rng.random() < 0.7}
    if op == "uneven":
        return {"op": op, "n": _log_uniform(rng, 1 << 15, 1 << 20), "count": rng.randint(8, 64),
                "mix": rng.randint(100, 1 << 20)}
    if op == "noalloc":
        return {"op": op, "n": _log_uniform(rng, 1000, 1 << 16)}
    if op == "ntt":
        return {"op": op, "log_n": rng.randint(10, 24), "inverse": rng.random() < 0.5}
    log_n = rng.randint(12, 22)
    return {"op": op, "log_n": log_n, "batch": rng.randint(1, 4), "inverse": rng.random() < 0.5}


def _mix(case):
    """Sizes and base offsets of an uneven batch: 2^U points, U uniform from 10 to log2 n."""
    rng = np.random.default_rng(case["mix"])
    sizes = [int(2 ** u) for u in rng.uniform(10, np.log2(case["n"]), case["count"])]
    return sizes, [int(rng.integers(0, case["n"] - s + 1)) for s in sizes]


def _prepare_ntt(case, seed):
    n, gen = 1 << case["log_n"], torch.Generator(device="cuda").manual_seed(seed)
    count = case.get("batch", 1)
    # 64-bit patterns, as good as uniform below p (inputs are taken modulo p)
    x = torch.randint(-(1 << 63), (1 << 63) - 1, (count * n,), generator=gen, device="cuda")
    s = {"op": case["op"], "ctx": NttContext(case["log_n"], inverse=case["inverse"])}
    if case["op"] == "ntt_host":
        s["x"] = x.cpu().numpy().view(np.uint64).reshape(count, n)
        s["out"] = np.zeros_like(s["x"])
        return s
    s.update(x=x, out=torch.zeros_like(x), stream=_stream())
    s["stream"].wait_stream(torch.cuda.current_stream())
    return s


def prepare(case, seed):
    op = case["op"]
    if op in ("ntt", "ntt_host"):
        return _prepare_ntt(case, seed)
    n = case["n"]
    points = eng.generate_bases(seed, n)
    s = {"op": op, "ctx": eng.multi_scalar_mult_init(points)}
    if op == "harness":
        s.update(points=points, scalars=eng.generate_scalars(seed + 1, n * case["batch"]))
        return s
    if op == "uneven":
        sizes, offsets = _mix(case)
        scalars = np.concatenate([eng.generate_scalars(seed + 1, k, kind=1, msm_index=j)
                                  for j, k in enumerate(sizes)])
        s.update(sizes=sizes, offsets=offsets, opts={"mode": 2})
    else:
        scalars = eng.generate_scalars(seed + 1, n)
        s.update(sizes=[n], offsets=[0], opts={})
        if not case.get("tables", True):
            s["opts"] = {"fixed_base": 2}
    s["scalars"] = torch.from_numpy(scalars.view(np.uint8).reshape(-1)).cuda()
    if op == "noalloc":
        s.update(n=n, out=torch.zeros(eng.PROJ_BYTES, dtype=torch.uint8, device="cuda"))
    return s


def run(s):
    op, ctx = s["op"], s["ctx"]
    if op == "harness":
        return eng.multi_scalar_mult(ctx, s["points"], s["scalars"])
    if op == "ntt":
        ctx.evaluate_device(s["out"].data_ptr(), s["x"].data_ptr(), s["stream"].cuda_stream)
        return s["out"]
    if op == "ntt_host":
        return ctx.evaluate_batch(s["x"], s["out"]).view(np.int64)
    if op == "noalloc":  # every call shares one scratch array: all on the default stream
        ctx.mult_noalloc(s["n"], 0, s["scalars"].data_ptr(), s["out"].data_ptr())
        return s["out"]
    return ctx.mult_device(s["sizes"], s["offsets"], s["scalars"].data_ptr(), **s["opts"])


def _msm_work(n, bases=None):
    """One MSM of n points by buckets of signed c-bit digits, at the width that needs the fewest
    products: 7 field products per (point, window), 16 per bucket of one shared bucket array; a
    product of two 377-bit values is 276 wide multiplies of 32-bit words, two operations each."""
    products = min(7.0 * n * -(-253 // c) + 16.0 * 2 ** (c - 1) for c in range(4, 27))
    return {"bytes": 32.0 * n + 144.0 * (n if bases is None else bases) + 144, "flops": 552.0 * products}


def work(case):
    if case["op"] in ("ntt", "ntt_host"):
        n, count = 1 << case["log_n"], case.get("batch", 1)
        # one modular product (4 wide multiplies), sum and difference per butterfly
        return {"bytes": 16.0 * n * count, "flops": 0.5 * n * case["log_n"] * 10 * count}
    if case["op"] == "uneven":
        each = [_msm_work(k, 0) for k in _mix(case)[0]]
        return {"bytes": sum(w["bytes"] for w in each) + 144.0 * case["n"], "flops": sum(w["flops"] for w in each)}
    w, batch = _msm_work(case["n"]), case.get("batch", 1)
    return {"bytes": 144.0 * case["n"] + 32.0 * case["n"] * batch, "flops": w["flops"] * batch}
