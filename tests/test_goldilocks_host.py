"""The NTT kernels' field arithmetic (csrc/goldilocks.cuh) is plain integer C++ shared by host and
device; this compiles it for the host with g++ and checks it against Python integers: the product in
table form on edge and random values, and the transforms of 2 to 16 points, whose roots are shifts,
against the definition with the reference's roots (zprize/ntt/host/gf.h:65-99).  All are exact."""
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HDR = os.path.join(ROOT, "hardcaml_zprize_gb300", "csrc", "goldilocks.cuh")
P = 2**64 - 2**32 + 1
OMEGA = {1: P - 1, 2: 0x0001000000000000, 3: 0xFFFFFFFEFF000001, 4: 0xEFFFFFFF00000001}

DRIVER = r"""
#include <cstdio>
#include <cinttypes>
#include "%s"
template <int L> void dft() {
  uint64_t v[1 << L];
  gl3 x[1 << L];
  for (uint64_t &a : v) if (scanf("%%" SCNu64, &a) != 1) return;
  for (int i = 0; i < 1 << L; i++) x[i] = gl3_from(v[i]);
  x[0] = gl3_biased(x[0]);
  gl_dft<L>(x);
  for (gl3 &a : x) printf("%%" PRIu64 " ", gl_canon(gl3_fold(a)));
}
int main() {
  int op;
  while (scanf("%%d", &op) == 1) {
    if (op == 0) {
      uint64_t a, b;
      if (scanf("%%" SCNu64 " %%" SCNu64, &a, &b) != 2) return 1;
      printf("%%" PRIu64, gl_mul(a, b));
    }
    if (op == 1) dft<1>();
    if (op == 2) dft<2>();
    if (op == 3) dft<3>();
    if (op == 4) dft<4>();
    puts("");
  }
}
"""


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("gl")
    (d / "t.cpp").write_text(DRIVER % HDR)
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", str(d / "t"), str(d / "t.cpp")], check=True)

    def run(lines):
        out = subprocess.run([str(d / "t")], input="\n".join(lines), capture_output=True, text=True, check=True)
        return [[int(v) for v in line.split()] for line in out.stdout.strip().split("\n")]
    return run


EDGE = [0, 1, 2, 2**32 - 1, 2**32, 2**32 + 1, 2**63, P - 2, P - 1, P, P + 1, 2**64 - 2**32 - 1, 2**64 - 2, 2**64 - 1]


def test_product_in_table_form(ask):
    rng = random.Random(3)
    pairs = [(a, b) for a in EDGE for b in EDGE if b < P] + [(rng.getrandbits(64), rng.randrange(P)) for _ in range(5000)]
    got = ask([f"0 {a} {b}" for a, b in pairs])
    inv = pow(2**64, -1, P)
    for (a, b), g in zip(pairs, got):
        assert g == [a * b * inv % P], (a, b)  # canonical, for any 64-bit a


@pytest.mark.parametrize("log_n", [1, 2, 3, 4])
def test_short_transforms(ask, log_n):
    rng = random.Random(10 + log_n)
    n, w = 1 << log_n, OMEGA[log_n]
    xs = [[v] * n for v in EDGE] + [[v if i == j else 0 for i in range(n)] for j in range(n) for v in (1, 2**64 - 1)]
    xs += [[rng.choice(EDGE) for _ in range(n)] for _ in range(300)]
    xs += [[rng.getrandbits(64) for _ in range(n)] for _ in range(300)]
    got = ask([f"{log_n} " + " ".join(map(str, x)) for x in xs])
    for x, g in zip(xs, got):
        assert g == [sum(v * pow(w, j * k, P) for j, v in enumerate(x)) % P for k in range(n)]
