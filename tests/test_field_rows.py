"""Host-side check of the column-split field products (field.cuh: mul_redc,
mul_add_redc, redc_wide), compiled by nvcc for the CPU: a b R^-1, (a b + c d) R^-1
and t R^-1 mod p in [0, 2p) against Python integers.  Operands whose limbs are all
ones or zero make every row carry, and none may be lost at the vectors' ends."""
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
Q = 0x30644E72E131A029B85045B68181585D97816A916871CA8D3C208C16D87CFD47
R_ORDER = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001
R = 1 << 256

PROBE = r"""
#include <cstdio>
#include "field.cuh"
template <class P>
void run(int mode, unsigned (*a)[8], unsigned* r) {
    if (mode == 0) g16d::mul_redc<P>(a[0], a[1], r);
    else if (mode == 1) g16d::mul_add_redc<P>(a[0], a[1], a[2], a[3], r);
    else g16d::redc_wide<P>(a[0], r);   // a[0] low, a[1] high
}
// lines of: modulus (0 q, 1 r), mode, then 4 operands of 8 hex limbs
int main() {
    unsigned a[4][8], r[8];
    int field, mode;
    while (scanf("%d %d", &field, &mode) == 2) {
        for (int k = 0; k < 4; k++)
            for (int i = 0; i < 8; i++)
                if (scanf("%x", &a[k][i]) != 1) return 1;
        if (field == 0) run<g16d::FqParams>(mode, a, r);
        else run<g16d::FrParams>(mode, a, r);
        for (int i = 0; i < 8; i++) printf("%08x ", r[i]);
        printf("\n");
    }
    return 0;
}
"""


def _limbs(x):
    return " ".join("%x" % ((x >> (32 * i)) & 0xFFFFFFFF) for i in range(8))


@pytest.mark.parametrize("field,mod", [(0, Q), (1, R_ORDER)], ids=["q", "r"])
def test_products_and_reduction_match_big_integers(tmp_path, field, mod):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not on PATH")
    src, exe = tmp_path / "probe.cu", tmp_path / "probe"
    src.write_text(PROBE)
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "snarkrs_b200", "csrc"), "-o", str(exe),
                    str(src)], check=True, capture_output=True)
    rng = random.Random(13 + field)
    edge = [0, 1, mod - 1, mod - 2, (1 << 253) - 1, (1 << 224) - 1, (1 << 253) - (1 << 32), R % mod]
    quads = [(a, b, mod, mod - 1) for a in edge for b in edge] + [(a, b, b, a) for a in edge for b in edge]
    quads += [tuple(rng.randrange(mod) for _ in range(4)) for _ in range(300)]
    wide = [0, 1, mod * R - 1, (1 << 256) - 1, mod << 32] + [rng.randrange(mod * R) for _ in range(300)]
    cases = [(0, q, q[0] * q[1]) for q in quads] + [(1, q, q[0] * q[1] + q[2] * q[3]) for q in quads]
    cases += [(2, (t % R, t >> 256, 0, 0), t) for t in wide]
    text = "".join("%d %d %s\n" % (field, m, " ".join(map(_limbs, q))) for m, q, _ in cases)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
    r_inv = pow(R, -1, mod)
    assert len(out) == len(cases) + 1
    for (_, q, want), line in zip(cases, out):
        v = sum(int(w, 16) << (32 * i) for i, w in enumerate(line.split()))
        assert v < 2 * mod and v % mod == want * r_inv % mod, q
