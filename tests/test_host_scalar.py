"""The host's scalar products (host_bn254.hpp: fixed_base_mul over a table of
multiples, mul_pair with shared doublings), compiled here for the CPU: equal to
double-and-add on G1 and G2 for scalars at the edges of the signed digits
(0, 1, r - 1, runs of 8s and 9s that borrow or carry through every digit) and
random ones, and for operands at infinity."""
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
R_ORDER = 0x30644E72E131A029B85045B68181585D2833E84879B9709143E1F593F0000001

PROBE = r"""
#include <cstdio>
#include "host_bn254.hpp"
using namespace g16;
template <class F>
bool same(const Jac<F>& a, const Jac<F>& b) {
    Affine<F> x = a.to_affine(), y = b.to_affine();
    return x.inf == y.inf && x.x == y.x && x.y == y.y;
}
template <class F>
bool check(const Affine<F>& g, const uint64_t* k, const uint64_t* l) {
    const Jac<F> a = Jac<F>::from_affine(g), b = a.dbl() + a, o = Jac<F>::identity();
    const std::vector<Affine<F>> table = fixed_base_table(g);
    return same(fixed_base_mul(table, k), a.mul(k)) && same(mul_pair(a, k, b, l), a.mul(k) + b.mul(l)) &&
           same(mul_pair(o, k, b, l), b.mul(l)) && same(mul_pair(a, k, a.neg(), k), o);
}
int main() {
    host_init();
    uint64_t k[4], l[4];
    int n = 0;
    while (scanf("%lx %lx %lx %lx %lx %lx %lx %lx", &k[0], &k[1], &k[2], &k[3], &l[0], &l[1], &l[2], &l[3]) == 8) {
        if (!check(G1_GENERATOR, k, l) || !check(G2_GENERATOR, k, l)) return printf("case %d differs\n", n), 1;
        n++;
    }
    printf("%d\n", n);
    return 0;
}
"""


def test_products_equal_double_and_add(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not on PATH")
    src, exe = tmp_path / "probe.cpp", tmp_path / "probe"
    src.write_text(PROBE)
    csrc = os.path.join(ROOT, "snarkrs_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", csrc, "-o", str(exe), str(src),
                    os.path.join(csrc, "host_bn254.cpp")], check=True, capture_output=True)
    rng = random.Random(31)
    edge = [0, 1, 8, 9, 16, R_ORDER - 1, int("8" * 63, 16), int("9" * 62, 16), int("7" + "8" * 62, 16) % R_ORDER,
            (1 << 253) - 1]
    pairs = [(a, rng.choice(edge)) for a in edge] + [(rng.randrange(R_ORDER), rng.randrange(R_ORDER)) for _ in range(20)]
    words = lambda x: " ".join("%x" % ((x >> (64 * i)) & (2 ** 64 - 1)) for i in range(4))
    out = subprocess.run([str(exe)], input="".join("%s %s\n" % (words(a), words(b)) for a, b in pairs),
                         capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.split() == [str(len(pairs))], out.stdout
