"""Host-side check of the MSM bucket-reduction plan (msm_reduce_plan in
snarkrs_b200/csrc/msm.cuh), compiled here by nvcc for the CPU.

For every window width the prover and the standalone MSM can use, over G1 and
G2 and both piece targets, the plan must cover every bucket exactly once
(pieces x seg = B, blocks x 2^lb >= pieces), keep seg a power of two no larger
than 32, take the direct path only for at most two blocks in all, and give the
finish kernel no more bit terms than it has groups; a prover MSM's set sums fit
its readback slot (MSM_RESULT_SLOT_BYTES).
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include <cstdio>
#include "msm.cuh"
int main() {
    printf("%zu %u %u\n", g16::MSM_RESULT_SLOT_BYTES, g16::MSM_REDUCE_LB_G1, g16::MSM_REDUCE_LB_G2);
    unsigned sets, B, g2;
    unsigned long long target;
    while (scanf("%u %u %u %llu", &sets, &B, &g2, &target) == 4) {
        g16::MsmReducePlan p = g16::msm_reduce_plan(sets, B, g2 != 0, target);
        printf("%u %u %u %u %d %u %zu %zu\n", p.seg, p.lb, p.nb, p.hb, p.direct ? 1 : 0, p.set_terms(),
               p.block_points(), p.result_points());
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def plan():
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not on PATH")
    import tempfile
    d = tempfile.mkdtemp(prefix="plan_probe")
    src, exe = os.path.join(d, "probe.cu"), os.path.join(d, "probe")
    open(src, "w").write(PROBE)
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "snarkrs_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-o", exe, src], check=True, capture_output=True)

    def run(cases):
        text = "\n".join("%d %d %d %d" % c for c in cases) + "\n"
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
        run.slot_bytes, run.lb_g1, run.lb_g2 = map(int, out[0].split())
        keys = ("seg", "lb", "nb", "hb", "direct", "set_terms", "block_points", "result_points")
        return [dict(zip(keys, map(int, l.split()))) for l in out[1:] if l.strip()]
    yield run
    shutil.rmtree(d, ignore_errors=True)


def test_plans_cover_every_bucket(plan):
    cases = []
    for c in range(1, 23):
        B = 1 << (c - 1)
        for sets in (1, 2, 3, (255 + c - 1) // c):
            for g2 in (0, 1):
                for target in (8192, 32768):
                    cases.append((sets, B, g2, target))
    for (sets, B, g2, target), p in zip(cases, plan(cases)):
        seg, lb, nb = p["seg"], p["lb"], p["nb"]
        assert lb == (plan.lb_g2 if g2 else plan.lb_g1)
        assert seg & (seg - 1) == 0 and 1 <= seg <= 32 and seg <= B
        pieces = B // seg
        assert pieces * seg == B
        assert nb & (nb - 1) == 0 and nb << lb >= pieces and (nb - 1) << lb < pieces
        assert (1 << p["hb"]) == nb
        assert p["direct"] == (sets * nb <= 2)
        if seg < 32 and seg < B:
            assert sets * B // seg <= target      # seg stops growing once the target is met
        if seg > 1:
            assert sets * B // (seg // 2) > target
        assert p["block_points"] == sets * nb * (lb + 2)
        terms = nb * (lb + 2) if p["direct"] else lb + 1 + p["hb"]
        assert p["set_terms"] == terms and p["result_points"] == sets * terms


def test_results_fit_the_readback_slot(plan):
    # the prover reads each MSM's result, one point per bucket set, into a pinned slot: one
    # set with window tables, one per window with a compact key, at every window width a
    # plan or a tuning may set (8 to 20 bits)
    plan([(1, 1, 0, 8192)])
    for c in range(8, 21):
        assert (255 + c - 1) // c * 256 <= plan.slot_bytes


def test_finish_kernel_has_a_group_for_every_bit_term(plan):
    # 32 groups: the bit terms, T in the last (window widths up to 24, any piece target)
    cases = [(sets, 1 << (c - 1), g2, t) for c in range(4, 25) for sets in (1, (255 + c - 1) // c)
             for g2 in (0, 1) for t in (1, 8192, 32768, 1 << 40)]
    for _, p in zip(cases, plan(cases)):
        assert p["lb"] + p["hb"] < 31


LAYOUT_PROBE = r"""
#include <cstdio>
#include <vector>
#include "msm.cuh"
int main() {
    printf("%u %u %u\n", g16::MSM_REDUCE_LB_G1, g16::MSM_REDUCE_LB_G2, g16::MSM_REDUCE_MAX_SEG);
    unsigned nseg, g2, sms, override_len;
    unsigned long long target;
    while (scanf("%u %u %llu %u %u", &nseg, &g2, &target, &sms, &override_len) == 5) {
        std::vector<uint32_t> B(nseg);
        for (auto& b : B) scanf("%u", &b);
        g16::MsmSpaceReduceLayout L = g16::msm_space_reduce_layout(B, g2 != 0, target, sms, override_len);
        printf("%llu %llu %llu %llu %u %u\n", (unsigned long long)L.K, (unsigned long long)L.blocks,
               (unsigned long long)L.block_points, (unsigned long long)L.result_points, L.max_hb, L.piece_len);
        for (size_t j = 0; j < B.size(); j++) {
            const g16::MsmReducePlan& p = L.plans[j];
            printf("%u %u %u %u %u %d %u %u %u %u %u\n", p.seg, p.lb, p.nb, p.hb, p.sets, p.direct ? 1 : 0,
                   L.key_start[j], L.block_start[j], L.out_block[j], L.out_set[j], p.set_terms());
        }
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def layout():
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not on PATH")
    import tempfile
    d = tempfile.mkdtemp(prefix="layout_probe")
    src, exe = os.path.join(d, "probe.cu"), os.path.join(d, "probe")
    open(src, "w").write(LAYOUT_PROBE)
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "snarkrs_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-o", exe, src], check=True, capture_output=True)

    def run(cases):
        text = "".join("%d %d %d %d %d %s\n" % (len(Bs), g2, target, sms, ovr, " ".join(map(str, Bs)))
                       for Bs, g2, target, sms, ovr in cases)
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
        run.lb_g1, run.lb_g2, run.max_seg = map(int, out[0].split())
        res, i = [], 1
        for Bs, *_ in cases:
            tot = dict(zip(("K", "blocks", "block_points", "result_points", "max_hb", "piece_len"),
                           map(int, out[i].split())))
            segs = [dict(zip(("seg", "lb", "nb", "hb", "sets", "direct", "key_start", "block_start", "out_block",
                              "out_set", "set_terms"), map(int, out[i + 1 + j].split()))) for j in range(len(Bs))]
            res.append((tot, segs))
            i += 1 + len(Bs)
        return res
    yield run
    shutil.rmtree(d, ignore_errors=True)


def test_batched_reduction_layout_matches_the_kernels(layout):
    # Random mixes of segments (the batched engine's spaces) laid out by
    # msm_space_reduce_layout, then the indexing of k_reduce_pieces_multi and
    # k_reduce_sets_multi replayed on that layout: every block finds its own
    # segment, reads only its segment's buckets, and writes only its own points;
    # every sets-kernel read and write stays inside its segment and the buffers.
    import random
    rng = random.Random(11)
    cases = []
    for _ in range(300):
        nseg = rng.randrange(1, 40)
        Bs = [1 << (rng.randrange(4, 22) - 1) for _ in range(nseg)]
        g2 = rng.randrange(2)
        target = rng.choice([0, 0, 0, 8192, 32768, 1 << rng.randrange(4, 18)])
        sms = rng.choice([148, 132, 1, 7])
        ovr = rng.choice([0, 0, 0, 0, 1, 2, 8, 32, 3, 64])
        cases.append((Bs, g2, target, sms, ovr))
    for (Bs, g2, target, sms, ovr), (tot, segs) in zip(cases, layout(cases)):
        LB = layout.lb_g2 if g2 else layout.lb_g1   # the kernels' template argument
        assert tot["K"] == sum(Bs)
        if ovr in (1, 2, 4, 8, 16, 32):
            assert tot["piece_len"] == ovr
        k = b = bp = rp = 0
        for B, s in zip(Bs, segs):
            assert s["lb"] == LB and s["sets"] == 1 and s["direct"] == 0
            assert (s["key_start"], s["block_start"], s["out_block"], s["out_set"]) == (k, b, bp, rp)
            pieces = B // s["seg"]
            assert pieces * s["seg"] == B and 1 <= s["seg"] <= layout.max_seg
            nb, hb = s["nb"], s["hb"]
            assert nb >= 1 and (nb << LB) >= pieces and ((nb - 1) << LB) < pieces and (1 << hb) == nb
            # k_reduce_pieces_multi: block jb < nb of this segment reads buckets
            # key_start + p*seg + i (p*seg < B) and writes out_block + jb*(LB+2) + [0, LB+1]
            last_write = s["out_block"] + (nb - 1) * (LB + 2) + LB + 1
            assert last_write < bp + nb * (LB + 2) <= tot["block_points"]
            # k_reduce_sets_multi: term o < LB+1+hb reads out_block + j*(LB+2) + min(o, LB+1), j < nb,
            # and writes out_set + o
            assert s["set_terms"] == LB + 1 + hb
            assert s["out_set"] + LB + hb < rp + s["set_terms"] <= tot["result_points"]
            k += B
            b += nb
            bp += nb * (LB + 2)
            rp += s["set_terms"]
        assert (k, b, bp, rp) == (tot["K"], tot["blocks"], tot["block_points"], tot["result_points"])
        assert tot["max_hb"] == max(s["hb"] for s in segs)
        # a block finds its segment by the last block_start <= block (strictly increasing)
        starts = [s["block_start"] for s in segs]
        assert all(x < y for x, y in zip(starts, starts[1:]))


def _plan_probe(defines):
    """The plan probe compiled with extra -D flags (another reduction block size)."""
    import tempfile
    d = tempfile.mkdtemp(prefix="plan_probe_d")
    src, exe = os.path.join(d, "probe.cu"), os.path.join(d, "probe")
    open(src, "w").write(PROBE)
    subprocess.run(["nvcc", "-std=c++17", "-O1"] + defines + ["-I", os.path.join(ROOT, "snarkrs_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-o", exe, src], check=True, capture_output=True)

    def run(cases):
        text = "\n".join("%d %d %d %d" % c for c in cases) + "\n"
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
        keys = ("seg", "lb", "nb", "hb", "direct", "set_terms", "block_points", "result_points")
        return [dict(zip(keys, map(int, l.split()))) for l in out[1:] if l.strip()]
    return run, d


def _piece_block(S, g0s, seg, LB):
    """reduce_piece_block: the block's LB + 2 points from its 2^LB pieces (g0s: a piece's
    first bucket, None past the set's end).  Two groups a piece; slots are written only
    by their own group, and no step may read a slot that another group writes in it."""
    N, weighted = 1 << LB, seg > 1
    first, second = [0] * N, [0] * N
    nxt = [0 if g is None else S[g + seg - 1] for g in g0s]
    for j in range(seg + 1 if weighted else 1):
        second = [y + x for x, y in zip(first, second)]      # tot, one step behind run
        first = [x + v for x, v in zip(first, nxt)]
        nxt = [S[g + seg - 2 - j] if g is not None and j + 1 < seg else 0 for g in g0s]
    acc = [list(first), list(second)]
    slots = [list(first), list(second)]
    lg = [t.bit_length() - 1 if t else 0 for t in range(N)]
    for k in range(1, LB + 1):
        h = N >> k
        for half in (0, 1):
            src = {}
            for t in range(N):
                if t < h:
                    if not half or weighted:
                        src[t] = t + h
                elif t >= 2 * h and not half:
                    hs, s = 1 << lg[t], 1 << (k - (LB - lg[t]) - 1)
                    o = t - hs
                    if o & (2 * s - 1) == 0 and o + s < hs:
                        src[t] = t + s
            assert not set(src) & set(src.values()), "a slot read in the step that writes it"
            for t, x in src.items():
                acc[half][t] += slots[half][x]
            for t in src:
                slots[half][t] = acc[half][t]
    out = [None] * (LB + 2)
    out[0] = acc[1][0] if weighted else acc[0][0]            # T
    out[LB + 1] = acc[0][0]                                  # R
    for t in range(1, N):
        if t & (t - 1) == 0:
            out[1 + lg[t]] = acc[0][t]                       # G_lg
    return out


def _set_term(points, base, nb, o, LB):
    """reduce_set_term: one term of a set over its nb blocks."""
    bits = o > LB
    i, count = (o - LB - 1, nb // 2) if bits else (0, nb)
    at = lambda x: ((x >> i) << (i + 1)) | (1 << i) | (x & ((1 << i) - 1)) if bits else x
    js = [at(x) for x in range(count)]
    assert js == [j for j in range(nb) if not bits or (j >> i) & 1]
    return sum(points[base + j * (LB + 2) + (LB + 1 if bits else o)] for j in js)


def _finish(points, base, LB, nb, hb, direct, seg):
    """reduce_finish: 32 groups of lanes, the bit terms combined in a tree, T in the last."""
    m, G = LB + hb, 32
    assert m < G - 1 and (not direct or nb <= 2)
    acc = [0] * G
    for g in range(G):
        is_t = g == G - 1
        if not direct:
            if g < m or is_t:
                acc[g] = points[base + (0 if is_t else 1 + g)]
            continue
        low, o = is_t or g < LB, 0 if is_t else 1 + g
        if low:
            acc[g] = points[base + o]
        elif g < m:
            acc[g] = points[base + (LB + 2) + LB + 1]
        if nb > 1 and low:
            acc[g] += points[base + (LB + 2) + o]
    smem, s = [None] * G, 1
    while s < m:
        for g in range(G):
            if g & (2 * s - 1) == s and g < m:
                acc[g] <<= s                                 # s doublings
                assert smem[g] is None, "a slot written twice"
                smem[g] = acc[g]
        for g in range(G):
            if g & (2 * s - 1) == 0 and g + s < m:
                acc[g] += smem[g + s]
        s *= 2
    return acc[0] * seg + acc[G - 1]


def _emulate_reduction(S, sets, B, p):
    """k_reduce_pieces, k_reduce_sets and k_reduce_finish (msm.cu) on integers standing in
    for points (an addition is +, a doubling *2), step by step as the kernels index them."""
    LB, seg, nb, hb = p["lb"], p["seg"], p["nb"], p["hb"]
    points = []
    for st in range(sets):
        for jb in range(nb):
            pieces = [(jb << LB) + t for t in range(1 << LB)]
            points += _piece_block(S, [st * B + x * seg if x * seg < B else None for x in pieces], seg, LB)
    assert None not in points and len(points) == p["block_points"]
    stride = nb * (LB + 2)
    if not p["direct"]:
        points = [_set_term(points, st * stride, nb, o, LB) for st in range(sets) for o in range(LB + 1 + hb)]
        stride = LB + 1 + hb
    assert stride == p["set_terms"]
    return [_finish(points, st * stride, LB, nb, hb, p["direct"], seg) for st in range(sets)]


@pytest.mark.parametrize("defines", [[], ["-DG16_REDUCE_LB_G1=7", "-DG16_REDUCE_LB_G2=6"]],
                         ids=["blocks-of-2^5-and-2^4", "blocks-of-2^7-and-2^6"])
def test_reduction_algebra_by_integer_emulation(defines):
    # the pieces kernel's running sums, halvings and per-bit trees, the sets kernel and the
    # finish kernel's tree give sum_b (b + 1) S_b for every plan shape: direct (one block a
    # set, two blocks of one) and through the sets kernel, weighted (seg > 1) and not, one or
    # several sets; and as a batched space runs it, which never takes the direct path
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not on PATH")
    import random
    run, d = _plan_probe(defines)
    try:
        rng = random.Random(5)
        cases = []
        for B in (1, 2, 8, 64, 256, 1024, 4096):
            for sets in (1, 2, 3):
                for g2 in (0, 1):
                    for target in (1, 16, 256, 8192, 32768):
                        cases.append((sets, B, g2, target))
        shapes = set()
        for (sets, B, g2, target), p in zip(cases, run(cases)):
            shape = (sets, B, p["seg"], p["nb"], p["direct"], p["lb"])
            if shape in shapes:
                continue
            shapes.add(shape)
            S = [rng.randrange(1, 1 << 20) for _ in range(sets * B)]
            want = [sum((b + 1) * S[st * B + b] for b in range(B)) for st in range(sets)]
            assert _emulate_reduction(S, sets, B, p) == want, (sets, B, g2, target, p)
            assert _emulate_reduction(S, sets, B, dict(p, direct=0, set_terms=p["lb"] + 1 + p["hb"])) == want
        assert any(s[4] == 1 for s in shapes) and any(s[4] == 0 for s in shapes)
        assert any(s[2] > 1 for s in shapes) and any(s[2] == 1 for s in shapes)
        assert {s[3] for s in shapes if s[4]} == {1, 2}
        assert any((s[5] + s[3].bit_length() - 1) & (s[5] + s[3].bit_length() - 2) for s in shapes)   # uneven trees
    finally:
        shutil.rmtree(d, ignore_errors=True)


@pytest.mark.parametrize("define,ok", [("G16_REDUCE_LB_G1=7", True), ("G16_REDUCE_LB_G1=8", False),
                                       ("G16_REDUCE_LB_G1=1", False), ("G16_REDUCE_LB_G2=6", True),
                                       ("G16_REDUCE_LB_G2=7", False), ("G16_REDUCE_LB_G2=0", False)])
def test_block_sizes_that_cannot_launch_do_not_compile(tmp_path, define, ok):
    # two groups of 4 (G1) or 8 (G2) lanes a piece, a block of one warp to 1024 threads
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not on PATH")
    src = tmp_path / "probe.cu"
    src.write_text('#include "msm.cuh"\nint main() { return 0; }\n')
    r = subprocess.run(["nvcc", "-std=c++17", "-O0", "-D" + define, "-I", os.path.join(ROOT, "snarkrs_b200", "csrc"),
                        "-I", os.path.join(ROOT, "include"), "-c", "-o", str(tmp_path / "probe.o"), str(src)],
                       capture_output=True, text=True)
    assert (r.returncode == 0) == ok, r.stderr
    assert ok or "32 to 1024 threads" in r.stderr
