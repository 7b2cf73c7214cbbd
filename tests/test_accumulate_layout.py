"""The MSM accumulate's chunking and partial-sum layout (msm.cu: min_chunk, chunk_len,
k_plan_sums/_offsets/_segments, accumulate_chunks, k_fat_merge_jobs/_final,
k_bucket_sums), restated line for line on Python integers (a point becomes the
integer it stands for, an addition a +).  For skewed bucket sizes -- empty buckets, a bucket holding most entries
(a witness full of ones), single entries -- every chunk's partial sum lands in
its own slot of its bucket's range, every slot is written once, the fat-bucket
jobs and the bucket sums give each bucket the sum of its entries, and the chunk
length keeps the thread count within its cap and within the chunks that the
buffers are sized for (msm_max_chunks, compiled here from msm.cuh).  The GPU parity
tests check the CUDA code itself."""
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
ACC_THREADS = 1 << 19
FAT_PARTIALS, FAT_JOBS, FAT_JOB_MIN = 16, 64, 128
SPREAD_THREADS = 148 * 512


def min_chunk(M, floor):
    return max(floor, min(16, (M + SPREAD_THREADS - 1) // SPREAD_THREADS))


def chunk_len(M, K, L_min, wave):
    L = (M + ACC_THREADS - 1) // ACC_THREADS
    per_bucket = (M + 4 * K - 1) // (4 * K)
    L = max(L, per_bucket, L_min)
    if wave and M:
        chunks = (M + L - 1) // L
        waves = (chunks + wave - 1) // wave
        if waves > 1:
            L2 = (M + (waves - 1) * wave - 1) // ((waves - 1) * wave)
            if 20 * (waves - 1) * L2 < 19 * waves * L:
                L = L2
    return L


def fat_job_len(ns):
    return max(FAT_JOB_MIN, (ns + FAT_JOBS - 1) // FAT_JOBS)


def plan(sizes, K, L_floor, wave, tile=1024, per_block=1):
    """k_plan_sums, k_plan_offsets and k_plan_segments: M, L, the bucket offsets, the
    partial sums per bucket, their bases and the fat list, block by block."""
    Ks = len(sizes)
    tiles = (Ks + tile - 1) // tile
    blocks = max(1, (tiles + per_block - 1) // per_block)
    mine = lambda b: [range(t * tile, min((t + 1) * tile, Ks))
                      for t in range(b * per_block, min((b + 1) * per_block, tiles))]
    sums = [sum(sizes[g] for t in mine(b) for g in t) for b in range(blocks)]
    M = sum(sums)
    L = chunk_len(M, K, min_chunk(M, L_floor), wave)
    offsets, counts, fat = [None] * Ks + [M], [None] * Ks, []
    psums = [0] * blocks
    for b in range(blocks):
        off = sum(sums[:b])
        for g in (g for t in mine(b) for g in t):
            assert offsets[g] is None
            offsets[g], hi = off, off + sizes[g]
            counts[g] = (hi - 1) // L - off // L + 1 if sizes[g] else 0
            if g < K and counts[g] > FAT_PARTIALS:
                fat.append(g)
            psums[b] += counts[g]
            off = hi
    seg_base = [None] * Ks + [sum(psums)]
    for b in range(blocks):
        off = sum(psums[:b])
        for g in (g for t in mine(b) for g in t):
            seg_base[g] = off
            off += counts[g]
    return M, L, offsets, counts, seg_base, fat


def layout_and_sums(sizes, values, K, L_floor, wave, tile=1024, per_block=1):
    Ks = len(sizes)
    M, L, offsets, nseg, seg_base, fat = plan(sizes, K, L_floor, wave, tile, per_block)
    assert M == len(values) and None not in offsets and None not in seg_base
    partials = [None] * seg_base[-1]

    def store(g, t, acc):
        slot = seg_base[g] + (t - offsets[g] // L)
        assert seg_base[g] <= slot < seg_base[g] + nseg[g], (g, t)
        assert partials[slot] is None, "a slot written twice"
        partials[slot] = acc

    for t in range((M + L - 1) // L):   # accumulate_chunks, one thread per chunk
        start, end = t * L, min(t * L + L, M)
        lo, hi = 0, Ks
        while hi - lo > 1:
            mid = (lo + hi) >> 1
            if offsets[mid] <= start:
                lo = mid
            else:
                hi = mid
        g, nxt, acc = lo, offsets[lo + 1], 0
        for k in range(start, end):
            if k == nxt:
                store(g, t, acc)
                acc = 0
                g += 1
                nxt = offsets[g + 1]
                while nxt <= k:
                    g += 1
                    nxt = offsets[g + 1]
            acc += values[k]
        store(g, t, acc)
    assert None not in partials, "a partial slot no chunk wrote"
    # fat buckets: FAT_JOBS jobs of J partials folded into each job's first slot, then
    # the job results (slots base + t J, one thread each) into the first slot
    assert sorted(fat) == [g for g in range(K) if nseg[g] > FAT_PARTIALS]
    for g in fat:
        ns, base = nseg[g], seg_base[g]
        J = fat_job_len(ns)
        assert FAT_JOBS * J >= ns
        for j in range(FAT_JOBS):
            a = j * J
            if a < ns:
                partials[base + a] = sum(partials[base + a:base + min(a + J, ns)])
        partials[base] = sum(partials[base + t * J] for t in range(64) if t * J < ns)
    # k_bucket_sums, over the real buckets
    return [partials[seg_base[g]] if nseg[g] > FAT_PARTIALS else sum(partials[seg_base[g]:seg_base[g] + nseg[g]])
            for g in range(K)], offsets, L


def test_chunk_partials_fold_back_to_each_bucket():
    rng = random.Random(21)
    for trial in range(48):
        K = rng.choice([1, 2, 7, 64, 512, 2048, 3000])
        kind = trial % 4
        if kind == 0:     # uniform
            sizes = [rng.randrange(0, 12) for _ in range(K)]
        elif kind == 1:   # a witness of ones: one bucket holds most entries
            sizes = [rng.randrange(0, 3) for _ in range(K)]
            sizes[rng.randrange(K)] += rng.randrange(2000, 12000)
        elif kind == 2:   # mostly empty
            sizes = [rng.choice([0, 0, 0, 0, 1, 30]) for _ in range(K)]
        else:             # a few giant buckets
            sizes = [rng.choice([0, 0, 0, 1, 3000]) for _ in range(min(K, 64))]
        K = len(sizes)
        if rng.randrange(2):
            sizes.append(rng.randrange(0, 2000))   # the constant-work sink bucket, accumulated, never reduced
        M = sum(sizes)
        if M == 0:
            continue
        values = [rng.randrange(1, 1 << 30) for _ in range(M)]
        floor = rng.choice([4, 16])
        sums, offsets, L = layout_and_sums(sizes, values, K, floor, rng.choice([0, 148 * 512, 148]),
                                           *rng.choice([(1024, 1), (16, 1), (16, 3), (4, 2)]))
        assert L >= floor and (M + L - 1) // L <= ACC_THREADS
        for g in range(K):
            assert sums[g] == sum(values[offsets[g]:offsets[g + 1]]), (trial, g)


def test_every_short_chunk_length_folds_back():
    # 4 to 16 entries a chunk, over buckets that start and end anywhere in one
    rng = random.Random(22)
    for L in range(4, 17):
        sizes = [rng.choice([0, 0, 0, 1, 2, 3, 5, 17, 60]) for _ in range(120)]   # below 4 L a bucket on average
        values = [rng.randrange(1, 1 << 30) for _ in range(sum(sizes))]
        sums, offsets, got = layout_and_sums(sizes, values, len(sizes), L, 0)
        assert got == L
        assert sums == [sum(values[a:b]) for a, b in zip(offsets, offsets[1:])]


def test_min_chunk_cases():
    # down to the floor while the chunks leave SMs without their 512 threads, 16 from there on
    assert [min_chunk(M, 4) for M in (0, 1, 4 * SPREAD_THREADS, 4 * SPREAD_THREADS + 1, 15 * SPREAD_THREADS,
                                      15 * SPREAD_THREADS + 1, 1 << 30)] == [4, 4, 4, 5, 15, 16, 16]
    assert {min_chunk(M, 16) for M in (0, 1, 1 << 18, 1 << 30)} == {16}


CHUNKS_PROBE = r"""
#include <cstdio>
#include "msm.cuh"
int main() {
    unsigned long long m;
    unsigned floor;
    while (scanf("%llu %u", &m, &floor) == 2) printf("%zu\n", g16::msm_max_chunks(m, floor));
    return 0;
}
"""


def test_chunks_never_exceed_what_the_buffers_hold(tmp_path):
    """ceil(M / L) <= msm_max_chunks(max_entries) for every entry count M up to the maximum
    that a call's buffers and its accumulate launch are sized for."""
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not on PATH")
    src, exe = tmp_path / "probe.cu", tmp_path / "probe"
    src.write_text(CHUNKS_PROBE)
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "snarkrs_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-o", str(exe), str(src)], check=True, capture_output=True)
    rng = random.Random(23)
    edges = [k * SPREAD_THREADS + d for k in (1, 2, 3, 4, 5, 8, 15, 16, 17, 20, 32, 33, 48) for d in (-1, 0, 1)]
    Ms = sorted(set([0, 1, 3, 4, 5, 15, 16, 17, 1000, 1 << 20, 1 << 26, (1 << 31) - 1] + edges +
                    [int(1.3 ** rng.uniform(1, 80)) for _ in range(300)]))
    for floor in (4, 16):
        out = subprocess.run([str(exe)], input=" ".join("%d %d" % (m, floor) for m in Ms), capture_output=True,
                             text=True, check=True).stdout.split()
        most, held = 0, list(map(int, out))
        for M, cap in zip(Ms, held):
            assert cap >= most, "a larger maximum never holds fewer chunks"
            for K in (1, 1000, 1 << 13, 1 << 20):
                for wave in (0, 148, SPREAD_THREADS):
                    L = chunk_len(M, K, min_chunk(M, floor), wave)
                    assert L >= floor and (M + L - 1) // L <= cap, (M, K, floor, wave)
                    most = max(most, (M + L - 1) // L)


def test_chunk_len_cases():
    # the device's choice: at least L_min, about M / (4 K) or more, and wave fitting
    # only for a gain of 5% or more
    assert chunk_len(1000, 1 << 16, 16, 0) == 16
    assert chunk_len(1 << 26, 1 << 16, 16, 0) == 256          # M / (4K)
    assert chunk_len(1 << 30, 1 << 20, 16, 0) == 2048         # the thread cap, 2^19 threads
    wave = 148 * 512                                          # one 512-thread block per SM
    M = int(2.4 * wave * 16)                                  # 2.4 waves of 16 lose to 2 waves of 20
    assert chunk_len(M, 1 << 20, 16, wave) == 20
    M = int(2.97 * wave * 16)                                 # 3 waves of 16 against 2 of 24: kept
    assert chunk_len(M, 1 << 20, 16, wave) == 16


GRID_PROBE = r"""
#include <cstdio>
#include "msm.cuh"
int main() {
    unsigned long long k;
    while (scanf("%llu", &k) == 1) {
        const g16::MsmPlanGrid g = g16::msm_plan_grid(k);
        printf("%u %u %u\n", g.tiles, g.per_block, g.blocks);
    }
    return 0;
}
"""


def test_plan_blocks_read_a_bounded_number_of_sums(tmp_path):
    """Every block of the plan kernels adds up all blocks' sums: their number stays at
    4096 however many buckets there are, and the blocks' tiles cover each bucket once."""
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc not on PATH")
    src, exe = tmp_path / "probe.cu", tmp_path / "probe"
    src.write_text(GRID_PROBE)
    subprocess.run(["nvcc", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "snarkrs_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-o", str(exe), str(src)], check=True, capture_output=True)
    ks = [0, 1, 1023, 1024, 1025, 24576, 1 << 22, (1 << 22) + 1, 13 << 19, (13 << 19) + 1, 1 << 25, (1 << 31) - 1]
    out = subprocess.run([str(exe)], input=" ".join(map(str, ks)), capture_output=True, text=True, check=True).stdout
    for k, line in zip(ks, out.splitlines()):
        tiles, per, blocks = map(int, line.split())
        assert tiles == (k + 1023) // 1024 and 1 <= blocks <= 4096
        assert (per == 1) == (tiles <= 4096)
        covered = [t for b in range(blocks) for t in range(b * per, min((b + 1) * per, tiles))]
        assert covered == list(range(tiles))
