"""GPU parity at the sizes where a kernel's work is cut differently: the MSM's
chunks and blocks (1 to a few warps of chunks, the 2^18 scalars where a window's
digits stop being split over warps), bucket reductions whose lane groups meet
equal and opposite points, and the NTT's tilings by transform size.  Results are
group and field elements: equal to the oracle's byte for byte, no tolerance."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S():
    import snarkrs_b200
    return snarkrs_b200


@pytest.fixture(scope="module")
def O():
    import oracle
    oracle.build()
    return oracle


@pytest.fixture(scope="module")
def backend(S):
    b = S.CudaBackend(0)
    yield b
    b.close()


def _tiled(S, group, n, distinct):
    size = 64 if group == 1 else 128
    pts = S.synth_points(group, 5, min(n, distinct))
    return (pts * (n // min(n, distinct) + 1))[:n * size]


@pytest.mark.parametrize("n,dist", [(33, 0), (255, 1), (257, 0), (4099, 0), (40000, 1), ((1 << 18) - 1, 1),
                                    (1 << 18, 1)])
def test_g1_msm_sizes(S, O, backend, n, dist):
    bases, scalars = _tiled(S, 1, n, 1 << 14), S.synth_scalars(n, n, dist)
    assert S.CudaMsm(backend).msm_g1(bases, scalars) == O.msm_g1(bases, scalars)


@pytest.mark.parametrize("n,dist", [(5, 0), (129, 1), (3001, 0), (20011, 1)])
def test_g2_msm_sizes(S, O, backend, n, dist):
    bases, scalars = _tiled(S, 2, n, 1 << 10), S.synth_scalars(n, n, dist)
    assert S.CudaMsm(backend).msm_g2(bases, scalars) == O.msm_g2(bases, scalars)


@pytest.mark.parametrize("group", [1, 2])
def test_equal_and_opposite_partial_sums(S, O, backend, group):
    """One point, n times, with few distinct scalars: partial sums of a bucket and
    neighbouring buckets hold equal points (doublings) and, with r - k beside k,
    cancel to the identity."""
    n, size = 3000, 64 if group == 1 else 128
    bases = S.synth_points(group, 9, 1) * n
    values = [3, S.R_MOD - 3, 3, 1, S.R_MOD - 1, 1 << 200, S.R_MOD - (1 << 200), 0]
    scalars = b"".join(values[i % 8].to_bytes(32, "little") for i in range(n))
    msm = S.CudaMsm(backend)
    run, ref = (msm.msm_g1, O.msm_g1) if group == 1 else (msm.msm_g2, O.msm_g2)
    assert run(bases, scalars) == ref(bases, scalars)
    all_cancel = b"".join(values[i % 2].to_bytes(32, "little") for i in range(n))
    assert run(bases, all_cancel) == bytes(size)


@pytest.mark.parametrize("log_n", [4, 6, 7, 9, 14, 15, 17, 19])
def test_ntt_tilings(S, O, backend, log_n):
    """Sizes on both sides of every step of the default tiling's rule, and the
    transforms that fit one small tile."""
    ntt = S.CudaNtt(backend)
    data = S.synth_scalars(log_n, 1 << log_n, 0)   # below r: valid Montgomery words
    assert ntt.ntt(data) == O.ntt(log_n, O.NTT_FORWARD, data)
    assert ntt.intt_coset_ntt(data) == O.ntt(log_n, O.NTT_INTT_COSET_NTT, data)
    assert ntt.coset_ntt(data, inverse=True) == O.ntt(log_n, O.NTT_COSET_INVERSE, data)


@pytest.mark.parametrize("constant_work", [False, True])
def test_millions_of_buckets(S, O, constant_work):
    """A compact key at 20-bit windows sorts into 13 x 2^19 buckets (one more with constant
    work), past the 2^22 where a block of the plan kernels takes several tiles of them."""
    sc = S.SynthCircuit(seed=31, n_constraints=700, n_inputs=24, n_public=5)
    zk = sc.zkey(32)
    ok = O.Zkey(zk)
    os.environ["G16_CUDA_WINDOW_TABLES"] = "0"
    try:
        b = S.CudaBackend(0, constant_work=constant_work)
        c = b.prepare(S.ProvingKey.from_bytes(zk))
    finally:
        del os.environ["G16_CUDA_WINDOW_TABLES"]
    t = c.tuning()
    c.set_tuning(20, 20, t["ntt_tile_log"], t["ntt_outer_log_l"])
    w, (r, s) = sc.witness(3), [O.to_bytes(O.to_mont(x)) for x in (1234567, 7654321)]
    assert c.prove_with_blinders(w, r, s).to_bytes() == ok.prove(w, O.from_bytes(r), O.from_bytes(s))
    c.close()
    b.close()
    ok.close()


@pytest.mark.parametrize("group", [1, 2])
def test_empty_buckets_cost_little(S, backend, group):
    """A warp of lane groups that only meets identities forms no product: the pieces kernel
    takes a small part of its time on full buckets (with the products, the same time)."""
    n = 1 << (18 if group == 1 else 16)
    bases, msm = _tiled(S, group, n, 1 << 10), S.CudaMsm(backend)
    run = msm.msm_g1 if group == 1 else msm.msm_g2
    ms = {}
    for name, scalars in (("full", S.synth_scalars(3, n, 0)), ("empty", bytes(32 * n))):
        got = run(bases, scalars)
        S.kernel_timing(True)
        S.kernel_timing_reset()
        try:
            assert run(bases, scalars) == got
            ms[name] = S.kernel_timing_report()["msm_reduce"][0]
        finally:
            S.kernel_timing(False)
    assert got == bytes(64 * group)
    assert ms["empty"] < 0.5 * ms["full"], ms
