"""Device-memory budgets.  The short accumulate chunks that spread a small MSM over
the SMs take more scratch (up to 58 MB a proof); a budget that holds a key with the
ordinary chunks of 16 entries still does, and its proofs are the same."""
import random

import pytest

import oracle as O
import snarkrs_b200 as S


def _key(constraints):
    sc = S.SynthCircuit(seed=901, n_constraints=constraints, n_inputs=24, n_public=5)
    return sc, sc.zkey(902)


# the compact key with one workspace whose buffers hold one partial sum per 16 entries
@pytest.mark.parametrize("constraints,held", [(500, 22826468), (2000, 28253804), (8000, 55056932),
                                              (20000, 108306692)])
def test_short_chunks_do_not_refuse_a_key(constraints, held):
    pk = S.ProvingKey.from_bytes(_key(constraints)[1], check_points=False)
    pk.plan(held)


@pytest.mark.gpu
@pytest.mark.parametrize("tables", [True, False], ids=["tables", "compact"])
def test_proofs_within_the_least_budget_equal_the_oracle(tables):
    sc, zk = _key(3000)
    pk, ok = S.ProvingKey.from_bytes(zk), O.Zkey(zk)
    full = pk.plan(1 << 40)
    limit = full["key_bytes"] + full["workspace_bytes"]
    b = S.CudaBackend(0, vram_limit=limit if tables else limit - 1)
    c = b.prepare(pk)
    assert bool(c.window_tables()) == tables
    held, rng = c.device_bytes(), random.Random(5)
    for k in range(3):   # the third proof replays a captured graph
        w = sc.witness(k)
        r, s = (O.to_bytes(O.to_mont(rng.randrange(1, O.R_MOD))) for _ in range(2))
        assert c.prove_with_blinders(w, r, s).to_bytes() == ok.prove(w, O.from_bytes(r), O.from_bytes(s))
    assert c.device_bytes() - held == (full if tables else pk.plan(limit - 1))["workspace_bytes"]   # one workspace
    c.close()
    b.close()
    ok.close()


@pytest.mark.gpu
def test_short_chunks_do_not_refuse_a_batch(backend):
    """One engine's working set with chunks of 16 entries: what the reservation of an
    unlimited backend counts, less the short chunks' 75776 partial sums in each space."""
    sc, zk = _key(3000)
    pk, n = S.ProvingKey.from_bytes(zk), 12
    circ = backend.prepare(pk)
    engines = 4
    sized = S.CudaBackend(0)
    c = sized.prepare(pk)
    key = sized.vram_used()
    sized.batch_reserve([c] * n)
    need = (sized.vram_used() - key) // engines - 75776 * (2 * 128 + 256)
    c.close()
    sized.close()
    b = S.CudaBackend(0, vram_limit=key + engines * need)
    c = b.prepare(pk)
    b.batch_reserve([c] * n)
    rng = random.Random(6)
    jobs = [(sc.witness(k),) + tuple(O.to_bytes(O.to_mont(rng.randrange(1, O.R_MOD))) for _ in range(2))
            for k in range(n)]
    want = [circ.prove_with_blinders(*j) for j in jobs]
    allocs = S.device_alloc_count()
    for _ in range(3):   # laid out, captured, replayed
        assert b.prove_batch([(c,) + j for j in jobs]) == want
    assert S.device_alloc_count() == allocs
    c.close()
    b.close()
    circ.close()


@pytest.mark.gpu
def test_an_engine_with_room_keeps_short_chunks(backend):
    """An engine that holds enough for a larger mix with chunks of 16 entries still grows to
    its short chunks' scratch where the budget has room, and then holds it."""
    sc, zk = _key(3000)
    b = S.CudaBackend(0)
    c = b.prepare(S.ProvingKey.from_bytes(zk))
    one = S.fr_to_mont_bytes(1)
    job, used = (c, sc.witness(1), one, one), []
    for n in (4, 5, 5):   # a job's share is below the short chunks' 39 MB
        b.prove_batch([job] * n)
        used.append(b.vram_used())
    assert used[0] < used[1] == used[2]
    c.close()
    b.close()
