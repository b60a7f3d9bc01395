"""The cascade's GEMM steps against the oracle where they can go wrong: query words at the
edges of their range, and batches whose LWEs end inside, at and past a 128-LWE tile (with the
last 8-LWE group full and partial)."""
import numpy as np
import pytest

from via_rs_b200.params import paper_preset, secure_preset
from via_rs_b200.server import PublicKeys, Server

pytestmark = pytest.mark.gpu


def _setup(oracle, prm, seed):
    rng = np.random.default_rng(41)
    recs = rng.integers(0, 16, size=(prm.capacity, prm.n_rec), dtype=np.uint64)
    c = oracle.Client(prm, seed)
    gpu = Server.setup(prm, PublicKeys(c.cascade_key, c.conv_key, c.rsk), recs)
    return c, gpu, oracle.Server(prm, c.cascade_key, c.conv_key, c.rsk, recs)


@pytest.mark.parametrize("preset", ["paper", "secure"])
def test_edge_words(oracle, preset):
    prm = {"paper": paper_preset, "secure": secure_preset}[preset](2, 2)
    _, gpu, cpu = _setup(oracle, prm, b"gemm-edge")
    q, Q = prm.q1, prm.q1[0] * prm.q1[1]
    edges = [0, 1, Q - 1, Q // 2, Q // 2 + 1, Q // 18, 17 * (Q // 18)]
    query = np.zeros((prm.n_lwe, prm.lwe_len), dtype=np.uint64)
    rng = np.random.default_rng(42)
    for w in range(prm.n_lwe):
        for l in range(2):
            row = np.array([e % q[l] for e in edges], dtype=np.uint64)
            # whole LWEs of one value, then random mixtures of the edges
            pick = np.full(prm.n1 + 1, w) if w < len(edges) else rng.integers(len(edges), size=prm.n1 + 1)
            pick = rng.permutation(pick) if l == 0 else pick
            query[w, l * prm.n1:(l + 1) * prm.n1] = row[pick[:-1]]
            query[w, 2 * prm.n1 + l] = row[pick[-1]]
    assert np.array_equal(gpu.debug_stage(query.reshape(-1), 1), cpu.debug_stage(query.reshape(-1), 1))


@pytest.mark.parametrize("count", [2, 15, 16, 17, 33])
def test_tiles(oracle, count):
    """8 LWEs a query: 16, 120, 128, 136 and 264 LWEs a cascade."""
    prm = paper_preset(2, 2, 512)
    assert prm.n_lwe == 8
    c, gpu, cpu = _setup(oracle, prm, b"gemm-tiles")
    rng = np.random.default_rng(count)
    idx = rng.integers(prm.capacity, size=count)
    qs = np.stack([c.query(int(i), b"t-%03d" % k) for k, i in enumerate(idx)])
    masks, bodies = gpu.answer_many(qs)
    for k in {0, 1, count // 2, count - 2, count - 1}:
        m, b = cpu.answer(qs[k])
        assert np.array_equal(masks[k], m) and np.array_equal(bodies[k], b), k


@pytest.mark.parametrize("base,depth", [(32, 15), (21, 18), (300, 9)])
def test_other_gadgets(oracle, base, depth):
    """Gadgets the GEMM steps do not serve (depth, B^6 above 2^26, digits beyond a byte) keep the
    transform path for every step."""
    import dataclasses

    prm = dataclasses.replace(paper_preset(2, 2), ck_base=base, l_ck=depth)
    c, gpu, cpu = _setup(oracle, prm, b"gemm-other")
    q = c.query(3, b"other")
    assert np.array_equal(gpu.debug_stage(q, 2), cpu.debug_stage(q, 2))


def test_query_count_edges(oracle):
    """Two LWEs a thread in the late steps' multiply-accumulate: an odd number of LWEs."""
    prm = paper_preset(2, 2)
    c, gpu, cpu = _setup(oracle, prm, b"gemm-odd")
    # 41 queries x 2 LWEs (DMux group) and x 6 (the rest): both groups past the rule's line.
    qs = np.stack([c.query(k % prm.capacity, b"o-%03d" % k) for k in range(41)])
    masks, bodies = gpu.answer_many(qs)
    for k in (0, 20, 40):
        m, b = cpu.answer(qs[k])
        assert np.array_equal(masks[k], m) and np.array_equal(bodies[k], b), k
