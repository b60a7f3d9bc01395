"""Caller words that are not canonical residues are taken mod their prime: the results are
compared with the oracle's on the reduced words, at values where double-precision integers
(2^52, 2^53) and the transforms' bounds (2^47) end."""
import numpy as np
import pytest

from via_rs_b200.params import paper_preset, secure_preset
from via_rs_b200.server import PublicKeys, Server

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 1 << 44, (1 << 47) - 1, 1 << 47, (1 << 51) - 1, 1 << 51, (1 << 52) - 1, 1 << 52, (1 << 53) + 1,
         (1 << 60) + 7, (1 << 63) + 5, (1 << 64) - 1]


def _words(rng, q, shape):
    """A third canonical residues, the others edge words or any word."""
    w = rng.integers(0, q, size=shape, dtype=np.uint64)
    edge = np.array(EDGES + [q - 1, q, q + 1, 2 * q - 1, 2 * q], dtype=np.uint64)
    pick = rng.integers(3, size=shape)
    w = np.where(pick == 1, rng.choice(edge, size=shape), w)
    return np.where(pick == 2, rng.integers(0, 1 << 64, size=shape, dtype=np.uint64), w)


@pytest.mark.parametrize("part", ["body", "mask"])
@pytest.mark.parametrize("preset", ["paper", "secure"])
def test_query_words(oracle, preset, part):
    prm = {"paper": paper_preset, "secure": secure_preset}[preset](2, 2)
    recs = np.zeros((prm.capacity, prm.n_rec), dtype=np.uint64)
    c = oracle.Client(prm, b"raw-query")
    gpu = Server.setup(prm, PublicKeys(c.cascade_key, c.conv_key, c.rsk), recs)
    cpu = oracle.Server(prm, c.cascade_key, c.conv_key, c.rsk, recs)
    rng = np.random.default_rng(61)
    raw = c.query(1, b"raw").reshape(prm.n_lwe, prm.lwe_len).copy()
    at = slice(prm.nl * prm.n1, None) if part == "body" else slice(0, prm.nl * prm.n1)
    primes = np.array(prm.q1, dtype=np.uint64).repeat(1 if part == "body" else prm.n1)
    if part == "body":  # every edge in turn
        raw[:, at] = np.array((EDGES * 8)[:raw[:, at].size], dtype=np.uint64).reshape(raw[:, at].shape)
        raw[0, at] = np.array(prm.q1, dtype=np.uint64)
    else:
        for w in range(prm.n_lwe):
            raw[w, at] = np.concatenate([_words(rng, q, prm.n1) for q in prm.q1])
    red = raw.copy()
    red[:, at] %= primes
    assert np.array_equal(gpu.debug_stage(raw.reshape(-1), 1), cpu.debug_stage(red.reshape(-1), 1))
