"""Caller words that are not canonical residues are taken mod their prime: the results are
compared with the oracle's on the reduced words, at values where double-precision integers
(2^52, 2^53) and the transforms' bounds (2^47) end."""
import dataclasses

import numpy as np
import pytest

from via_rs_b200 import prims
from via_rs_b200.client import Client
from via_rs_b200.params import PAPER_Q1, PAPER_Q2, PAPER_Q3, SECURE_Q1, paper_preset, secure_preset, toy_preset
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


def _raw(rng, primes, polys, n):
    """Raw words [polys][nl][n] and the same words reduced."""
    raw = np.stack([_words(rng, q, (polys, n)) for q in primes], axis=1)
    return raw, raw % np.array(primes, dtype=np.uint64)[:, None]


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()


def _host(t):
    return t.cpu().numpy().view(np.uint64).reshape(-1)


PRESETS = {
    "paper": lambda: paper_preset(2, 2),
    "secure": lambda: secure_preset(2, 2),
    # Key gadgets without GEMM steps: byte digits, 64-bit digits.
    "bytes": lambda: dataclasses.replace(paper_preset(2, 2), ck_base=21, l_ck=18),
    "words": lambda: dataclasses.replace(paper_preset(2, 2), ck_base=300, l_ck=9),
    "wide": lambda: dataclasses.replace(paper_preset(2, 2), q1=(35184371884033, 35184371703809)),  # integer transforms
    "toy": lambda: toy_preset(2, 2),  # no transforms
    "degree_512": lambda: dataclasses.replace(paper_preset(2, 2), n1=512),  # its body has kernels of its own
}


@pytest.mark.parametrize("part", ["body", "mask"])
@pytest.mark.parametrize("preset", sorted(PRESETS))
def test_query_words(oracle, preset, part):
    prm = PRESETS[preset]()
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


@pytest.mark.parametrize("primes,n,base,L,count", [(PAPER_Q1, 256, 55879, 2, 3), (PAPER_Q1, 2048, 55879, 2, 3),
                                                   ((PAPER_Q2,), 2048, 81, 2, 3), (SECURE_Q1, 4096, 18073, 2, 32)])
@pytest.mark.parametrize("in_place", [False, True])
def test_external_product_words(oracle, primes, n, base, L, count, in_place):
    import torch

    rng = np.random.default_rng(62)
    rgsw, rgsw_red = _raw(rng, primes, count * 4 * L, n)
    ct, ct_red = _raw(rng, primes, count * 2, n)
    d_rgsw, d_ct = _dev(torch, rgsw), _dev(torch, ct)
    out = d_ct if in_place else torch.empty_like(d_ct)
    prims.external_product_dev(prims.ring(n, primes), base, L, d_rgsw.data_ptr(), d_ct.data_ptr(), count, out.data_ptr())
    want = oracle.external_product(primes, n, base, L, rgsw_red.reshape(-1), ct_red.reshape(-1))
    assert np.array_equal(_host(out), want)


@pytest.mark.parametrize("n,count", [(16, 3), (256, 3), (2048, 2), (2048, 256)])
def test_key_switch_mask_words(oracle, n, count):
    import torch

    rng = np.random.default_rng(63)
    base = L = 18
    key, key_red = _raw(rng, PAPER_Q1, L * 2, n)
    ct, ct_red = _raw(rng, PAPER_Q1, count * 2, n)
    ct[1::2] = ct_red[1::2]  # bodies: residues
    shifts = rng.integers(0, 2 * n, size=count, dtype=np.uint64)
    d = [_dev(torch, x) for x in (key, ct, shifts)]
    out = torch.empty((count * 2, 2, n), dtype=torch.int64, device="cuda")
    prims.key_switch_dev(prims.ring(n, PAPER_Q1), base, L, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), count,
                         out.data_ptr())
    want = oracle.key_switch(PAPER_Q1, n, base, L, key_red.reshape(-1), ct_red.reshape(-1), shifts)
    assert np.array_equal(_host(out), want)


# A prime of each of the inverse's schedules: up to 2^35, up to 2^40, below 2^44.
@pytest.mark.parametrize("primes,n", [((PAPER_Q2,), 2048), ((PAPER_Q3,), 512), (PAPER_Q1, 2048), (PAPER_Q1, 64),
                                      (SECURE_Q1, 4096), ((17_592_186_028_033,), 4096)])
@pytest.mark.parametrize("inverse", [False, True])
def test_transform_words(oracle, primes, n, inverse):
    import torch

    rng = np.random.default_rng(64)
    blocks = n.bit_length() - 1
    count = 5 + blocks
    raw, _ = _raw(rng, primes, count, n)
    # Where an inverse grows most: 2^b equal words, then 2^b zeros, so that the words add up for b
    # stages and the next one takes the difference.
    for b in range(blocks):
        raw[b] = np.where(np.arange(n) >> b & 1, 0, (1 << 47) - 1).astype(np.uint64)
    red = raw % np.array(primes, dtype=np.uint64)[:, None]
    ring, d = prims.ring(n, primes), _dev(torch, raw)
    if not inverse:
        prims.ntt_forward_dev(ring, d.data_ptr(), count)
        assert np.array_equal(_host(d), oracle.ntt(primes, n, red).reshape(-1))
    else:  # canonical coefficients whose transform is the reduced input
        prims.ntt_inverse_dev(ring, d.data_ptr(), count)
        got = d.cpu().numpy().view(np.uint64).reshape(red.shape)
        assert (got < np.array(primes, dtype=np.uint64)[:, None]).all()
        assert np.array_equal(oracle.ntt(primes, n, got).reshape(-1), red.reshape(-1))


@pytest.mark.parametrize("below", [1 << 64, 1 << 33, 1 << 32])
def test_client_key_words(oracle, below):
    """Recovery with a key of words up to `below`, and the same residues."""
    prm = paper_preset(2, 2)
    oc = oracle.Client(prm, b"raw-key")
    sk1, sk2 = oc.secret_keys()
    rng = np.random.default_rng(65)
    lifts = rng.integers(0, below // prm.q3 - 1, size=prm.n2, dtype=np.uint64)
    raw = sk2 + lifts * np.uint64(prm.q3)
    assert np.array_equal(raw % np.uint64(prm.q3), sk2)
    assert below < 1 << 64 or int(np.bitwise_or.reduce(raw)) == below - 1  # an or that leaves no word above it
    client = Client(prm, sk1, raw)
    masks = rng.integers(0, prm.q3, size=(3, prm.n2), dtype=np.uint64)
    masks[0] = prm.q3 - 1
    bodies = rng.integers(0, prm.q4, size=(3, prm.n2), dtype=np.uint64)
    got = client.recover_many(masks, bodies)
    for k in range(3):
        assert np.array_equal(got[k], oc.recover(masks[k], bodies[k]))
