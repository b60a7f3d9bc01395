"""The parallel rejection walk of wire ingest and the device client against Shake256Prg and
the oracle's client, where it can go wrong: primes that reject a third of the draws (several
chunks of candidates a mask), a mask of exactly one chunk, masks below one thread's share,
one-limb rings, and limbs whose draws take different numbers of bytes (the general walk)."""
import dataclasses

import numpy as np
import pytest

from via_rs_b200.client import Client
from via_rs_b200.params import n8_preset, paper_preset, secure_preset, toy_preset
from via_rs_b200.prg import Shake256Prg
from via_rs_b200.server import PublicKeys, Server
from via_rs_b200.wire import from_wire, prg_packet

pytestmark = pytest.mark.gpu

PRESETS = {
    "paper": lambda: paper_preset(1, 4),  # 4096 draws: one chunk
    "secure": lambda: secure_preset(1, 2),  # acceptance 0.63: several chunks
    "toy": lambda: toy_preset(1, 2),  # one limb, acceptance 0.5, 64 draws
    "n8": lambda: n8_preset(1, 2),  # 8 draws
}


@pytest.mark.parametrize("preset", sorted(PRESETS))
def test_wire_masks(preset):
    prm = PRESETS[preset]()
    rng = np.random.default_rng(31)
    keys = PublicKeys(np.zeros(prm.cascade_key_len), np.zeros(prm.conv_key_len), np.zeros(prm.rsk_len))
    server = Server.setup(prm, keys, np.zeros((prm.capacity, prm.n_rec), dtype=np.uint64))
    packets, want = [], []
    for _ in range(prm.n_lwe):
        seed = rng.bytes(32)
        body = rng.integers(0, min(prm.q1), size=prm.nl, dtype=np.uint64)
        prg = Shake256Prg(seed)
        mask = np.array([[prg.uniform_below(q) for q in prm.q1] for _ in range(prm.n1)], dtype=np.uint64)
        packets.append(prg_packet(seed, body))
        want.append(np.concatenate([mask.T.reshape(-1), body]))
    assert np.array_equal(from_wire(server, b"".join(packets)), np.concatenate(want))


@pytest.mark.parametrize("err", [(0, 0), (1, 5), (1, 1 << 20)])
@pytest.mark.parametrize("preset", ["paper", "secure", "mixed_widths"])
def test_client_masks_and_errors(preset, err):
    """The stream of a query: every LWE's mask, then its error's draws, back to back."""
    if preset == "mixed_widths":  # a 37-bit and a 41-bit limb: five and six bytes a draw
        prm = dataclasses.replace(paper_preset(1, 4), q1=(paper_preset().q1[0], 1099511799809))
    else:
        prm = PRESETS[preset]()
    kind, bound = err
    rng = np.random.default_rng(32)
    sk1 = np.concatenate([rng.integers(0, 2, size=prm.n1, dtype=np.uint64) for _ in prm.q1])
    sk2 = rng.integers(0, 2, size=prm.n2, dtype=np.uint64)
    client = Client(prm, sk1, sk2, kind, bound)
    seed = b"walk-%d-%d" % err
    got = client.query(0, seed).reshape(prm.n_lwe, prm.lwe_len)  # index 0: every message is zero
    prg = Shake256Prg(seed)
    for j in range(prm.n_lwe):
        mask = np.array([[prg.uniform_below(q) for q in prm.q1] for _ in range(prm.n1)], dtype=object)
        r = prg.uniform_below(3 if kind == 0 else 2 * bound + 1)
        e = (0, 1, -1)[r] if kind == 0 else r - bound
        for l, q in enumerate(prm.q1):
            assert np.array_equal(got[j, l * prm.n1:(l + 1) * prm.n1], mask[:, l].astype(np.uint64)), (j, l)
            s = sk1[l * prm.n1:(l + 1) * prm.n1].astype(object)
            assert int(got[j, prm.nl * prm.n1 + l]) == (int((mask[:, l] * s).sum()) + e) % q, (j, l)


@pytest.mark.parametrize("wide", [False, True])
def test_recover_sums(oracle, wide):
    """64-bit and 128-bit sums of the recovery (the latter for words above 32 bits)."""
    prm = paper_preset(2, 2)
    if wide:
        prm = dataclasses.replace(prm, q3=PRESETS["paper"]().q1[0])
    oc = oracle.Client(prm, b"recover-sums")
    client = Client(prm, *oc.secret_keys())
    rng = np.random.default_rng(33)
    masks = rng.integers(0, prm.q3, size=(3, prm.n2), dtype=np.uint64)
    masks[0] = prm.q3 - 1
    bodies = rng.integers(0, prm.q4, size=(3, prm.n2), dtype=np.uint64)
    got = client.recover_many(masks, bodies)
    for k in range(3):
        assert np.array_equal(got[k], oc.recover(masks[k], bodies[k]))
