"""Servers on rings below the presets' degrees, against the oracle: the degrees around the least the
cascade's GEMM steps serve, and those whose cascade body is assembled by kernels of its own."""
import dataclasses

import numpy as np
import pytest

from via_rs_b200.params import paper_preset
from via_rs_b200.server import PublicKeys, Server

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1", [128, 256, 512, 1024])
@pytest.mark.parametrize("queries", [1, 17])  # 17: more than one tile of 128 LWEs
def test_cascade_and_answers(oracle, n1, queries):
    prm = paper_preset(2, 2)
    prm = dataclasses.replace(prm, n1=n1, n2=min(n1, prm.n2), n_rec=min(n1, prm.n_rec) // 2)
    recs = np.random.default_rng(n1).integers(0, 16, size=(prm.capacity, prm.n_rec), dtype=np.uint64)
    c = oracle.Client(prm, b"small-%d" % n1)
    gpu = Server.setup(prm, PublicKeys(c.cascade_key, c.conv_key, c.rsk), recs)
    cpu = oracle.Server(prm, c.cascade_key, c.conv_key, c.rsk, recs)
    qs = np.stack([c.query(k % prm.capacity, b"s-%02d" % k) for k in range(queries)])
    if queries == 1:
        assert np.array_equal(gpu.debug_stage(qs[0], 1), cpu.debug_stage(qs[0], 1))
    masks, bodies = gpu.answer_many(qs)
    for k in {0, queries - 1}:
        m, b = cpu.answer(qs[k])
        assert np.array_equal(masks[k], m) and np.array_equal(bodies[k], b), k


@pytest.mark.parametrize("base", [482, 509])  # the last gadget the fused CMux takes at this prime's size, and one past it
def test_cmux_gadgets_at_the_scaling_line(oracle, base):
    prm = dataclasses.replace(paper_preset(2, 8), q2=34_347_294_721, b_cmux=base)
    recs = np.random.default_rng(base).integers(0, 16, size=(prm.capacity, prm.n_rec), dtype=np.uint64)
    c = oracle.Client(prm, b"line-%d" % base)
    gpu = Server.setup(prm, PublicKeys(c.cascade_key, c.conv_key, c.rsk), recs)
    cpu = oracle.Server(prm, c.cascade_key, c.conv_key, c.rsk, recs)
    q = c.query(prm.capacity - 1, b"q")
    got, want = gpu.answer(q), cpu.answer(q)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
