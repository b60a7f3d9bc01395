"""The fused gadget products (shared key, and RGSWs of their own) against the oracle over the ring
degrees they are instantiated for and the ones just outside, with the counts at the line to
separate kernels (512 CTAs); outputs in place of an input take the general path. DMux trees
whose levels lie on both sides of the line between a cluster a product and one CTA."""
import numpy as np
import pytest

from via_rs_b200 import prims
from via_rs_b200.params import PAPER_Q1, PAPER_Q2, SECURE_Q1, paper_preset, secure_preset
from via_rs_b200.server import PublicKeys, Server

pytestmark = pytest.mark.gpu


def _rand(rng, q, n, count):
    return np.stack([rng.integers(0, p, size=(count, n), dtype=np.uint64) for p in q], axis=1)


def _dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()


@pytest.mark.parametrize("q,n,base,L", [(PAPER_Q1, 128, 18, 3), (PAPER_Q1, 256, 55879, 2), (PAPER_Q1, 512, 18, 4),
                                        (PAPER_Q1, 1024, 7, 1), ((PAPER_Q2,), 2048, 307, 2),
                                        (SECURE_Q1, 4096, 18073, 2)])
@pytest.mark.parametrize("in_place", [False, True])
def test_external_products(oracle, q, n, base, L, in_place):
    import torch

    rng = np.random.default_rng(n)
    count = 5
    rgsw = _rand(rng, q, n, count * 4 * L)
    ct = _rand(rng, q, n, count * 2)
    ct[1] = np.array(q, dtype=np.uint64)[:, None] - 1
    rgsw[:4 * L] = np.array(q, dtype=np.uint64)[:, None] - 1
    want = oracle.external_product(q, n, base, L, rgsw.reshape(-1), ct.reshape(-1))
    d_rgsw, d_ct = _dev(torch, rgsw), _dev(torch, ct)
    out = d_ct if in_place else torch.empty_like(d_ct)
    prims.external_product_dev(prims.ring(n, q), base, L, d_rgsw.data_ptr(), d_ct.data_ptr(), count, out.data_ptr())
    assert np.array_equal(out.cpu().numpy().view(np.uint64).reshape(-1), want)


@pytest.mark.parametrize("q,n,count", [(PAPER_Q1, 128, 3), (PAPER_Q1, 256, 3), (PAPER_Q1, 512, 3), (PAPER_Q1, 1024, 3),
                                       (PAPER_Q1, 2048, 255), (PAPER_Q1, 2048, 256), (SECURE_Q1, 4096, 2),
                                       (SECURE_Q1, 4096, 256)])
def test_key_switches(oracle, q, n, count):
    import torch

    rng = np.random.default_rng(n + count)
    base = L = 18
    key = _rand(rng, q, n, L * 2)
    key[:2] = np.array(q, dtype=np.uint64)[:, None] - 1
    ct = _rand(rng, q, n, count * 2)
    shifts = rng.integers(0, 3 * n, size=count, dtype=np.uint64)
    out = torch.empty((count * 2, len(q), n), dtype=torch.int64, device="cuda")
    d = [_dev(torch, x) for x in (key, ct, shifts)]
    prims.key_switch_dev(prims.ring(n, q), base, L, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), count,
                         out.data_ptr())
    want = oracle.key_switch(q, n, base, L, key.reshape(-1), ct.reshape(-1), shifts)
    assert np.array_equal(out.cpu().numpy().view(np.uint64).reshape(-1), want)


@pytest.mark.parametrize("preset,rows", [("paper", 128), ("secure", 64)])
def test_dmux_levels(oracle, preset, rows):
    prm = {"paper": paper_preset, "secure": secure_preset}[preset](rows, 2)
    c = oracle.Client(prm, b"dmux-levels")
    recs = np.random.default_rng(7).integers(0, 16, size=(prm.capacity, prm.n_rec), dtype=np.uint64)
    gpu = Server.setup(prm, PublicKeys(c.cascade_key, c.conv_key, c.rsk), recs)
    cpu = oracle.Server(prm, c.cascade_key, c.conv_key, c.rsk, recs)
    q = c.query(prm.capacity - 1, b"q")
    assert np.array_equal(gpu.debug_stage(q, 3), cpu.debug_stage(q, 3))
