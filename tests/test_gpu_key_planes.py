"""The key planes of the cascade's GEMM steps take 409 MB a key set at degree 2048: a handle that
lacks the memory does without them."""
import numpy as np
import pytest

from via_rs_b200.params import paper_preset
from via_rs_b200.server import PublicKeys, Server

pytestmark = pytest.mark.gpu

PLANES = 406 << 20  # bytes, degree 2048


def _setup(oracle, prm, seed=b"key-planes"):
    recs = np.random.default_rng(81).integers(0, 16, size=(prm.capacity, prm.n_rec), dtype=np.uint64)
    c = oracle.Client(prm, seed)
    return c, recs, PublicKeys(c.cascade_key, c.conv_key, c.rsk)


def _free(torch):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("short", [250 << 20, 50 << 20])  # short of the planes; of the workspace after them
def test_setup_without_room_for_the_planes(oracle, short):
    import torch

    prm = paper_preset(2, 4)
    c, recs, keys = _setup(oracle, prm)
    q = c.query(5, b"q")
    want = oracle.Server(prm, c.cascade_key, c.conv_key, c.rsk, recs).answer(q)
    gpu = Server.setup(prm, keys, recs)
    gpu.answer(q)
    gpu.close()
    before = _free(torch)
    gpu = Server.setup(prm, keys, recs)
    used = before - _free(torch)
    gpu.close()
    assert used > PLANES
    filler = torch.empty(_free(torch) - (used - short), dtype=torch.uint8, device="cuda")
    gpu = Server.setup(prm, keys, recs)
    m, b = gpu.answer(q)
    gpu.close()
    del filler
    _free(torch)
    assert np.array_equal(m, want[0]) and np.array_equal(b, want[1])


def test_reserve_without_room_beside_the_planes(oracle):
    import torch

    prm = paper_preset(2, 4)
    c, recs, keys = _setup(oracle, prm)
    gpu = Server.setup(prm, keys, recs)
    qs = np.stack([c.query(k % prm.capacity, b"r-%02d" % k) for k in range(64)])
    before = _free(torch)
    gpu.reserve(64)
    used = before - _free(torch)
    want = gpu.answer_many(qs)
    gpu.close()
    gpu = Server.setup(prm, keys, recs)
    filler = torch.empty(_free(torch) - (used - (250 << 20)), dtype=torch.uint8, device="cuda")
    gpu.reserve(64)
    got = gpu.answer_many(qs)
    gpu.close()
    del filler
    _free(torch)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
