"""The key planes of the cascade's GEMM steps take 409 MB a key set at degree 2048: a handle that
lacks the memory does without them, and views of one key share them."""
import numpy as np
import pytest

from via_rs_b200.params import paper_preset
from via_rs_b200.server import DeviceError, PublicKeys, Server

pytestmark = pytest.mark.gpu

PLANES = 406_000_000  # bytes, degree 2048 (and 3 MB of constants)
VIA_ERR_OUT_OF_MEMORY = 101


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


def test_reserve_that_does_not_fit(oracle):
    """The handle goes on answering with the workspace it had."""
    import torch

    prm = paper_preset(2, 4)
    c, recs, keys = _setup(oracle, prm)
    q = c.query(5, b"q")
    gpu = Server.setup(prm, keys, recs)
    want = gpu.answer(q)
    filler = torch.empty(_free(torch) - (2 << 30), dtype=torch.uint8, device="cuda")
    with pytest.raises(DeviceError) as e:
        gpu.reserve(4096)
    got = gpu.answer(q)
    gpu.close()
    del filler
    _free(torch)
    assert e.value.code == VIA_ERR_OUT_OF_MEMORY
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


def test_views_share_planes_of_one_key(oracle):
    import torch

    prm = paper_preset(2, 4)
    pv = prm.with_dims(prm.num_rows, prm.num_cols, 256)
    c, recs, keys = _setup(oracle, prm)
    cv, _, vkeys = _setup(oracle, pv)
    co, _, okeys = _setup(oracle, prm, b"other")
    base = Server.setup(prm, keys, recs)
    cells = recs.reshape(prm.n1 // prm.n_rec, -1, prm.n_rec).transpose(1, 2, 0).reshape(-1, prm.n1)
    d = prm.n1 // pv.n_rec
    vrecs = np.concatenate([cells[:, k::d] for k in range(d)])
    free = [_free(torch)]
    view = base.view(256, vkeys)
    free.append(_free(torch))
    other = base.view(prm.n2, okeys)
    free.append(_free(torch))
    assert np.array_equal(c.cascade_key, cv.cascade_key) and not np.array_equal(c.cascade_key, co.cascade_key)
    assert free[0] - free[1] < PLANES < free[1] - free[2]
    base.close()  # what it lent stays
    idx = [1, prm.capacity - 1]
    m, b = view.answer_batch(cv.batch_query(idx, b"v"))
    for t, rec in enumerate(cv.recover_batch(m, b)):
        assert np.array_equal(rec, vrecs[idx[t]])
    q = co.query(7, b"o")
    assert np.array_equal(co.recover(*other.answer(q)), recs[7])
