"""The scan's tiled columns and the CMux level that gathers them, at the edges of the rule that
chooses them (first levels of 64 and 65+ CMuxes) and of the column tiles: fewer columns than a
tile, exactly one, two; batches inside one c-tile and over several; both ring degrees. Answers
of a batch equal the oracle's and the single-query answers."""
import numpy as np
import pytest

from via_rs_b200.params import paper_preset, secure_preset
from via_rs_b200.server import PublicKeys, Server

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset,cols,batch", [("paper", 128, 1), ("paper", 256, 1), ("paper", 2, 65), ("paper", 64, 3),
                                               ("paper", 128, 25), ("secure", 64, 3), ("secure", 256, 1)])
def test_answers(oracle, preset, cols, batch):
    prm = {"paper": paper_preset, "secure": secure_preset}[preset](2, cols)
    rng = np.random.default_rng(cols + batch)
    recs = rng.integers(0, 16, size=(prm.capacity, prm.n_rec), dtype=np.uint64)
    c = oracle.Client(prm, b"tiled")
    gpu = Server.setup(prm, PublicKeys(c.cascade_key, c.conv_key, c.rsk), recs)
    cpu = oracle.Server(prm, c.cascade_key, c.conv_key, c.rsk, recs)
    idx = [int(i) for i in rng.integers(prm.capacity, size=batch)]
    idx[-1] = prm.capacity - 1
    qs = np.stack([c.query(i, b"t-%03d" % k) for k, i in enumerate(idx)])
    masks, bodies = gpu.answer_many(qs) if batch > 1 else [x[None] for x in gpu.answer(qs[0])]
    for k in {0, batch // 2, batch - 1}:
        m, b = cpu.answer(qs[k])
        assert np.array_equal(masks[k], m) and np.array_equal(bodies[k], b), k
        assert np.array_equal(c.recover(masks[k], bodies[k]), recs[idx[k]])
