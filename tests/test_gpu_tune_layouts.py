"""Scan tiles measured for one output layout are not read back for the other: two servers that differ
only in the CMux gadget (one the fused CMux takes tiles for, one not) share a cache file."""
import dataclasses

import numpy as np
import pytest

from via_rs_b200.params import paper_preset
from via_rs_b200.server import PublicKeys, Server

pytestmark = pytest.mark.gpu


def test_cache_keeps_layouts_apart(tmp_path):
    path = str(tmp_path / "tiles")
    prm = paper_preset(4, 64)
    measured = []
    for base in (prm.b_cmux, 1000, prm.b_cmux, 1000):  # 81: tiles; 1000: past the small gadgets
        p = dataclasses.replace(prm, b_cmux=base)
        keys = PublicKeys(np.zeros(p.cascade_key_len), np.zeros(p.conv_key_len), np.zeros(p.rsk_len))
        server = Server.setup(p, keys, np.zeros((p.capacity, p.n_rec), dtype=np.uint64))
        measured.append(server.autotune([8], path)[0]["candidates"])
        server.close()
    assert measured[0] > 0 and measured[1] > 0 and measured[2:] == [0, 0], measured
