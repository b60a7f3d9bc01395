"""Every synchronous answer reports a bounded device wait that ran out. The waits are made to run
out by via_server_set_scan_fault (a barrier nothing completes, for a few milliseconds): the
kernels give up, set the handle's error word and return, and the handle answers again once the
hook is off."""
import numpy as np
import pytest

from via_rs_b200.params import paper_preset
from via_rs_b200.server import DeviceError, PublicKeys, Server
from via_rs_b200.wire import answer_wire, prg_packet

pytestmark = pytest.mark.gpu

VIA_ERR_TIMEOUT = 103


def _setup(oracle, prm):
    recs = np.random.default_rng(71).integers(0, 16, size=(prm.capacity, prm.n_rec), dtype=np.uint64)
    c = oracle.Client(prm, b"wait-limits")
    gpu = Server.setup(prm, PublicKeys(c.cascade_key, c.conv_key, c.rsk), recs)
    return c, gpu, oracle.Server(prm, c.cascade_key, c.conv_key, c.rsk, recs)


def _times_out(call):
    with pytest.raises(DeviceError) as e:
        call()
    assert e.value.code == VIA_ERR_TIMEOUT and "bounded device wait" in str(e.value)


def test_wire_answer_reports_the_wait(oracle):
    prm = paper_preset(4, 8)
    _, gpu, _ = _setup(oracle, prm)
    rng = np.random.default_rng(72)
    wire = b"".join(prg_packet(rng.bytes(32), rng.integers(0, min(prm.q1), size=prm.nl, dtype=np.uint64))
                    for _ in range(prm.n_lwe))
    want = answer_wire(gpu, wire)
    gpu.set_scan_fault(2000)
    _times_out(lambda: answer_wire(gpu, wire))
    gpu.set_scan_fault(0)
    got = answer_wire(gpu, wire)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


def test_batched_scan_reports_the_wait(oracle):
    import torch

    prm = paper_preset(4, 8)
    _, gpu, _ = _setup(oracle, prm)
    sel = torch.zeros(2 * prm.num_rows * 2 * prm.n1, dtype=torch.int64, device="cuda")
    out = torch.empty(2 * prm.num_cols * 2 * prm.n1, dtype=torch.int64, device="cuda")
    gpu.set_scan_fault(2000)
    _times_out(lambda: gpu.scan_many_dev(sel.data_ptr(), 2, out.data_ptr()))
    gpu.set_scan_fault(0)
    gpu.scan_many_dev(sel.data_ptr(), 2, out.data_ptr())
    assert not out.any()


@pytest.mark.parametrize("queries", [1, 17])  # 8 and 136 LWEs: part of one tile, two tiles
def test_cascade_wait_runs_out_and_handle_recovers(oracle, queries):
    prm = paper_preset(2, 2, 512)
    c, gpu, cpu = _setup(oracle, prm)
    qs = np.stack([c.query(k % prm.capacity, b"w-%02d" % k) for k in range(queries)])
    gpu.set_scan_fault(2000)
    with pytest.raises(DeviceError) as e:
        gpu.debug_stage(qs[0], 1)  # the cascade alone
    flag = int(str(e.value).split("flag ")[1].rstrip(")"))
    assert e.value.code == VIA_ERR_TIMEOUT and flag & 64 and not flag & 15, flag
    _times_out(lambda: gpu.answer_many(qs))
    gpu.set_scan_fault(0)
    assert np.array_equal(gpu.debug_stage(qs[0], 1), cpu.debug_stage(qs[0], 1))
    masks, bodies = gpu.answer_many(qs)
    for k in (0, queries - 1):
        m, b = cpu.answer(qs[k])
        assert np.array_equal(masks[k], m) and np.array_equal(bodies[k], b), k
