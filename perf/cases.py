"""The work a user has this framework do, as measured cases.

A case is a dict: `op` names the public entry point, the rest are its sizes.

    answer        Server.answer, one query in host memory (the server's request path)
    answer_wire   wire.answer_wire, one PrgCompressed wire query in host memory
    answer_many   via_server_answer_many_dev, a batch of queries in HBM, one database scan
    answer_batch  Server.answer_batch (VIA-B), T = n2 / n_rec queries, one packed answer
    client        Client.queries_dev and Client.recover_many (load generation)
    ntt           prims.ntt_forward_dev on one batch, prims.ntt_inverse_dev on another
    external      prims.external_product_dev
    key_switch    prims.key_switch_dev

Server cases run the paper preset (n1 = 2048) or the secure preset (n1 = 4096) on a
rows x cols grid of seeded 4-bit records. Queries come from the device client with seeded
ternary secrets at seeded indices; key residues, ciphertexts and RGSWs are uniform, which
is what encryptions look like to a server. All outputs are residues: whole numbers.
"""
import ctypes

import numpy as np
import torch

from via_rs_b200 import _lib, prims, wire
from via_rs_b200.client import Client
from via_rs_b200.params import PAPER_Q1, PAPER_Q2, PAPER_Q3, SECURE_Q1, paper_preset, secure_preset
from via_rs_b200.server import VIA_RECORDS_NIBBLE, PublicKeys, Server, check

# Rings of the primitive operations: primes, degree.
RINGS = {
    "q1": (PAPER_Q1, 2048),
    "q2": ((PAPER_Q2,), 2048),
    "q3": ((PAPER_Q3,), 512),
    "secure_q1": (SECURE_Q1, 4096),
    "q1_256": (PAPER_Q1, 256),
}
# Gadgets (base, levels) the external product and the key switch meet in each ring.
EXTERNAL_GADGETS = {"q1": (55879, 2), "q2": (81, 2), "secure_q1": (18073, 2), "q1_256": (18, 3)}
SWITCH_GADGETS = {"q1": (18, 18), "q2": (18, 18), "secure_q1": (18, 18), "q1_256": (18, 18)}


def listed():
    return [
        # A private lookup in a small table (16 MiB): latency and launches are everything.
        {"name": "answer_small", "op": "answer", "preset": "paper", "rows": 16, "cols": 128},
        # The headline: one query against the 1 GiB database of the paper preset.
        {"name": "answer_1gib", "op": "answer", "preset": "paper", "rows": 256, "cols": 4096},
        # The 120-bit preset (n1 = 4096, other gadgets), 256 MiB.
        {"name": "answer_secure", "op": "answer", "preset": "secure", "rows": 64, "cols": 1024},
        # A query as clients send it, seeds instead of masks, 256 MiB.
        {"name": "answer_wire", "op": "answer_wire", "preset": "paper", "rows": 128, "cols": 2048},
        # A full serving batch: 64 distinct queries share one scan of 1 GiB.
        {"name": "many_64_1gib", "op": "answer_many", "preset": "paper", "rows": 256, "cols": 4096, "batch": 64},
        # What a lightly loaded service sees: a handful of queries joined in one scan, 64 MiB.
        {"name": "many_5", "op": "answer_many", "preset": "paper", "rows": 64, "cols": 1024, "batch": 5},
        # VIA-B at the preset's T = 8 (records of degree 64), 512 MiB.
        {"name": "batch_t8", "op": "answer_batch", "preset": "paper", "rows": 256, "cols": 2048, "n_rec": 64},
        # VIA-B with small records, many per answer.
        {"name": "batch_t64", "op": "answer_batch", "preset": "paper", "rows": 32, "cols": 256, "n_rec": 8},
        # A load generator's client: queries into HBM, answers recovered.
        {"name": "client_24", "op": "client", "preset": "paper", "rows": 256, "cols": 4096, "batch": 24},
        # The kernel micro-benchmarks' operations, on caller buffers.
        {"name": "ntt_q1", "op": "ntt", "ring": "q1", "count": 16384},
        {"name": "external_q1", "op": "external", "ring": "q1", "count": 4099},
        {"name": "key_switch_q1", "op": "key_switch", "ring": "q1", "count": 2048},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    op = rng.choice(["answer", "answer", "answer_wire", "answer_many", "answer_many", "answer_batch", "answer_batch",
                     "client", "ntt", "external", "key_switch"])
    if op in ("answer", "answer_wire"):
        preset = rng.choice(["paper", "paper", "paper", "secure"])
        top = 12 if preset == "paper" else 10
        return {"op": op, "preset": preset, "rows": 1 << rng.randint(2, 8), "cols": 1 << rng.randint(3, top)}
    if op == "answer_many":
        preset = rng.choice(["paper", "paper", "paper", "secure"])
        top, most = (12, 64) if preset == "paper" else (9, 16)
        return {"op": op, "preset": preset, "rows": 1 << rng.randint(2, 8), "cols": 1 << rng.randint(3, top),
                "batch": _log_uniform(rng, 2, most)}
    if op == "answer_batch":
        n_rec = 1 << rng.randint(3, 8)  # T = 64 .. 2
        return {"op": op, "preset": "paper", "rows": 1 << rng.randint(2, 8), "cols": 1 << rng.randint(3, 11),
                "n_rec": n_rec}
    if op == "client":
        return {"op": op, "preset": rng.choice(["paper", "secure"]), "rows": 1 << rng.randint(2, 8),
                "cols": 1 << rng.randint(3, 12), "batch": _log_uniform(rng, 1, 48)}
    if op == "ntt":
        ring = rng.choice(sorted(RINGS))
        primes, n = RINGS[ring]
        return {"op": op, "ring": ring, "count": _log_uniform(rng, 3, 16384 * 4096 // (len(primes) * n))}
    if op == "external":
        return {"op": op, "ring": rng.choice(sorted(EXTERNAL_GADGETS)), "count": _log_uniform(rng, 1, 4096)}
    return {"op": op, "ring": rng.choice(sorted(SWITCH_GADGETS)), "count": _log_uniform(rng, 1, 2048)}


def _params(case):
    make = paper_preset if case["preset"] == "paper" else secure_preset
    prm = make(case["rows"], case["cols"])
    return prm.with_dims(case["rows"], case["cols"], case.get("n_rec", prm.n_rec))


def _ternary(rng, n, primes):
    t = rng.integers(-1, 2, size=n)
    return np.concatenate([np.where(t < 0, q + t, t).astype(np.uint64) for q in primes])


def _client(prm, rng):
    return Client(prm, _ternary(rng, prm.n1, prm.q1), _ternary(rng, prm.n2, (prm.q3,)))


def _queries(prm, rng, count):
    client = _client(prm, rng)
    idx = rng.integers(prm.capacity, size=count)
    seeds = [rng.bytes(32) for _ in range(count)]
    out = client.queries(idx, seeds)
    client.close()
    return out


def _limb_uniform(rng, primes, polys, n):
    """[polys][nl][n] uniform residues, flat."""
    return np.stack([rng.integers(0, q, size=(polys, n), dtype=np.uint64) for q in primes], axis=1).reshape(-1)


def _keys(prm, rng):
    cascade = []
    for k in range(1, prm.n1.bit_length()):
        deg = 1 << k
        cascade.append(_limb_uniform(rng, prm.q1, 2 * prm.n1 // deg * prm.l_ck * 2, deg))
    conv = _limb_uniform(rng, prm.q1, prm.l_ck * 2, prm.n1)
    rsk = rng.integers(0, prm.q3, size=prm.rsk_len, dtype=np.uint64)
    return PublicKeys(np.concatenate(cascade), conv, rsk)


def _server(prm, seed, rng):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    size = prm.capacity * prm.n_rec // 2
    records = torch.randint(0, 256, (size,), dtype=torch.uint8, device="cuda", generator=gen).cpu().numpy()
    return Server.setup(prm, _keys(prm, rng), records, VIA_RECORDS_NIBBLE)


def _dev_uniform(gen, primes, polys, n):
    return torch.stack([torch.randint(0, q, (polys, n), dtype=torch.int64, device="cuda", generator=gen)
                        for q in primes], dim=1).contiguous()


def _to_device(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int64)).cuda()


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    op = case["op"]
    state = {"op": op, "stream": torch.cuda.Stream()}  # the caller's own stream
    if op in ("answer", "answer_wire", "answer_many", "answer_batch"):
        prm = _params(case)
        state["prm"], state["server"] = prm, _server(prm, seed, rng)
        if op == "answer":
            state["query"] = _queries(prm, rng, 1)[0]
        elif op == "answer_wire":
            q = _queries(prm, rng, 1)[0].reshape(prm.n_lwe, prm.lwe_len)
            state["wire"] = b"".join(wire.prg_packet(rng.bytes(32), lwe[-prm.nl:]) for lwe in q)
        elif op == "answer_many":
            b = case["batch"]
            state["queries"] = _to_device(_queries(prm, rng, b))
            state["masks"] = torch.empty((b, prm.n2), dtype=torch.int64, device="cuda")
            state["bodies"] = torch.empty_like(state["masks"])
            state["server"].reserve(b)
        else:
            state["queries"] = _queries(prm, rng, prm.n2 // prm.n_rec)
        return state
    if op == "client":
        prm, b = _params(case), case["batch"]
        state["client"] = _client(prm, rng)
        state["indices"] = rng.integers(prm.capacity, size=b)
        state["seeds"] = [rng.bytes(32) for _ in range(b)]
        state["out"] = torch.empty((b, prm.n_lwe * prm.lwe_len), dtype=torch.int64, device="cuda")
        state["masks"] = rng.integers(0, prm.q3, size=(b, prm.n2), dtype=np.uint64)
        state["bodies"] = rng.integers(0, prm.q4, size=(b, prm.n2), dtype=np.uint64)
        return state
    primes, n = RINGS[case["ring"]]
    count = case["count"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    state["ring"], state["count"] = prims.ring(n, primes), count
    if op == "ntt":
        # Transforms work in place; residues transformed again are residues again.
        state["fwd"] = _dev_uniform(gen, primes, count, n)
        state["inv"] = _dev_uniform(gen, primes, count, n)
    elif op == "external":
        base, levels = EXTERNAL_GADGETS[case["ring"]]
        state["gadget"] = (base, levels)
        state["rgsw"] = _dev_uniform(gen, primes, count * 2 * levels * 2, n)
        state["ct"] = _dev_uniform(gen, primes, count * 2, n)
        state["out"] = torch.empty_like(state["ct"])
    else:
        base, levels = SWITCH_GADGETS[case["ring"]]
        state["gadget"] = (base, levels)
        state["key"] = _dev_uniform(gen, primes, levels * 2, n)
        state["ct"] = _dev_uniform(gen, primes, count * 2, n)
        state["shifts"] = _to_device(rng.integers(0, 2 * n, size=count, dtype=np.uint64))
        state["out"] = torch.empty_like(state["ct"])
    return state


def run(s):
    op = s["op"]
    stream = s["stream"].cuda_stream
    if op == "answer":
        return s["server"].answer(s["query"])
    if op == "answer_wire":
        return wire.answer_wire(s["server"], s["wire"])
    if op == "answer_batch":
        return s["server"].answer_batch(s["queries"])
    if op == "answer_many":
        b, prm = s["masks"].shape[0], s["prm"]
        check(_lib.lib().via_server_answer_many_dev(
            s["server"]._h, ctypes.c_void_p(s["queries"].data_ptr()), b, prm.n_lwe,
            ctypes.c_void_p(s["masks"].data_ptr()), ctypes.c_void_p(s["bodies"].data_ptr()), ctypes.c_void_p(stream)))
        return s["masks"], s["bodies"]
    if op == "client":
        s["client"].queries_dev(s["indices"], s["seeds"], s["out"].data_ptr(), stream)
        return s["out"], s["client"].recover_many(s["masks"], s["bodies"])
    if op == "ntt":
        prims.ntt_forward_dev(s["ring"], s["fwd"].data_ptr(), s["count"], stream)
        prims.ntt_inverse_dev(s["ring"], s["inv"].data_ptr(), s["count"], stream)
        return s["fwd"], s["inv"]
    base, levels = s["gadget"]
    if op == "external":
        prims.external_product_dev(s["ring"], base, levels, s["rgsw"].data_ptr(), s["ct"].data_ptr(), s["count"],
                                   s["out"].data_ptr(), stream)
    else:
        prims.key_switch_dev(s["ring"], base, levels, s["key"].data_ptr(), s["ct"].data_ptr(),
                             s["shifts"].data_ptr(), s["count"], s["out"].data_ptr(), stream)
    return s["out"]


def _butterflies(n):
    return n // 2 * (n.bit_length() - 1)


def _expansion_products(prm):
    """Modular products of one query's expansion through CRot, transforms included."""
    n, nl, lck, lq = prm.n1, prm.nl, prm.l_ck, prm.l_query
    steps = n.bit_length() - 1
    cascade = 0
    for k in range(steps):  # n / deg masks of degree deg, each lck digits in nl limbs
        deg = 1 << k
        cascade += n // deg * lck * nl * (_butterflies(deg) if deg > 1 else 0)  # digit transforms
        cascade += n * lck * nl * 4  # every digit slot meets two output slots, mask and body
        cascade += (n // deg // 2) * nl * _butterflies(2 * deg)  # back to coefficients
    convert = nl * (lck + 2) * _butterflies(n) + 2 * lck * nl * n
    gate = lambda limbs: limbs * ((2 * lq + 2) * _butterflies(n) + 2 * lq * 2 * n)  # one external product
    gates = (prm.num_rows - 1) * gate(nl) + (prm.num_cols - 1 + prm.num_crot) * gate(1)
    select = prm.num_rows * 2 * _butterflies(n)
    return prm.n_lwe * (cascade + convert) + gates + select


def work(case):
    """Bytes each input and output takes once (database and key residues at their moduli's
    widths, everything else as the 8-byte words callers pass), and operations: a modular
    product and its addition count as two."""
    op = case["op"]
    if op in ("answer", "answer_wire", "answer_many", "answer_batch"):
        prm = _params(case)
        nq = case.get("batch", 1) if op == "answer_many" else (prm.n2 // prm.n_rec if op == "answer_batch" else 1)
        answers = nq if op == "answer_many" else 1
        cells = prm.num_rows * prm.num_cols * prm.n1
        keys = (prm.cascade_key_len + prm.conv_key_len) * 5 + prm.rsk_len * 3
        query = prm.n_lwe * (41 + 8 * prm.nl if op == "answer_wire" else 8 * prm.lwe_len)
        nbytes = cells * prm.q2.bit_length() / 8 + keys + nq * query + answers * 2 * prm.n2 * 8
        return {"bytes": nbytes, "flops": nq * (2.0 * 2 * cells + 2.0 * _expansion_products(prm))}
    if op == "client":
        prm, b = _params(case), case["batch"]
        words = b * (prm.n_lwe * prm.lwe_len + 3 * prm.n2)
        return {"bytes": words * 8, "flops": 2.0 * b * (prm.n_lwe * prm.nl * prm.n1 + prm.n2 * prm.n2)}
    primes, n = RINGS[case["ring"]]
    count, nl = case["count"], len(primes)
    poly = nl * n * 8
    if op == "ntt":
        return {"bytes": 4 * count * poly, "flops": 2.0 * 2 * count * nl * _butterflies(n)}
    if op == "external":
        levels = EXTERNAL_GADGETS[case["ring"]][1]
        transforms = (4 * levels + 2 * levels + 2) * nl * _butterflies(n)
        return {"bytes": count * (4 * levels + 4) * poly,
                "flops": 2.0 * count * (transforms + 4 * levels * nl * n)}
    levels = SWITCH_GADGETS[case["ring"]][1]
    return {"bytes": (2 * levels + 4 * count) * poly + 8 * count,
            "flops": 2.0 * count * nl * ((levels + 2) * _butterflies(n) + 2 * levels * n)}


def exact(case, seed):
    """Every output is a residue, compared for equality: there is no rounding to measure."""
    return None
