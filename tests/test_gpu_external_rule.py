"""External products on both sides of the line between the fused kernel and separate ones: deep
gadgets and degree 4096 at 62 or 63 CTAs and at 64, against the oracle."""
import numpy as np
import pytest

from via_rs_b200 import prims
from via_rs_b200.params import PAPER_Q1, PAPER_Q2, SECURE_Q1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("primes,n,base,L,count", [(PAPER_Q1, 256, 18, 11, 31), (PAPER_Q1, 256, 18, 11, 32),
                                                   (PAPER_Q1, 1024, 600, 5, 2), (PAPER_Q1, 1024, 600, 5, 32),
                                                   ((PAPER_Q2,), 2048, 13, 4, 63), ((PAPER_Q2,), 2048, 13, 4, 64),
                                                   (SECURE_Q1, 4096, 18073, 2, 31), (SECURE_Q1, 4096, 18073, 2, 32)])
def test_both_sides(oracle, primes, n, base, L, count):
    import torch

    rng = np.random.default_rng(n + count)
    draw = lambda polys: np.stack([rng.integers(0, q, size=(polys, n), dtype=np.uint64) for q in primes], axis=1)
    rgsw, ct = draw(count * 4 * L), draw(count * 2)
    d = [torch.from_numpy(x.view(np.int64)).cuda() for x in (rgsw, ct)]
    out = torch.empty_like(d[1])
    prims.external_product_dev(prims.ring(n, primes), base, L, d[0].data_ptr(), d[1].data_ptr(), count, out.data_ptr())
    want = oracle.external_product(primes, n, base, L, rgsw.reshape(-1), ct.reshape(-1))
    assert np.array_equal(out.cpu().numpy().view(np.uint64).reshape(-1), want)


def test_fused_products_take_no_scratch():
    """A batch of the fused kernel runs in the memory its buffers leave (the separate kernels would want
    1.5 times the RGSWs again)."""
    import torch

    n, L, count = 2048, 2, 2048
    rgsw = torch.randint(0, min(PAPER_Q1), (count * 4 * L, 2, n), dtype=torch.int64, device="cuda")
    ct = torch.randint(0, min(PAPER_Q1), (count * 2, 2, n), dtype=torch.int64, device="cuda")
    out = torch.empty_like(ct)
    ring = prims.ring(n, PAPER_Q1)
    prims.external_product_dev(ring, 55879, L, rgsw.data_ptr(), ct.data_ptr(), 1, out.data_ptr())
    want = out[:2].clone()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (200 << 20), dtype=torch.uint8, device="cuda")
    prims.external_product_dev(ring, 55879, L, rgsw.data_ptr(), ct.data_ptr(), count, out.data_ptr())
    del filler
    torch.cuda.empty_cache()
    assert torch.equal(out[:2], want)
