"""GPU: the register-radix tiles' root tables go by the sizes that a plan's batches
have: small batches of a plan made for large ones hold little, a larger size adds
its own table, and batches made before stay valid; exact."""
import numpy as np
import pytest

from conftest import to_dev, to_host
from oracle import oracle as O
import ntt_b200 as nb

pytestmark = pytest.mark.gpu


def job(torch, rng, moduli, lg, first, inv):
    x = np.stack([rng.integers(0, q, 1 << lg, dtype=np.uint64) for q in moduli[first:first + 2]]).astype(np.uint32)
    want = O.rns(x[None], moduli[first:first + 2], negacyclic=True, inverse=inv)[0]
    return x, (to_dev(torch, x.reshape(-1)), lg, 2, first, inv, True), want


def check(torch, b, jobs):
    for x, j, _ in jobs:
        j[0].copy_(to_dev(torch, x.reshape(-1)))
    b.launch()
    torch.cuda.synchronize()
    for _, j, want in jobs:
        assert (to_host(j[0], np.uint32).reshape(want.shape) == want).all(), j[1:]


def test_tables_grow_with_the_sizes_in_use(torch_cuda):
    torch = torch_cuda
    rng = np.random.default_rng(4)
    moduli = nb.generate_primes(31, 21, 24)
    warm = nb.BatchPlan(moduli[:2], 20, negacyclic=True)
    for sizes in ([10, 14], [20]):  # the kernels and a first workspace
        jobs = [job(torch, rng, moduli, lg, 0, False) for lg in sizes]
        check(torch, warm.batch([j for _, j, _ in jobs]), jobs)
    plan = nb.BatchPlan(moduli, 20, negacyclic=True)
    batches = []
    for sizes, table in (([10, 12, 13], 13), ([14, 11, 15], 15), ([17], 17), ([20, 16, 10], 20), ([18], None)):
        jobs = [job(torch, rng, moduli, lg, f, inv) for lg in sizes for f in (0, 22) for inv in (False, True)]
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        b = plan.batch([j for _, j, _ in jobs])
        held = before - torch.cuda.mem_get_info()[0] - b.info()["ws_bytes"]
        # two kinds of 4 bytes a root; the queue and an allocator's granules below 16 MB
        assert held <= (2 * 4 * len(moduli) << table if table else 0) + (16 << 20), (sizes, held)
        check(torch, b, jobs)
        batches.append((b, jobs))
        for b, jobs in batches:
            check(torch, b, jobs)
    assert nb.device_errors() == 0
