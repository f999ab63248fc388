"""GPU: which tiles a batch of mixed sizes runs: the register-radix queue where
sizes of its range carry the work, the CUDA-core kernel where sizes outside it do
(its tiles hold half as many limbs of 2^10); every route exact.  A server of small
polynomials chooses batch by batch."""
import numpy as np
import pytest

from conftest import to_dev, to_host
from oracle import oracle as O
import ntt_b200 as nb

pytestmark = pytest.mark.gpu

PRIMES = nb.generate_primes(31, 23, 8)


def host(rng, lg, limbs):
    return np.stack([rng.integers(0, q, 1 << lg, dtype=np.uint64) for q in PRIMES[:limbs]]).astype(np.uint32)


# (log2 n, polynomials) of 8 limbs; register-radix tiles?
@pytest.mark.parametrize("shapes,radix", [([(10, 1)], True), ([(8, 40), (10, 1)], False), ([(9, 2), (10, 2)], True),
                                          ([(9, 3), (10, 1)], False), ([(4, 300), (10, 1)], False),
                                          ([(8, 40), (10, 1), (13, 1)], True), ([(21, 1), (10, 1)], False),
                                          ([(2, 3), (5, 2), (10, 700), (21, 1)], True)])
def test_route(torch_cuda, shapes, radix):
    rng = np.random.default_rng(1)
    plan = nb.BatchPlan(PRIMES, 22, negacyclic=True)
    jobs, want = [], []
    for i, lg in enumerate(lg for lg, polys in shapes for _ in range(polys)):
        x = host(rng, lg, 8)
        inv, nega = i % 2 == 1, i % 3 == 0
        jobs.append((to_dev(torch_cuda, x.reshape(-1)), lg, 8, 0, inv, nega))
        want.append(O.rns(x[None], PRIMES, inverse=inv, negacyclic=nega)[0])
    b = plan.batch(jobs)
    alone = plan.batch([j for j in jobs if j[1] != 10]).info()["tiles"] if len(shapes) > 1 else 0
    b.launch()
    torch_cuda.cuda.synchronize()
    for j, w in zip(jobs, want):
        assert (to_host(j[0], np.uint32).reshape(w.shape) == w).all(), j[1:]
    n10 = dict(shapes)[10]
    if not any(lg > 12 for lg, _ in shapes):  # 8 limbs of 2^10: one tile, or two of 4096 residues
        assert b.info()["tiles"] - alone == (n10 if radix else 2 * n10)
    assert nb.device_errors() == 0


def test_server_of_small_polynomials(torch_cuda):
    rng = np.random.default_rng(2)
    srv = nb.Server(PRIMES, hbm_budget_bytes=64 << 20, max_log_n=12, slots=2, max_batch_requests=4)
    for sizes in ([4, 8, 9], [12, 12, 5], [9] * 20, [10, 9, 3, 11], [6] * 9 + [12]):
        reqs = []
        for lg in sizes:
            x = host(rng, lg, 3)
            out = np.zeros_like(x)
            reqs.append((x, out, srv.submit_ntt(x, out, lg, 3, 0)))
        for x, out, i in reqs:
            srv.wait(i)
            assert (out == O.rns(x[None], PRIMES[:3], negacyclic=True)[0]).all()
    srv.close()
    assert nb.device_errors() == 0
