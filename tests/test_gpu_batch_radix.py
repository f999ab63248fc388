"""GPU: the batch queue's register-radix tiles (csrc/batch_radix.cuh) against
the oracle, bit for bit: every size they serve with limb counts that leave rows
of a tile empty, both directions and twists, products, jobs off a 16-byte
boundary (other tiles), and uint64 plan transforms through the queue."""
import numpy as np
import pytest

from conftest import BABYBEAR, to_dev, to_host
from oracle import oracle as O
import ntt_b200 as nb

pytestmark = pytest.mark.gpu

PRIMES = nb.generate_primes(31, 21, 3) + nb.generate_primes(28, 21, 6)


def host(rng, lg, limbs, first):
    x = np.stack([rng.integers(0, PRIMES[first + l], 1 << lg, dtype=np.uint64) for l in range(limbs)])
    x[0, : 1 << (lg - 1)] = PRIMES[first] - 1
    return x.astype(np.uint32)


@pytest.mark.parametrize("lg,limbs", [(10, 1), (10, 9), (11, 5), (12, 3), (13, 2), (14, 3), (15, 1), (16, 2), (17, 1),
                                      (18, 2), (19, 1), (20, 1)])
def test_sizes(torch_cuda, lg, limbs):
    rng = np.random.default_rng(lg)
    plan = nb.BatchPlan(PRIMES, 20, negacyclic=True)
    jobs, want = [], []
    for i, (inv, nega) in enumerate([(a, b) for a in (False, True) for b in (False, True)] * 2):
        first = i % (len(PRIMES) - limbs + 1)
        x = host(rng, lg, limbs, first)
        jobs.append((to_dev(torch_cuda, x.reshape(-1)), lg, limbs, first, inv, nega))
        want.append(O.rns(x[None], PRIMES[first:first + limbs], inverse=inv, negacyclic=nega)[0])
    b = plan.batch(jobs)
    b.launch()
    torch_cuda.cuda.synchronize()
    for j, w in zip(jobs, want):
        assert (to_host(j[0], np.uint32).reshape(w.shape) == w).all(), j[1:]
    assert nb.device_errors() == 0


@pytest.mark.parametrize("nega", [False, True])
@pytest.mark.parametrize("lg", [10, 12, 13, 14, 17, 20])
def test_products(torch_cuda, lg, nega):
    rng = np.random.default_rng(100 + lg)
    plan = nb.BatchPlan(PRIMES, 20, negacyclic=nega)
    jobs, want = [], []
    for first in (0, 4):
        mods = PRIMES[first:first + 3]
        a, b = host(rng, lg, 3, first), host(rng, lg, 3, first)
        fa, fb = (O.rns(v[None], mods, negacyclic=nega)[0] for v in (a, b))
        prod = (fa * fb) % np.array(mods, dtype=np.uint64)[:, None]
        jobs.append((to_dev(torch_cuda, a.reshape(-1)), lg, 3, first, "mul", nega, to_dev(torch_cuda, b.reshape(-1))))
        want.append((O.rns(prod[None], mods, inverse=True, negacyclic=nega)[0], fb))
    plan.batch(jobs).launch()
    torch_cuda.cuda.synchronize()
    for j, (w, fb) in zip(jobs, want):
        assert (to_host(j[0], np.uint32).reshape(w.shape) == w).all()
        assert (to_host(j[6], np.uint32).reshape(w.shape) == fb).all()
    assert nb.device_errors() == 0


@pytest.mark.parametrize("lg", [10, 13, 14, 16])
def test_jobs_off_the_copy_alignment(torch_cuda, lg):
    rng = np.random.default_rng(7)
    plan = nb.BatchPlan(PRIMES, 16, negacyclic=True)
    x = host(rng, lg, 2, 0)
    buf = torch_cuda.zeros((2 << lg) + 1, dtype=torch_cuda.int32, device="cuda")
    buf[1:] = to_dev(torch_cuda, x.reshape(-1))
    y = host(rng, lg, 2, 1)
    d = to_dev(torch_cuda, y.reshape(-1))
    plan.batch([(buf[1:], lg, 2, 0, False, True), (d, lg, 2, 1, True, False)]).launch()
    torch_cuda.cuda.synchronize()
    assert (to_host(buf, np.uint32)[1:].reshape(x.shape) == O.rns(x[None], PRIMES[:2], negacyclic=True)[0]).all()
    assert (to_host(d, np.uint32).reshape(y.shape) == O.rns(y[None], PRIMES[1:3], inverse=True)[0]).all()


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("lg,batch", [(17, 9), (18, 5), (19, 3), (20, 1)])
def test_uint64_transforms_through_the_queue(torch_cuda, lg, batch, inverse):
    n = 1 << lg
    x = np.random.default_rng(lg).integers(0, BABYBEAR, (batch, n), dtype=np.uint64)
    words = np.where(np.arange(n) % 3 == 0, x + BABYBEAR, x).astype(np.uint64)  # any word below 2^32
    plan = nb.Plan(n, BABYBEAR)
    d = to_dev(torch_cuda, words.reshape(-1))
    plan.transform(d, batch=batch, inverse=inverse)
    torch_cuda.cuda.synchronize()
    got = to_host(d, np.uint64).reshape(batch, n)
    for i in {0, batch - 1}:
        assert (got[i] == O.ntt(x[i], BABYBEAR, inverse=inverse)).all()
    assert nb.device_errors() == 0
