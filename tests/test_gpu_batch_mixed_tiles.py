"""GPU: batches of the register-radix queue whose other units run its CUDA-core
tiles: sizes above 2^20 and below 2^10 beside sizes in its range, both directions
and twists, products; exact."""
import numpy as np
import pytest

from conftest import to_dev, to_host
from oracle import oracle as O
import ntt_b200 as nb

pytestmark = pytest.mark.gpu

MAX_LOG = 22
PRIMES = nb.generate_primes(31, MAX_LOG + 1, 3)


def host(rng, lg, limbs):
    return np.stack([rng.integers(0, q, 1 << lg, dtype=np.uint64) for q in PRIMES[:limbs]]).astype(np.uint32)


@pytest.mark.parametrize("shapes", [[(21, 2), (15, 3)], [(22, 1), (10, 1)], [(1, 3), (4, 2), (9, 3), (13, 2), (20, 1)],
                                    [(21, 1), (9, 2), (12, 3), (14, 1), (22, 1)]])
def test_units_out_of_range(torch_cuda, shapes):
    rng = np.random.default_rng(len(shapes))
    plan = nb.BatchPlan(PRIMES, MAX_LOG, negacyclic=True)
    jobs, want = [], []
    for lg, limbs in shapes:
        mods = PRIMES[:limbs]
        for inv in (False, True):
            for nega in (False, True):
                x = host(rng, lg, limbs)
                jobs.append((to_dev(torch_cuda, x.reshape(-1)), lg, limbs, 0, inv, nega))
                want.append(O.rns(x[None], mods, inverse=inv, negacyclic=nega)[0])
        a, b = host(rng, lg, limbs), host(rng, lg, limbs)
        fa, fb = (O.rns(v[None], mods, negacyclic=True)[0] for v in (a, b))
        prod = (fa * fb) % np.array(mods, dtype=np.uint64)[:, None]
        jobs.append((to_dev(torch_cuda, a.reshape(-1)), lg, limbs, 0, "mul", True, to_dev(torch_cuda, b.reshape(-1))))
        want.append(O.rns(prod[None], mods, inverse=True, negacyclic=True)[0])
    plan.batch(jobs).launch()
    torch_cuda.cuda.synchronize()
    for j, w in zip(jobs, want):
        assert (to_host(j[0], np.uint32).reshape(w.shape) == w).all(), j[1:6]
    assert nb.device_errors() == 0
