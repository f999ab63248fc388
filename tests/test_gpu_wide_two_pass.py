"""GPU: 64-bit transforms at the size where one launch becomes two passes, and its
neighbours: both directions and twists, in place and out of place, limbs and
polynomials around a wave of blocks, under capture; exact."""
import numpy as np
import pytest

from conftest import to_dev, to_host
from oracle import oracle as O
import ntt_b200 as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nega", [False, True])
@pytest.mark.parametrize("lg,limbs,polys", [(12, 2, 3), (13, 1, 1), (13, 3, 2), (13, 1, 75), (13, 2, 80), (14, 1, 2)])
def test_in_and_out_of_place(torch_cuda, lg, limbs, polys, nega):
    torch = torch_cuda
    rng = np.random.default_rng(lg + polys)
    moduli = nb.generate_primes(60, lg + 1, limbs)
    plan = nb.WidePlan(lg, moduli, negacyclic=nega)
    x = np.stack([np.stack([rng.integers(0, q, 1 << lg, dtype=np.uint64) for q in moduli]) for _ in range(polys)])
    x[0, 0, :16] = moduli[0] - 1
    for inverse in (False, True):
        want = O.rns(x, moduli, negacyclic=nega, inverse=inverse)
        s = to_dev(torch, x.reshape(-1))
        o = torch.empty_like(s)
        plan.transform(o, s, polys, inverse=inverse)
        plan.transform(s, s, polys, inverse=inverse)
        torch.cuda.synchronize()
        assert (to_host(o, np.uint64).reshape(x.shape) == want).all()
        assert (to_host(s, np.uint64).reshape(x.shape) == want).all()


def test_under_capture(torch_cuda):
    torch = torch_cuda
    q = nb.generate_primes(60, 14, 1)
    plan = nb.WidePlan(13, q)
    x = np.random.default_rng(5).integers(0, q[0], 1 << 13, dtype=np.uint64)
    d = to_dev(torch, x)
    plan.transform(d, d, 1)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan.transform(d, d, 1, stream=torch.cuda.current_stream())
    d.copy_(to_dev(torch, x))
    g.replay()
    torch.cuda.synchronize()
    assert (to_host(d, np.uint64) == O.ntt(x, q[0])).all()
