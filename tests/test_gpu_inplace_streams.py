"""GPU: in-place transforms of one plan on several streams and threads at once
(more streams than a plan keeps workspaces for), the fused round trip at every
size, and in-place calls under stream capture; exact."""
import threading

import numpy as np
import pytest

from conftest import to_dev, to_host
from oracle import oracle as O
import ntt_b200 as nb

pytestmark = pytest.mark.gpu


def batch(moduli, polys, lg, seed):
    rng = np.random.default_rng(seed)
    return np.stack([np.stack([rng.integers(0, q, 1 << lg, dtype=np.uint64) for q in moduli]) for _ in range(polys)])


@pytest.mark.parametrize("lg,limbs,polys", [(5, 3, 7), (9, 2, 1), (11, 1, 150), (12, 4, 1), (13, 2, 1), (14, 2, 3), (15, 1, 1),
                                            (16, 9, 1), (17, 2, 1), (18, 1, 1), (19, 2, 1), (20, 1, 2)])
@pytest.mark.parametrize("nega", [False, True])
@pytest.mark.parametrize("engine", ["auto", "scalar"])
def test_round_trip(torch_cuda, lg, limbs, polys, nega, engine):
    moduli = nb.generate_primes(31, lg + 1, limbs)
    x = batch(moduli, polys, lg, lg)
    plan = nb.RnsPlan(lg, moduli, negacyclic=nega)
    d = to_dev(torch_cuda, x.astype(np.uint32).reshape(-1))
    nb.profile_start()
    plan.forward_inverse(d, polys, engine=engine)
    torch_cuda.cuda.synchronize()
    launches = sum(v[0] for v in nb.profile_stop().values())
    assert launches == (1 if lg <= 13 else 3)
    assert (to_host(d, np.uint32).reshape(x.shape) == x).all()


@pytest.mark.parametrize("lg,limbs", [(14, 3), (16, 8), (17, 8)])
def test_streams_and_threads_share_a_plan(torch_cuda, lg, limbs):
    torch = torch_cuda
    moduli = nb.generate_primes(31, lg + 1, limbs)
    plan = nb.RnsPlan(lg, moduli, negacyclic=True)
    xs = [batch(moduli, 1, lg, 50 + i) for i in range(6)]
    ds = [to_dev(torch, x.astype(np.uint32).reshape(-1)) for x in xs]
    torch.cuda.synchronize()

    def work(i):
        s = torch.cuda.Stream()
        for _ in range(20):
            plan.transform(ds[i], ds[i], 1, stream=s)
            plan.transform(ds[i], ds[i], 1, inverse=True, stream=s)
            plan.forward_inverse(ds[i], 1, stream=s)
        plan.transform(ds[i], ds[i], 1, stream=s)
        s.synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for x, d in zip(xs, ds):
        assert (to_host(d, np.uint32).reshape(x.shape) == O.rns(x, moduli, negacyclic=True)).all()
    assert nb.device_errors() == 0


@pytest.mark.parametrize("lg,limbs", [(12, 2), (16, 8)])
def test_in_place_under_capture(torch_cuda, lg, limbs):
    torch = torch_cuda
    moduli = nb.generate_primes(31, lg + 1, limbs)
    plan = nb.RnsPlan(lg, moduli, negacyclic=True)
    x = batch(moduli, 1, lg, 9)
    d = to_dev(torch, x.astype(np.uint32).reshape(-1))
    s = torch.cuda.Stream()
    plan.transform(d, d, 1, stream=s, engine="int8" if lg == 16 else "auto")  # sets up what a capture may not
    plan.transform(d, d, 1, inverse=True, stream=s)
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        plan.transform(d, d, 1, stream=torch.cuda.current_stream())
    for _ in range(2):
        d.copy_(to_dev(torch, x.astype(np.uint32).reshape(-1)))
        g.replay()
        torch.cuda.synchronize()
        assert (to_host(d, np.uint32).reshape(x.shape) == O.rns(x, moduli, negacyclic=True)).all()
