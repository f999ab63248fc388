"""GPU: plans destroyed while their in-place calls are still queued.  Destroying
waits for them before it gives their workspaces back, so the results are the
oracle's although the memory is handed out again at once; exact."""
import numpy as np
import pytest

from conftest import BABYBEAR, Q60, to_dev, to_host
from oracle import oracle as O
import ntt_b200 as nb

pytestmark = pytest.mark.gpu


def plan_and_oracle(kind, lg):
    if kind == "u64":
        return nb.Plan(1 << lg, BABYBEAR), [BABYBEAR], lambda p, d, s: p.transform(d, stream=s), np.uint64
    if kind == "wide":
        return nb.WidePlan(lg, [Q60]), [Q60], lambda p, d, s: p.transform(d, d, 1, stream=s), np.uint64
    moduli = nb.generate_primes(31, lg + 1, 3)
    call = {"rns": lambda p, d, s: p.transform(d, d, 1, stream=s),
            "round trip": lambda p, d, s: (p.forward_inverse(d, 1, stream=s), p.transform(d, d, 1, stream=s))}[kind]
    return nb.RnsPlan(lg, moduli), moduli, call, np.uint32


# one stream: its kept workspace; six: more than a plan keeps
@pytest.mark.parametrize("n_streams", [1, 6])
@pytest.mark.parametrize("kind,lg", [("rns", 14), ("rns", 17), ("round trip", 16), ("wide", 15), ("u64", 15)])
def test_destroyed_with_calls_queued(torch_cuda, kind, lg, n_streams):
    torch = torch_cuda
    rng = np.random.default_rng(lg)
    plan, moduli, call, dtype = plan_and_oracle(kind, lg)
    x = np.stack([rng.integers(0, q, 1 << lg, dtype=np.uint64) for q in moduli])
    reps = 5
    ds = [[to_dev(torch, x.astype(dtype).reshape(-1)) for _ in range(reps)] for _ in range(n_streams)]
    streams = [torch.cuda.Stream() for _ in range(n_streams)]
    busy = torch.zeros((n_streams, 16 << 20), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for s, row, b in zip(streams, ds, busy):
        with torch.cuda.stream(s):
            for _ in range(50):
                b.add_(1)  # keeps the calls queued
        for d in row:
            call(plan, d, s)
    plan.close()
    other = torch.full((64 << 20,), -1, dtype=torch.int32, device="cuda")  # takes what was given back
    torch.cuda.synchronize()
    want = O.rns(x[None], moduli)[0]
    for row in ds:
        for d in row:
            assert (to_host(d, dtype).reshape(x.shape) == want).all()
    assert int(other[0]) == -1
