"""GPU: in-place calls captured into CUDA graphs after one eager call of the same
kind and nothing else: every entry point that stages a pass, replayed on fresh
data; graphs of one plan on several streams at once and beside eager calls; a
call outside that needs more memory than the captured one; exact."""
import numpy as np
import pytest

from conftest import BABYBEAR, Q60, to_dev, to_host
from oracle import oracle as O
import ntt_b200 as nb

pytestmark = pytest.mark.gpu


def make(kind, lg, rows):
    """plan, moduli, call(data, stream), forward?, word type"""
    if kind == "u64":
        p = nb.Plan(1 << lg, BABYBEAR)
        return p, [BABYBEAR] * rows, lambda d, s: p.transform(d, batch=rows, stream=s), np.uint64
    if kind == "wide":
        p = nb.WidePlan(lg, [Q60])
        return p, [Q60] * rows, lambda d, s: p.transform(d, d, rows, stream=s), np.uint64
    moduli = nb.generate_primes(31, lg + 1, rows)
    p = nb.RnsPlan(lg, moduli)
    engine = "scalar" if kind.endswith("scalar") else "auto"
    if kind.startswith("round trip"):
        # the round trip, then a forward transform: the oracle's forward
        return p, moduli, lambda d, s: (p.forward_inverse(d, 1, engine=engine, stream=s),
                                        p.transform(d, d, 1, engine=engine, stream=s)), np.uint32
    return p, moduli, lambda d, s: p.transform(d, d, 1, engine=engine, stream=s), np.uint32


def data(rng, moduli, lg):
    return np.stack([rng.integers(0, q, 1 << lg, dtype=np.uint64) for q in moduli])


def forward(x, moduli):
    return np.stack([O.ntt(r, q) for r, q in zip(x, moduli)])


CASES = [("rns", 14, 3), ("rns", 15, 1), ("rns", 16, 2), ("rns", 16, 8), ("rns", 17, 2), ("rns", 17, 8), ("rns", 20, 1),
         ("rns scalar", 14, 2), ("rns scalar", 17, 8), ("round trip", 14, 2), ("round trip", 16, 8), ("round trip", 17, 8),
         ("round trip scalar", 15, 2), ("wide", 14, 1), ("wide", 15, 3), ("wide", 20, 1), ("u64", 14, 2), ("u64", 15, 1),
         ("u64", 16, 8), ("u64", 19, 1), ("u64", 20, 1)]


@pytest.mark.parametrize("kind,lg,rows", CASES)
def test_capture_after_one_eager_call(torch_cuda, kind, lg, rows):
    torch = torch_cuda
    rng = np.random.default_rng(lg)
    plan, moduli, call, dtype = make(kind, lg, rows)
    x = data(rng, moduli, lg)
    d = to_dev(torch, x.astype(dtype).reshape(-1))
    call(d, None)
    torch.cuda.synchronize()
    want = forward(x, moduli)
    assert (to_host(d, dtype).reshape(x.shape) == want).all()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call(d, torch.cuda.current_stream())
    for _ in range(2):
        x = data(rng, moduli, lg)
        d.copy_(to_dev(torch, x.astype(dtype).reshape(-1)))
        g.replay()
        torch.cuda.synchronize()
        assert (to_host(d, dtype).reshape(x.shape) == forward(x, moduli)).all()
    assert nb.device_errors() == 0


@pytest.mark.parametrize("kind,lg,rows", [("rns", 14, 3), ("rns", 17, 8), ("round trip", 16, 8), ("wide", 15, 3), ("u64", 15, 2)])
def test_graphs_of_one_plan_run_at_once(torch_cuda, kind, lg, rows):
    torch = torch_cuda
    rng = np.random.default_rng(lg + 1)
    plan, moduli, call, dtype = make(kind, lg, rows)
    x = data(rng, moduli, lg)
    words = x.astype(dtype).reshape(-1)
    n = 4
    ds = [to_dev(torch, words) for _ in range(n)]
    graphs = []
    for d in ds[:-1]:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            call(d, torch.cuda.current_stream())
        graphs.append(g)
    streams = [torch.cuda.Stream() for _ in range(n)]
    want = forward(x, moduli)
    for _ in range(10):
        for d in ds:
            d.copy_(to_dev(torch, words))
        torch.cuda.synchronize()
        for s, d, g in zip(streams, ds, graphs + [None]):
            with torch.cuda.stream(s):
                g.replay() if g else call(d, s)
        torch.cuda.synchronize()
        for d in ds:
            assert (to_host(d, dtype).reshape(x.shape) == want).all()


def test_captured_workspace_outlives_larger_calls(torch_cuda):
    torch = torch_cuda
    lg, limbs, polys = 15, 2, 40
    moduli = nb.generate_primes(31, lg + 1, limbs)
    plan = nb.RnsPlan(lg, moduli)
    rng = np.random.default_rng(3)
    x, big = data(rng, moduli, lg), np.stack([data(rng, moduli, lg) for _ in range(polys)])
    d, e = to_dev(torch, x.astype(np.uint32).reshape(-1)), to_dev(torch, big.astype(np.uint32).reshape(-1))
    plan.transform(d, d, 1)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        plan.transform(d, d, 1, stream=torch.cuda.current_stream())
    plan.transform(e, e, polys)
    d.copy_(to_dev(torch, x.astype(np.uint32).reshape(-1)))
    g.replay()
    torch.cuda.synchronize()
    assert (to_host(d, np.uint32).reshape(x.shape) == forward(x, moduli)).all()
    assert (to_host(e, np.uint32).reshape(big.shape) == O.rns(big, moduli)).all()


def test_workspaces_of_destroyed_graphs_are_taken_again(torch_cuda):
    torch = torch_cuda
    lg, limbs = 16, 128  # 32 MB staged a call
    moduli = nb.generate_primes(31, lg + 1, limbs)
    plan = nb.RnsPlan(lg, moduli)
    d = torch.zeros(limbs << lg, dtype=torch.int32, device="cuda")
    plan.transform(d, d, 1)
    torch.cuda.synchronize()

    def capture():
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            plan.transform(d, d, 1, stream=torch.cuda.current_stream())
            plan.transform(d, d, 1, inverse=True, stream=torch.cuda.current_stream())
        g.replay()
        torch.cuda.synchronize()
        g.reset()

    capture()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(8):
        capture()
    assert before - torch.cuda.mem_get_info()[0] <= 64 << 20  # at most two of them, not eight
