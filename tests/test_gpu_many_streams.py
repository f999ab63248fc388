"""GPU: in-place calls of one plan on more streams than keep a workspace, by count
and by memory, from several threads on one stream, and with growing calls; equal
to the out-of-place call, which stages nothing."""
import threading

import pytest

import ntt_b200 as nb

pytestmark = pytest.mark.gpu


def rows(torch, moduli, polys, lg, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.empty((polys, len(moduli), 1 << lg), dtype=torch.int32, device="cuda")
    for l, q in enumerate(moduli):
        x[:, l] = torch.randint(0, q, (polys, 1 << lg), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    return x


@pytest.mark.parametrize("lg,limbs,polys,streams,reps", [(14, 2, 1, 40, 4), (16, 24, 22, 6, 2), (20, 3, 1, 36, 1)])
def test_more_streams_than_workspaces(torch_cuda, lg, limbs, polys, streams, reps):
    torch = torch_cuda
    moduli = nb.generate_primes(31, lg + 1, limbs)
    plan = nb.RnsPlan(lg, moduli, negacyclic=True)
    x = rows(torch, moduli, polys, lg, lg)
    want = torch.empty_like(x)
    plan.transform(want, x, polys)
    ds, ss = [x.clone() for _ in range(streams)], [torch.cuda.Stream() for _ in range(streams)]
    torch.cuda.synchronize()
    for _ in range(reps):
        for d, s in zip(ds, ss):
            plan.transform(d, d, polys, stream=s)
            plan.transform(d, d, polys, inverse=True, stream=s)
            plan.forward_inverse(d, polys, stream=s)
    for d, s in zip(ds, ss):
        plan.transform(d, d, polys, stream=s)
    torch.cuda.synchronize()
    for d in ds:
        assert torch.equal(d, want)


def test_growing_calls_and_threads_on_one_stream(torch_cuda):
    torch = torch_cuda
    lg, moduli = 14, nb.generate_primes(31, 15, 2)
    plan = nb.RnsPlan(lg, moduli)
    s = torch.cuda.Stream()
    sizes = [1, 7, 3, 40, 2, 200]
    xs = [rows(torch, moduli, p, lg, p) for p in sizes]
    wants = [torch.empty_like(x) for x in xs]
    for x, w in zip(xs, wants):
        plan.transform(w, x, x.shape[0])
    torch.cuda.synchronize()

    def work(x):
        for _ in range(10):
            plan.transform(x, x, x.shape[0], stream=s)
            plan.transform(x, x, x.shape[0], inverse=True, stream=s)
        plan.transform(x, x, x.shape[0], stream=s)

    threads = [threading.Thread(target=work, args=(x,)) for x in xs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for x, w in zip(xs, wants):
        assert torch.equal(x, w)
