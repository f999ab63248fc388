"""GPU: in-place calls of more rows than are staged at a time: groups of whole
polynomials, groups of one polynomial's limbs, remainders, every word type, the
round trip; equal to the out-of-place call and, at the first, last and middle
rows, to the oracle; and the memory that they hold is that of one group."""
import numpy as np
import pytest

from conftest import BABYBEAR, Q60, to_dev, to_host
from oracle import oracle as O
import ntt_b200 as nb

pytestmark = pytest.mark.gpu


def random_rows(torch, moduli, polys, lg, dtype):
    g = torch.Generator(device="cuda").manual_seed(lg)
    x = torch.empty((polys, len(moduli), 1 << lg), dtype=dtype, device="cuda")
    for l, q in enumerate(moduli):
        x[:, l] = torch.randint(0, q, (polys, 1 << lg), generator=g, device="cuda", dtype=torch.int64).to(dtype)
    return x


def host_rows(x, rows, dtype):
    flat = x.reshape(-1, x.shape[-1])
    return [to_host(flat[r], dtype).astype(np.uint64) for r in rows]


# rows of 2^lg staged at a time: 2^25 >> lg
@pytest.mark.parametrize("lg,limbs,polys", [(14, 7, 300), (16, 24, 23), (16, 600, 1), (17, 3, 91), (20, 17, 2), (20, 40, 1),
                                            (21, 17, 1), (23, 1, 5)])
@pytest.mark.parametrize("inverse", [False, True])
def test_rns(torch_cuda, lg, limbs, polys, inverse):
    torch = torch_cuda
    moduli = nb.generate_primes(31, lg + 1, limbs) if limbs <= 24 else nb.generate_primes(31, lg, 20) * (limbs // 20)
    plan = nb.RnsPlan(lg, moduli, negacyclic=limbs <= 24)
    x = random_rows(torch, moduli, polys, lg, torch.int32)
    d, o = x.clone(), torch.empty_like(x)
    plan.transform(o, x, polys, inverse=inverse, engine="scalar")
    plan.transform(d, d, polys, inverse=inverse)
    torch.cuda.synchronize()
    assert torch.equal(d, o)
    rows = sorted({0, limbs * polys // 2, limbs * polys - 1})
    f = O.negacyclic if limbs <= 24 else O.ntt
    for r, a, b in zip(rows, host_rows(x, rows, np.uint32), host_rows(d, rows, np.uint32)):
        assert (f(a, moduli[r % limbs], inverse=inverse) == b).all()
    if lg <= 20 and not inverse:
        plan.forward_inverse(x, polys)
        plan.transform(x, x, polys)
        torch.cuda.synchronize()
        assert torch.equal(x, o)


@pytest.mark.parametrize("kind,lg,polys", [("wide", 16, 600), ("wide", 20, 33), ("wide", 22, 9), ("u64", 16, 600), ("u64", 20, 33),
                                           ("u64", 22, 9)])
def test_uint64_words(torch_cuda, kind, lg, polys):
    torch = torch_cuda
    q = Q60 if kind == "wide" else BABYBEAR
    x = random_rows(torch, [q], polys, lg, torch.int64)
    d = x.clone()
    if kind == "wide":
        nb_plan = nb.WidePlan(lg, [q])
        nb_plan.transform(d, d, polys)
    else:
        nb_plan = nb.Plan(1 << lg, q)
        nb_plan.transform(d, batch=polys, engine="scalar")
    torch.cuda.synchronize()
    rows = [0, 1, polys // 2, polys // 2 + 1, polys - 1]
    for a, b in zip(host_rows(x, rows, np.uint64), host_rows(d, rows, np.uint64)):
        assert (O.ntt(a, q) == b).all()


def test_memory_held(torch_cuda):
    torch = torch_cuda
    moduli = nb.generate_primes(31, 17, 24)
    small, plan = nb.RnsPlan(16, moduli), nb.RnsPlan(16, moduli)
    d = torch.zeros(128 * 24 << 16, dtype=torch.int32, device="cuda")  # 805 MB a call
    streams = [torch.cuda.Stream() for _ in range(3)]
    for s in streams:  # what the streams and the kernels take
        for polys in (1, 24):
            small.transform(d, d, polys, stream=s)
            small.forward_inverse(d, polys, stream=s)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for s in streams:
        plan.transform(d, d, 128, stream=s)
        plan.forward_inverse(d, 128, stream=s)
        s.synchronize()
    held = before - torch.cuda.mem_get_info()[0]
    assert held <= 3 * (128 << 20) + (64 << 20)  # one group of 2^25 words a stream, and an allocator's granule
