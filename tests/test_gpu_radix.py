"""GPU: the register-radix passes of the CUDA-core engine (csrc/radix.cuh)
against the oracle, bit for bit: every size they serve that no other file
covers, row counts around the CTA grouping, several polynomials per CTA,
moduli at both ends of their range."""
import numpy as np
import pytest

from conftest import BABYBEAR, to_dev, to_host
from oracle import oracle as O
import ntt_b200 as nb

pytestmark = pytest.mark.gpu


def rows(moduli, polys, n, seed):
    rng = np.random.default_rng(seed)
    return np.stack([np.stack([rng.integers(0, q, n, dtype=np.uint64) for q in moduli]) for _ in range(polys)])


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("nega", [False, True])
@pytest.mark.parametrize("lg,limbs,polys", [(5, 1, 1), (5, 3, 101), (7, 2, 3), (8, 1, 149), (9, 3, 1), (11, 5, 1),
                                            (13, 1, 2), (14, 1, 1), (14, 3, 2), (15, 2, 1), (16, 9, 1), (19, 1, 1),
                                            (14, 1, 300)])
def test_u32_sizes(torch_cuda, lg, limbs, polys, nega, inverse):
    moduli = (nb.generate_primes(31, lg + 1, 2) + nb.generate_primes(27, lg + 1, limbs))[:limbs]
    x = rows(moduli, polys, 1 << lg, 100 * lg + limbs)
    x[0, 0, :] = moduli[0] - 1  # every residue at its largest
    plan = nb.RnsPlan(lg, moduli, negacyclic=nega)
    d = to_dev(torch_cuda, x.astype(np.uint32).reshape(-1))
    out = torch_cuda.empty_like(d)
    plan.transform(out, d, polys, inverse=inverse, engine="scalar")
    torch_cuda.cuda.synchronize()
    assert (to_host(d, np.uint32).reshape(x.shape) == x).all()  # the source is left alone
    pick = [0, polys - 1]
    want = O.rns(x[pick], moduli, inverse=inverse, negacyclic=nega)
    assert (to_host(out, np.uint32).reshape(x.shape)[pick] == want).all()
    plan.transform(out, out, polys, inverse=not inverse, engine="scalar")  # and back, in place
    torch_cuda.cuda.synchronize()
    assert (to_host(out, np.uint32).reshape(x.shape) == x).all()


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("lg,batch", [(5, 1), (9, 7), (11, 150), (14, 3), (15, 1), (19, 1), (20, 2)])
def test_u64_words(torch_cuda, lg, batch, inverse):
    n = 1 << lg
    x = rows([BABYBEAR], batch, n, lg)[:, 0]
    # any word below 2^32 stands for its residue
    words = np.where(x < (1 << 32) - BABYBEAR, x + BABYBEAR, x).astype(np.uint64)
    plan = nb.Plan(n, BABYBEAR)
    d = to_dev(torch_cuda, words.reshape(-1))
    plan.transform(d, batch=batch, inverse=inverse, engine="scalar")
    torch_cuda.cuda.synchronize()
    got = to_host(d, np.uint64).reshape(batch, n)
    for i in {0, batch - 1}:
        assert (got[i] == O.ntt(x[i], BABYBEAR, inverse=inverse)).all()


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("nega", [False, True])
@pytest.mark.parametrize("lg,limbs,polys", [(5, 2, 65), (8, 3, 1), (11, 1, 3), (13, 2, 1), (14, 1, 2), (15, 3, 1),
                                            (17, 2, 1), (20, 1, 1)])
def test_wide_sizes(torch_cuda, lg, limbs, polys, nega, inverse):
    moduli = (nb.generate_primes(62, lg + 1, 2) + nb.generate_primes(33, lg + 1, limbs))[:limbs]
    x = rows(moduli, polys, 1 << lg, 7 * lg + limbs)
    x[0, 0, :] = moduli[0] - 1
    plan = nb.WidePlan(lg, moduli, negacyclic=nega)
    d = to_dev(torch_cuda, x.reshape(-1))
    out = torch_cuda.empty_like(d)
    plan.transform(out, d, polys, inverse=inverse, engine="scalar")
    torch_cuda.cuda.synchronize()
    pick = [0, polys - 1]
    want = O.rns(x[pick], moduli, inverse=inverse, negacyclic=nega)
    assert (to_host(out, np.uint64).reshape(x.shape)[pick] == want).all()
    plan.transform(out, out, polys, inverse=not inverse, engine="scalar")
    torch_cuda.cuda.synchronize()
    assert (to_host(out, np.uint64).reshape(x.shape) == x).all()
