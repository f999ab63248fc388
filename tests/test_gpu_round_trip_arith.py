"""GPU: the fused round trip on inputs that only its arithmetic brings back: words
in [q, 2q), which the forward butterflies reduce, return canonical, so passes that
moved data without transforming it fail; exact."""
import numpy as np
import pytest

from conftest import to_dev, to_host
import ntt_b200 as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nega", [False, True])
@pytest.mark.parametrize("lg,limbs,polys", [(5, 2, 3), (7, 3, 5), (10, 1, 1), (12, 4, 1), (13, 2, 2), (14, 2, 3), (15, 3, 1),
                                            (16, 24, 1), (17, 2, 1), (18, 1, 1), (19, 2, 1), (20, 1, 2)])
def test_round_trip_reduces(torch_cuda, lg, limbs, polys, nega):
    rng = np.random.default_rng(lg)
    moduli = nb.generate_primes(31, lg + 1, limbs)
    x = np.stack([np.stack([rng.integers(0, q, 1 << lg, dtype=np.uint64) for q in moduli]) for _ in range(polys)])
    q = np.array(moduli, dtype=np.uint64)[None, :, None]
    words = np.where(rng.integers(0, 2, x.shape, dtype=np.uint64) == 1, x + q, x)
    plan = nb.RnsPlan(lg, moduli, negacyclic=nega)
    d = to_dev(torch_cuda, words.astype(np.uint32).reshape(-1))
    plan.forward_inverse(d, polys)
    torch_cuda.cuda.synchronize()
    assert (to_host(d, np.uint32).reshape(x.shape) == x).all()
