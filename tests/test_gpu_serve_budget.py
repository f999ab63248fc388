"""GPU: a server whose budget has no room for the register-radix tiles' root
tables runs on the smaller tables: it is created with what they leave, and gives
the oracle's products; exact."""
import numpy as np
import pytest

from oracle import oracle as O
import ntt_b200 as nb

pytestmark = pytest.mark.gpu

PRIMES = nb.generate_primes(31, 18, 8)
MAX_LOG = 17
# 16 ring slots of 2^14 .. 2^17 words and 2 x (4 x 2^17 + 8 x 2^10) bytes of roots a modulus;
# of 2^13 .. 2^17 words and 212 KB of images a modulus; below 1 MB of other tables and queue
RADIX = 64 * ((1 << 18) - (1 << 14)) + 8 * 2 * ((4 << 17) + (8 << 10))
SMALL = 64 * ((1 << 18) - (1 << 13)) + 8 * (212 << 10)


def product(a, b, moduli):
    fa, fb = (O.rns(v[None].astype(np.uint64), moduli, negacyclic=True)[0] for v in (a, b))
    q = np.array(moduli, dtype=np.uint64)[:, None]
    return O.rns(((fa * fb) % q)[None], moduli, negacyclic=True, inverse=True)[0].astype(np.uint32)


@pytest.mark.parametrize("mib", [20, 23, 24, 25, 26, 27, 36, 256])
def test_budget(torch_cuda, mib):
    rng = np.random.default_rng(mib)
    srv = nb.Server(PRIMES, hbm_budget_bytes=mib << 20, max_log_n=MAX_LOG, slots=1)
    st = srv.stats()
    assert st["resident_bytes"] + st["region_bytes"] <= mib << 20
    assert st["region_bytes"] > 1 << 20  # what a server needs
    if (mib << 20) - RADIX <= 1 << 20:  # no room for the roots
        assert st["region_bytes"] >= (mib << 20) - SMALL - (1 << 20)
    else:
        assert st["region_bytes"] >= (mib << 20) - RADIX - (1 << 20)
    jobs = []
    for lg, limbs in ((5, 2), (12, 3), (14, 8), (14, 1), (17, 8 if st["region_bytes"] >= 64 << 17 else 1), (16, 1)):
        a, b = (np.stack([rng.integers(0, q, 1 << lg, dtype=np.uint64) for q in PRIMES[:limbs]]).astype(np.uint32)
                for _ in range(2))
        out = np.zeros_like(a)
        jobs.append((a, b, limbs, out, srv.submit(a, b, out, lg, limbs, 0)))
    for a, b, limbs, out, i in jobs:
        srv.wait(i)
        assert (out == product(a, b, PRIMES[:limbs])).all()
    srv.close()
    assert nb.device_errors() == 0
