"""GPU: NTT_B200_ENGINE names the engine of single AUTO transforms only: the
round trip and the host stream keep AUTO's own choice, at sizes that the named
engine does not serve too."""
import numpy as np
import pytest

from conftest import to_dev, to_host
from oracle import oracle as O
import ntt_b200 as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", ["scalar", "dmma", "int8", "tiles"])
@pytest.mark.parametrize("lg,limbs", [(4, 2), (12, 3), (14, 2), (16, 2), (16, 8), (17, 8), (21, 1)])
def test_round_trip_and_host_stream(torch_cuda, monkeypatch, engine, lg, limbs):
    monkeypatch.setenv("NTT_B200_ENGINE", engine)
    rng = np.random.default_rng(lg)
    moduli = nb.generate_primes(31, lg + 1, limbs)
    plan = nb.RnsPlan(lg, moduli, negacyclic=True)
    x = np.stack([rng.integers(0, q, 1 << lg, dtype=np.uint64) for q in moduli])
    d = to_dev(torch_cuda, x.astype(np.uint32).reshape(-1))
    plan.forward_inverse(d, 1)
    torch_cuda.cuda.synchronize()
    assert (to_host(d, np.uint32).reshape(x.shape) == x).all()
    src, out = x.astype(np.uint32).reshape(-1), np.zeros(x.size, dtype=np.uint32)
    plan.stream_host(src, out, 1, 1, mode="forward")
    torch_cuda.cuda.synchronize()
    assert (out.reshape(x.shape) == O.rns(x[None], moduli, negacyclic=True)[0]).all()
