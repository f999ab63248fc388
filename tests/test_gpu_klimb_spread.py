"""GPU: K-limb transforms whose passes are one to four blocks an SM (they ask for a
share of its shared memory), for every form of a residue, against the network in
Z/p; whole numbers: no tolerance."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_klimb_words import MODULI, rows
import ntt_b200 as nb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,log_n", [("bn254", 16), ("bn254", 17), ("from_2e254", 16), ("from_2e254", 17), ("goldilocks", 17),
                                        ("goldilocks", 18), ("from_2e64", 18), ("k2", 18)])
def test_spread_passes(torch_cuda, name, log_n):
    torch = torch_cuda
    K, p = MODULI[name]
    n, R = 1 << log_n, 1 << (24 * K)
    rng = np.random.default_rng(log_n)
    xs = [int(v) * 0x9E3779B97F4A7C15F39CC0605CEDC834 % p for v in rng.integers(1, 2 ** 62, n, dtype=np.uint64)]
    omega, tw, t = 0x9E3779B97F4A7C15 * 0xF39CC0605CEDC835 % p, [], 1
    for _ in range(n):
        tw.append(t * R % p)
        t = t * omega % p
    want = rows([v * R % p for v in O.host_ntt_naive(xs, omega, p)], K)
    d = torch.from_numpy(rows([v * R % p for v in xs], K).reshape(-1).view(np.int32)).cuda()
    w = torch.from_numpy(rows(tw, K).reshape(-1).view(np.int32)).cuda()
    prime = [int(v) for v in rows([p], K)[0]]
    for _ in range(2):  # the second call's first pass starts behind the first call's last
        x = d.clone()
        nb.klimb_forward(K, x, w, log_n, prime, nb.klimb_neg_inv24(prime[0]))
    torch.cuda.synchronize()
    assert (x.cpu().numpy().view(np.uint32).reshape(n, K) == want).all()
