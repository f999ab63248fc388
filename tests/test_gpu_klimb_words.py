"""The K-limb forward transform over the moduli and pointers that decide how
residues are held between stages: K = 11 below and from 2^254, K = 3 below and
from 2^64, 16-byte aligned pointers or not.  The network is compared in Z/p (any
odd p) at tile edges: one tile, the first size above, two and three passes.
Whole numbers: no tolerance."""
import numpy as np
import pytest

from oracle import oracle as O
import ntt_b200 as nb

pytestmark = pytest.mark.gpu

BN254 = 21888242871839275222246405745257275088548364400416034343698204186575808495617
MODULI = {
    "bn254": (11, BN254),
    "below_2e254": (11, (1 << 254) - 1),
    "from_2e254": (11, (1 << 254) + 1),
    "below_2e264": (11, (1 << 264) - 1),
    "small_k11": (11, 65537),
    "goldilocks": (3, 0xFFFFFFFF00000001),
    "below_2e64": (3, (1 << 64) - 1),
    "from_2e64": (3, (1 << 64) + 1),
    "small_k3": (3, 3),
    "k2": (2, (1 << 48) - 59),
}


def rows(vals, K):
    return np.array([[(v >> (24 * k)) & 0xFFFFFF for k in range(K)] for v in vals], dtype=np.uint32)


@pytest.mark.parametrize("log_n", [0, 1, 2, 5, 8, 9, 11, 12])
@pytest.mark.parametrize("name", sorted(MODULI))
def test_network_over_moduli(torch_cuda, name, log_n):
    torch = torch_cuda
    K, p = MODULI[name]
    n, R = 1 << log_n, 1 << (24 * K)
    rng = np.random.default_rng(log_n + p % 1000)
    draw = lambda: int.from_bytes(rng.bytes(40), "little") % p  # noqa: E731
    omega = draw() | 1
    xs = [draw() for _ in range(n)]
    xs[0] = p - 1
    xs[-1] = p - 1
    tw, t = [], 1
    for _ in range(n):
        tw.append(t * R % p)
        t = t * omega % p
    want = rows([v * R % p for v in O.host_ntt_naive(xs, omega % p, p)], K)
    data, table = rows([v * R % p for v in xs], K).reshape(-1), rows(tw, K).reshape(-1)
    prime = [int(v) for v in rows([p], K)[0]]
    for off in (0, 1):  # words off a 16-byte boundary
        d = torch.zeros(n * K + 8, dtype=torch.int32, device="cuda")
        w = torch.zeros(n * K + 8, dtype=torch.int32, device="cuda")
        d[off:off + n * K] = torch.from_numpy(data.view(np.int32)).cuda()
        w[off:off + n * K] = torch.from_numpy(table.view(np.int32)).cuda()
        nb.klimb_forward(K, d[off:], w[off:], log_n, prime, nb.klimb_neg_inv24(prime[0]))
        torch.cuda.synchronize()
        got = d.cpu().numpy().view(np.uint32)
        assert (got[off:off + n * K].reshape(n, K) == want).all()
        assert not got[:off].any() and not got[off + n * K:].any()
