"""GPU: K-limb transforms whose table is the output of the call just before them on
the stream, so that the first pass's blocks may start before the table is whole;
whole numbers: no tolerance."""
import numpy as np
import pytest

from test_gpu_klimb_words import MODULI, rows
import ntt_b200 as nb

pytestmark = pytest.mark.gpu


def network(xs, tw, p):
    """The radix-2 DIT network over any table: stage s multiplies by tw[k n / 2^(s+1)]."""
    n = len(xs)
    lg = n.bit_length() - 1
    a = [xs[int(format(i, "0%db" % lg)[::-1], 2)] for i in range(n)]
    half = 1
    while half < n:
        step = n // (2 * half)
        for g in range(0, n, 2 * half):
            for k in range(half):
                u, t = a[g + k], a[g + k + half] * tw[k * step] % p
                a[g + k], a[g + k + half] = (u + t) % p, (u - t) % p
        half *= 2
    return a


@pytest.mark.parametrize("name,log_n", [("bn254", 7), ("bn254", 11), ("from_2e254", 9), ("goldilocks", 10), ("goldilocks", 12),
                                        ("from_2e64", 11), ("k2", 12)])
def test_output_as_table(torch_cuda, name, log_n):
    torch = torch_cuda
    K, p = MODULI[name]
    n, R = 1 << log_n, 1 << (24 * K)
    rng = np.random.default_rng(log_n)
    draw = lambda: [int(v) * 0x9E3779B97F4A7C15F39CC0605CEDC834 % p for v in rng.integers(1, 2 ** 62, n, dtype=np.uint64)]  # noqa: E731
    table, ys, xs = draw(), draw(), draw()
    mid = network(ys, table, p)
    want = rows([v * R % p for v in network(xs, mid, p)], K)
    put = lambda v: torch.from_numpy(rows([x * R % p for x in v], K).reshape(-1).view(np.int32)).cuda()  # noqa: E731
    t, y, x = put(table), put(ys), put(xs)
    prime = [int(v) for v in rows([p], K)[0]]
    np_ = nb.klimb_neg_inv24(prime[0])
    for _ in range(5):
        w, d = y.clone(), x.clone()
        torch.cuda.synchronize()
        nb.klimb_forward(K, w, t, log_n, prime, np_)
        nb.klimb_forward(K, d, w, log_n, prime, np_)
        torch.cuda.synchronize()
        assert (d.cpu().numpy().view(np.uint32).reshape(n, K) == want).all()
