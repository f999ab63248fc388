"""The work that is timed: NTT calls through the Python binding (ntt_b200),
over the sizes of this repository's benchmark, tests and drop-in programs.

Kinds of case:
  rns      RnsPlan on [poly][limb][n] uint32 residues (31-bit primes)
  u64      Plan on uint64 words, one modulus (the drop-in API's transforms)
  wide     WidePlan on uint64 residues (60-bit primes)
  batch    BatchPlan: an uneven list of transforms in one launch
  product  BatchPlan: polynomial products in one launch
  klimb    klimb_forward on K-limb Montgomery residues

listed() has twelve of them, draw(rng) gives more of the same ranges.
"""
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "ntt-tensorcore_b200"))
import ntt_b200 as nb  # noqa: E402

BABYBEAR = 2013265921
BN254_R = 21888242871839275222246405745257275088548364400416034343698204186575808495617
GOLDILOCKS = 0xFFFFFFFF00000001
# residues of one drawn case at most (the largest listed transform batch)
MOST_RESIDUES = 12 << 20


def listed():
    return [
        # one small ciphertext polynomial: the call's latency is what a user waits for
        {"name": "rns_2e12_l4", "kind": "rns", "log_n": 12, "limbs": 4, "polys": 1, "op": "forward", "nega": True},
        # a few mid-size CRT polynomials back to coefficients (odd limb count)
        {"name": "rns_2e14_l13_p4_inv", "kind": "rns", "log_n": 14, "limbs": 13, "polys": 4, "op": "inverse", "nega": True},
        # the benchmark's headline step: 24 limbs of 2^16, forward then inverse in place
        {"name": "rns_2e16_l24_roundtrip", "kind": "rns", "log_n": 16, "limbs": 24, "polys": 1, "op": "round_trip", "nega": True},
        # a batch of eight such polynomials into the NTT domain: throughput
        {"name": "rns_2e16_l24_p8_fwd", "kind": "rns", "log_n": 16, "limbs": 24, "polys": 8, "op": "forward", "nega": True},
        # the largest ring of the serving mix, above the cluster kernel's size
        {"name": "rns_2e17_l33_fwd", "kind": "rns", "log_n": 17, "limbs": 33, "polys": 1, "op": "forward", "nega": True},
        # the drop-in API at the first size of the reference's benchmark program
        {"name": "u64_2e12_fwd", "kind": "u64", "log_n": 12, "batch": 1, "inverse": False},
        # and at its largest
        {"name": "u64_2e20_fwd", "kind": "u64", "log_n": 20, "batch": 1, "inverse": False},
        # one polynomial mod a 60-bit prime, the big-prime benchmark's size
        {"name": "wide_2e20_fwd", "kind": "wide", "log_n": 20, "limbs": 1, "polys": 1, "inverse": False, "nega": False},
        # a negacyclic CRT basis of 60-bit primes, back to coefficients
        {"name": "wide_2e15_l9_p2_inv", "kind": "wide", "log_n": 15, "limbs": 9, "polys": 2, "inverse": True, "nega": True},
        # polynomials of many sizes, limb counts and directions in one launch (the largest case)
        {"name": "batch_mixed_96", "kind": "batch", "jobs": 96, "low": 12, "high": 20, "limbs": 32, "mix": 4},
        # ciphertext products as the server runs them
        {"name": "product_2e14_l12_x12", "kind": "product", "log_n": 14, "limbs": 12, "count": 12},
        # the K-limb drop-in on the BN254 field
        {"name": "klimb_bn254_2e15", "kind": "klimb", "K": 11, "log_n": 15},
    ]


def _spread(rng, low, high):
    """A whole number from [low, high], even over its logarithm."""
    return max(low, min(high, int(round(low * (high / low) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["rns", "rns", "rns", "u64", "u64", "wide", "wide", "batch", "product", "klimb"])
    if kind == "rns":
        log_n = rng.randint(11, 17)
        limbs = _spread(rng, 1, 48)
        polys = _spread(rng, 1, max(1, min(64, MOST_RESIDUES // (limbs << log_n))))
        return {"kind": kind, "log_n": log_n, "limbs": limbs, "polys": polys,
                "op": rng.choice(["forward", "inverse", "round_trip"]), "nega": rng.random() < 0.75}
    if kind == "u64":
        log_n = rng.randint(10, 20)
        return {"kind": kind, "log_n": log_n, "batch": _spread(rng, 1, max(1, min(33, MOST_RESIDUES // 2 >> log_n))),
                "inverse": rng.random() < 0.5}
    if kind == "wide":
        log_n = rng.randint(12, 20)
        nega = rng.random() < 0.5
        limbs = _spread(rng, 1, max(1, min(16, MOST_RESIDUES // 4 >> log_n)))
        polys = _spread(rng, 1, max(1, min(16, MOST_RESIDUES // 4 // (limbs << log_n))))
        return {"kind": kind, "log_n": log_n, "limbs": limbs, "polys": polys, "inverse": rng.random() < 0.5, "nega": nega}
    if kind == "batch":
        low = rng.randint(10, 14)
        return {"kind": kind, "jobs": _spread(rng, 8, 64), "low": low, "high": rng.randint(low + 2, 19),
                "limbs": _spread(rng, 4, 32), "mix": rng.randint(1, 1 << 20)}
    if kind == "product":
        log_n = rng.randint(12, 17)
        limbs = _spread(rng, 4, 48)
        return {"kind": kind, "log_n": log_n, "limbs": limbs,
                "count": _spread(rng, 1, max(1, min(24, MOST_RESIDUES // 4 // (limbs << log_n))))}
    K = rng.choice([3, 11])
    return {"kind": kind, "K": K, "log_n": rng.randint(7, 18 if K == 3 else 16)}


# ------------------------------------------------------------------ moduli
def _is_prime(n):
    small = (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37)
    for p in small:
        if n % p == 0:
            return n == p
    d, r = n - 1, 0
    while d % 2 == 0:
        d //= 2
        r += 1
    for a in small:
        x = pow(a, d, n)
        if x in (1, n - 1):
            continue
        for _ in range(r - 1):
            x = x * x % n
            if x == n - 1:
                break
        else:
            return False
    return True


def _primes(bits, two_adicity, count):
    """The `count` largest primes below 2^bits that are 1 mod 2^two_adicity."""
    out, k = [], ((1 << bits) - 1) >> two_adicity
    while len(out) < count:
        q = (k << two_adicity) + 1
        if _is_prime(q):
            out.append(q)
        k -= 1
    return out


def _moduli(case):
    kind = case["kind"]
    if kind == "u64":
        return [BABYBEAR]
    if kind == "batch":
        return _primes(31, case["high"] + 1, case["limbs"])
    if kind == "wide":
        return _primes(60, case["log_n"] + 1, case["limbs"])
    return _primes(31, case["log_n"] + 1, case["limbs"])


def _residues(qs, rows, n, gen, dtype):
    """rows x len(qs) x n uniform residues, limb l below qs[l], on the GPU."""
    q = torch.tensor(qs, dtype=torch.int64, device="cuda").view(1, -1, 1)
    x = torch.randint(0, 1 << 62, (rows, len(qs), n), generator=gen, device="cuda", dtype=torch.int64)
    return x.remainder_(q).to(dtype).contiguous()


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


def _batch_shapes(case):
    """(log_n, limbs, inverse) of each job: sizes and limb counts uniform, half of them inverse."""
    r = random.Random(case["mix"])
    return [(r.randint(case["low"], case["high"]), r.randint(1, case["limbs"]), r.random() < 0.5)
            for _ in range(case["jobs"])]


# ------------------------------------------------------------------ K-limb
def _limbs(values, K):
    """Whole numbers below 2^(24 K) -> [len][K] uint32 24-bit limbs."""
    raw = np.frombuffer(b"".join(v.to_bytes(3 * K, "little") for v in values), dtype=np.uint8)
    raw = raw.reshape(len(values), K, 3).astype(np.uint32)
    return np.ascontiguousarray(raw[..., 0] | raw[..., 1] << 8 | raw[..., 2] << 16)


def _klimb_field(case):
    p, g = (BN254_R, 5) if case["K"] == 11 else (GOLDILOCKS, 7)
    return p, pow(g, (p - 1) >> case["log_n"], p)


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    kind, gen = case["kind"], _generator(seed)
    if kind == "rns":
        qs = _moduli(case)
        x = _residues(qs, case["polys"], 1 << case["log_n"], gen, torch.int32)
        plan = nb.RnsPlan(case["log_n"], qs, negacyclic=case["nega"])
        return {"case": case, "plan": plan, "x": x, "y": torch.empty_like(x)}
    if kind == "u64":
        x = _residues(_moduli(case), case["batch"], 1 << case["log_n"], gen, torch.int64)
        return {"case": case, "plan": nb.Plan(1 << case["log_n"], BABYBEAR), "x": x}
    if kind == "wide":
        qs = _moduli(case)
        x = _residues(qs, case["polys"], 1 << case["log_n"], gen, torch.int64)
        plan = nb.WidePlan(case["log_n"], qs, negacyclic=case["nega"])
        return {"case": case, "plan": plan, "x": x, "y": torch.empty_like(x)}
    if kind == "batch":
        qs, shapes = _moduli(case), _batch_shapes(case)
        x = torch.empty(sum(l << lg for lg, l, _ in shapes), dtype=torch.int32, device="cuda")
        jobs, at = [], 0
        for lg, limbs, inv in shapes:
            view = x[at:at + (limbs << lg)]
            view.copy_(_residues(qs[:limbs], 1, 1 << lg, gen, torch.int32).view(-1))
            jobs.append((view, lg, limbs, 0, inv, False))
            at += limbs << lg
        plan = nb.BatchPlan(qs, case["high"])
        return {"case": case, "plan": plan, "x": x, "batch": plan.batch(jobs)}
    if kind == "product":
        qs = _moduli(case)
        a = _residues(qs, case["count"], 1 << case["log_n"], gen, torch.int32)
        b = _residues(qs, case["count"], 1 << case["log_n"], gen, torch.int32)
        plan = nb.BatchPlan(qs, case["log_n"], negacyclic=True)
        jobs = [(a[i], case["log_n"], case["limbs"], 0, "mul", True, b[i]) for i in range(case["count"])]
        return {"case": case, "plan": plan, "a": a, "b": b, "batch": plan.batch(jobs)}
    K, n = case["K"], 1 << case["log_n"]
    p, w = _klimb_field(case)
    tw, t = [], (1 << (24 * K)) % p
    for _ in range(n):
        tw.append(t)
        t = t * w % p
    # residues below p: the top limb below p's own, the others any 24 bits
    x = torch.randint(0, 1 << 24, (n, K), generator=gen, device="cuda", dtype=torch.int32)
    x[:, K - 1] = torch.randint(0, p >> (24 * (K - 1)), (n,), generator=gen, device="cuda", dtype=torch.int32)
    prime = [int(v) for v in _limbs([p], K)[0]]
    return {"case": case, "x": x, "tw": torch.from_numpy(_limbs(tw, K).view(np.int32)).cuda(), "prime": prime,
            "np": nb.klimb_neg_inv24(prime[0])}


# --------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rns":
        if case["op"] == "round_trip":
            state["plan"].forward_inverse(state["x"], case["polys"])
            return state["x"]
        state["plan"].transform(state["y"], state["x"], case["polys"], inverse=case["op"] == "inverse")
        return state["y"]
    if kind == "u64":  # in place, as the drop-in API is
        state["plan"].transform(state["x"], batch=case["batch"], inverse=case["inverse"])
        return state["x"]
    if kind == "wide":
        state["plan"].transform(state["y"], state["x"], case["polys"], inverse=case["inverse"])
        return state["y"]
    if kind == "batch":
        state["batch"].launch()
        return state["x"]
    if kind == "product":  # the products, and the second operands' transforms that it leaves
        state["batch"].launch()
        return [state["a"], state["b"]]
    nb.klimb_forward(case["K"], state["x"], state["tw"], case["log_n"], state["prime"], state["np"])
    return state["x"]


# -------------------------------------------------------------------- work
def work(case):
    """Each residue read and written once per transform; per transform and
    residue log2(n) / 2 butterflies of one modular product and two sums."""
    kind = case["kind"]
    if kind == "batch":
        shapes = _batch_shapes(case)
        return {"bytes": sum(8 * (l << lg) for lg, l, _ in shapes), "flops": sum(1.5 * lg * (l << lg) for lg, l, _ in shapes)}
    lg = case["log_n"]
    if kind == "product":  # a and b read, the product and b's transform written
        r = case["count"] * case["limbs"] << lg
        return {"bytes": 16 * r, "flops": 3 * 1.5 * lg * r}
    if kind == "klimb":
        return {"bytes": 12 * case["K"] << lg, "flops": 1.5 * lg * case["K"] ** 2 * (1 << lg)}
    if kind == "u64":
        return {"bytes": 16 * case["batch"] << lg, "flops": 1.5 * lg * (case["batch"] << lg)}
    r = case["polys"] * case["limbs"] << lg
    if kind == "wide":
        return {"bytes": 16 * r, "flops": 1.5 * lg * r}
    return {"bytes": 8 * r, "flops": (3 if case["op"] == "round_trip" else 1.5) * lg * r}


# ------------------------------------------------------------------- exact
def _powers(base, count, q):
    out = np.ones(count, dtype=np.uint64)
    step, done = base % q, 1
    while done < count:
        k = min(done, count - done)
        out[done:done + k] = out[:k] * np.uint64(step) % np.uint64(q)
        step, done = step * step % q, done + k
    return out


def _ntt(x, q, inverse, nega):
    """The transform of each row of x (q < 2^31), radix 2 on numpy uint64."""
    n = x.shape[1]
    lg, uq = n.bit_length() - 1, np.uint64(q)
    g = next(g for g in range(2, q) if all((q - 1) % p or pow(g, (q - 1) // p, q) != 1 for p in (2, 3, 5, 7)))
    psi = pow(g, (q - 1) >> (lg + 1), q) if nega else 1
    w = pow(g, (q - 1) >> lg, q)
    if inverse:
        w = pow(w, -1, q)
    elif nega:
        x = x * _powers(psi, n, q) % uq
    tw = _powers(w, n // 2, q)
    rev = np.zeros(n, dtype=np.int64)
    for b in range(lg):
        rev |= ((np.arange(n) >> b) & 1) << (lg - 1 - b)
    x = x[:, rev]
    for s in range(lg):
        half = 1 << s
        v = x.reshape(x.shape[0], -1, 2, half)
        t = v[:, :, 1] * tw[:: n >> (s + 1)][:half] % uq
        x = np.stack([(v[:, :, 0] + t) % uq, (v[:, :, 0] + (uq - t)) % uq], axis=2).reshape(x.shape)
    if inverse:
        x = x * np.uint64(pow(n, -1, q)) % uq
        if nega:
            x = x * _powers(pow(psi, -1, q), n, q) % uq
    return x


def exact(case, seed):
    """The same transforms in 64-bit whole numbers, without the library: for
    moduli below 2^31 (wider ones need more than 64 bits), and not for the
    mixed batch, which would take minutes."""
    kind, gen = case["kind"], _generator(seed)
    if kind not in ("rns", "u64", "product"):
        return None
    qs, n = _moduli(case), 1 << case["log_n"]
    rows = case["polys" if kind == "rns" else "batch" if kind == "u64" else "count"]
    wide = torch.int64 if kind == "u64" else torch.int32
    x = _residues(qs, rows, n, gen, wide)
    if kind == "rns" and case["op"] == "round_trip":
        return x
    out = x.cpu().numpy().astype(np.uint64)
    if kind == "product":
        b = _residues(qs, rows, n, gen, wide).cpu().numpy().astype(np.uint64)
        for l, q in enumerate(qs):
            b[:, l] = _ntt(b[:, l], q, False, True)
            out[:, l] = _ntt(_ntt(out[:, l], q, False, True) * b[:, l] % np.uint64(q), q, True, True)
        return [out.astype(np.int32), b.astype(np.int32)]
    inverse = case["inverse"] if kind == "u64" else case["op"] == "inverse"
    for l, q in enumerate(qs):
        out[:, l] = _ntt(out[:, l], q, inverse, kind == "rns" and case["nega"])
    return out.astype(np.int64 if kind == "u64" else np.int32)
