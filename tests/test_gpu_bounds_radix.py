"""GPU: the NTT_DEBUG_BOUNDS build over the register-radix passes, the batch
queue's register-radix tiles and the K-limb passes, every size that they serve:
their own tests pass there and no check fails; and a residue outside the input
contract is reported, so the checks of these kernels are in that build."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PATHS = "import sys\nROOT = %r\nsys.path[:0] = [ROOT, ROOT + '/ntt-tensorcore_b200', ROOT + '/tests']\n" % ROOT


def run_dbg(code):
    env = dict(os.environ, NTT_B200_LIB="dbg")
    r = subprocess.run([sys.executable, "-c", PATHS + code], env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


CLEAN = r'''
import json, pytest
import ntt_b200 as nb
assert nb.LIB_PATH.endswith("libntt_b200_dbg.so")
T = ROOT + "/tests/"
rc = pytest.main(["-q", "-x", "-p", "no:cacheprovider", T + "test_gpu_radix.py", T + "test_gpu_batch_radix.py",
                  T + "test_gpu_klimb_words.py", T + "test_gpu_klimb.py", T + "test_gpu_inplace_streams.py"])
enabled, flags = nb.bounds_errors()
print(json.dumps({"rc": int(rc), "enabled": enabled, "flags": flags}))
'''


def test_no_check_fails(torch_cuda):
    assert run_dbg(CLEAN) == {"rc": 0, "enabled": True, "flags": 0}


INPUT = r'''
import json, torch
import ntt_b200 as nb
def word(n, value, dtype):
    x = torch.zeros(n, dtype=dtype, device="cuda")
    x[n - 1] = value
    return x
got = {}
def flags(name, f):
    f()
    torch.cuda.synchronize()
    got[name] = nb.bounds_errors(clear=True)[1]
q = nb.generate_primes(30, 21, 1)
Q60 = 1152921504577486849
for lg in (8, 15):
    n = 1 << lg
    rns, wide = nb.RnsPlan(lg, q), nb.WidePlan(lg, [Q60])
    x, y = word(n, q[0], torch.int32), word(n, Q60, torch.int64)
    flags("rns %d" % lg, lambda: rns.transform(torch.empty_like(x), x, 1, inverse=True))
    flags("wide %d" % lg, lambda: wide.transform(torch.empty_like(y), y, 1))
for lg in (10, 15):
    x = word(1 << lg, q[0], torch.int32)
    b = nb.BatchPlan(q, 15).batch([(x, lg, 1, 0, True, False)])
    flags("batch %d" % lg, lambda: b.launch())
print(json.dumps(got))
'''


def test_input_outside_the_contract_is_reported(torch_cuda):
    got = run_dbg(INPUT)
    for name, flags in got.items():
        assert flags >> (16 if name.startswith("batch") else 24) & 1 << 6, (name, flags)
