"""GPU test of the bounded waits: a wait that cannot be satisfied gives up by itself, the kernel unwinds and
reports it, the Python layer raises, and the next launch on the same device is correct.

The failure is made in the allowed form only. A TEST BUILD of the library (-DKD_TEST_DROP_LOAD, wait limit
20 ms instead of 0.4 s) lets the TMA producer of one CTA leave out one K tile load when the environment
variable KD_TEST_DROP_LOAD=1 is set at launch (2 to 4: what the backward's producers leave out, see attn_bwd.cuh): no copy is issued and no bytes are expected, so nothing is in
flight for that stage. The first wait on the starved chain (the S issuer's for the tile, or a softmax warp's for
the scores) runs out after 20 ms, records
KD_STATUS_TIMEOUT | wait site in the plan's status word, raises the CTA's abort flag, and every role returns
through its normal exit (copies in flight drained with a bounded wait, TMEM freed). Nothing traps, faults or
spins without a limit. The test runs in a child process because the package binds one library per process.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

WAITTEST_FLAGS = ("-DKD_TEST_DROP_LOAD", "-DKD_WAIT_LIMIT_NS=20000000ull")

CHILD = r"""
import os, sys
sys.path.insert(0, %(root)r)
import numpy as np, torch
from kerneldev_b200 import _capi, flash_attention
from kerneldev_b200 import plan as plan_module
from oracle import attention_oracle as ao
assert "waittest" in str(_capi.LIB_PATH)
dev = torch.device("cuda:0")
B, H, T, D = %(shape)s
g = torch.Generator().manual_seed(5)
q, k, v = (torch.randn((B, H, T, D), generator=g).to(torch.bfloat16).to(dev) for _ in range(3))

os.environ["KD_TEST_DROP_LOAD"] = "0"
flash_attention(q, k, v, causal=True)                  # warm-up: the first launch on a cold GPU loads the module and ramps the clocks
torch.cuda.synchronize()
assert next(iter(plan_module._CACHE.values())).status() == 0
os.environ["KD_TEST_DROP_LOAD"] = "1"
o_bad = flash_attention(q, k, v, causal=True)          # returns: the failure is on the device
torch.cuda.synchronize()                               # the kernel ended by itself
plan = next(iter(plan_module._CACHE.values()))        # the plan the call above built; get_plan() would already raise
raw = int(plan._status_host[0]) & 0xFFFFFFFF
# whichever wait on the starved chain ran out first: an issuer's for the K tile (0x104), a softmax warp's for the scores (0x107), the
# producer's for the tile's stage (0x102)
assert raw in [_capi.KD_STATUS_TIMEOUT | site for site in (0x104, 0x107, 0x102)], hex(raw)
os.environ["KD_TEST_DROP_LOAD"] = "0"
try:
    flash_attention(q, k, v, causal=True)              # the next call on the plan raises, without a sync of its own
    raise SystemExit("no exception")
except RuntimeError as e:
    assert "timed out" in str(e) and any(site in str(e) for site in ("0x104", "0x107", "0x102")), str(e)
assert plan.status() == 0                              # reported once, then cleared on the device too
o = flash_attention(q, k, v, causal=True)              # and the device is still usable and correct
torch.cuda.synchronize()
ref, _ = ao.attention_forward(q.cpu(), k.cpu(), v.cpu(), ao.dense_mask(T, causal=True))
err = (o.float().cpu() - ref).abs()
assert bool((err <= 2e-2 + 1e-2 * ref.abs()).all()), float(err.max())
print("unwound and recovered")
"""


# both forward kernels; items of one query tile (4 pairs of tiles) and of two with work for both (80 pairs, four tiles each)
@pytest.mark.parametrize("shape", [(1, 2, 384, 64), (2, 20, 512, 64), (1, 2, 384, 128), (2, 20, 512, 128)])
def test_wait_timeout_unwinds_reports_and_recovers(shape):
    from kerneldev_b200.build import build
    lib = build(name="waittest", extra_flags=WAITTEST_FLAGS)
    env = dict(os.environ, KD_LIB_PATH=str(lib))
    env.pop("KD_CHECK_STATUS", None)     # the default, asynchronous reporting is what is under test
    r = subprocess.run([sys.executable, "-c", CHILD % {"root": ROOT, "shape": shape}], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "unwound and recovered" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]


CHILD_BACKWARD = r"""
import os, sys
sys.path.insert(0, %(root)r)
import torch
from kerneldev_b200 import _capi, flash_attention
from kerneldev_b200 import plan as plan_module
assert "waittest" in str(_capi.LIB_PATH)
dev = torch.device("cuda:0")
B, H, T, D = %(shape)s
q, k, v, do = (torch.randn((B, H, T, D), device=dev).to(torch.bfloat16) for _ in range(4))
x = [t.requires_grad_() for t in (q, k, v)]
os.environ["KD_TEST_DROP_LOAD"] = "0"

def gradients(deterministic, drop=0):
    o = flash_attention(*x, causal=True, deterministic=deterministic)
    os.environ["KD_TEST_DROP_LOAD"] = str(drop)
    try:
        return torch.autograd.grad(o, x, do)
    finally:
        os.environ["KD_TEST_DROP_LOAD"] = "0"

def same(a, b):   # fused dQ: fp32 sums in no fixed order, then a rounding (2^-8 covers bf16's, of any element)
    return all(torch.equal(s, t) or float((s.float() - t.float()).norm()) <= 2.0**-8 * float(t.float().norm()) for s, t in zip(a, b))

want = [gradients(det) for det in (False, True)]
torch.cuda.synchronize()
(plan,) = plan_module._CACHE.values()
assert plan.status() == 0
# what is left out, in which backward, and the kernel whose waits run out
for drop, deterministic, kernel in ((3, False, 0x400), (4, False, 0x400), (3, True, 0x400), (4, True, 0x400), (2, True, 0x200)):
    gradients(deterministic, drop)                     # returns: the failure is on the device
    torch.cuda.synchronize()                           # the kernel ended by itself
    raw = int(plan._status_host[0]) & 0xFFFFFFFF
    assert raw & _capi.KD_STATUS_TIMEOUT and (raw & 0xFF00) == kernel, (drop, deterministic, hex(raw))
    try:
        gradients(deterministic)                       # the next call on the plan raises, without a sync of its own
        raise SystemExit("no exception")
    except RuntimeError as e:
        assert "timed out" in str(e), str(e)
    assert plan.status() == 0                          # reported once, then cleared on the device too
    for det in (False, True):                          # and the device is still usable and correct
        got = gradients(det)
        torch.cuda.synchronize()
        assert plan.status() == 0 and same(got, want[det]), (drop, deterministic, det)
print("unwound and recovered")
"""


# the fused backward with and without its dQ, and the dQ kernel, at both tile widths; CTAs of one item (6 key tiles) and of several (320)
@pytest.mark.parametrize("shape", [(1, 2, 384, 64), (2, 40, 512, 64), (1, 2, 384, 128), (2, 40, 512, 128)])
def test_wait_timeout_in_the_backward(shape):
    from kerneldev_b200.build import build
    lib = build(name="waittest", extra_flags=WAITTEST_FLAGS)
    env = dict(os.environ, KD_LIB_PATH=str(lib))
    env.pop("KD_CHECK_STATUS", None)
    r = subprocess.run([sys.executable, "-c", CHILD_BACKWARD % {"root": ROOT, "shape": shape}], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "unwound and recovered" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]


CHILD_EARLY_START = r"""
import ctypes, os, sys
sys.path.insert(0, %(root)r)
import torch
from kerneldev_b200 import _capi, flash_attention
from kerneldev_b200 import plan as plan_module
assert "waittest" in str(_capi.LIB_PATH)
busy = _capi.load().kd_test_busy
busy.argtypes = [ctypes.c_uint64, ctypes.c_void_p]
dev = torch.device("cuda:0")
for D in (64, 128):
    q, k, v = (torch.randn((1, 4, 384, D), device=dev).to(torch.bfloat16) for _ in range(3))
    want = [flash_attention(q, k, v, causal=True) for _ in range(2)][1]   # the stream has used the plan: the next launch looks it up early
    torch.cuda.synchronize()
    assert busy(100_000_000, torch.cuda.current_stream().cuda_stream) == 0
    got = flash_attention(q, k, v, causal=True)
    torch.cuda.synchronize()
    assert all(p.status() == 0 for p in plan_module._CACHE.values())
    assert torch.equal(got, want)
print("no time-out")
"""


def test_waits_do_not_run_while_the_kernel_ahead_does():
    """A kernel of the caller's that lets its successor start at once and goes on for 100 ms, five times the wait limit of the
    test build: the forward's CTAs are resident all that time and must not count it against their waits."""
    from kerneldev_b200.build import build
    lib = build(name="waittest", extra_flags=WAITTEST_FLAGS)
    env = dict(os.environ, KD_LIB_PATH=str(lib))
    env.pop("KD_CHECK_STATUS", None)
    r = subprocess.run([sys.executable, "-c", CHILD_EARLY_START % {"root": ROOT}], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "no time-out" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]
