"""Failure detection of the one-launch block without a GPU fault: a wait that cannot be satisfied must run out,
end the launch by itself, be reported through the workspace's status word and leave the CUDA context usable."""

import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_CHILD = r"""
import json, sys
sys.path.insert(0, {root!r})
import torch
from zmlx_b200 import _lib, synthetic
from zmlx_b200.layer import MoELayer

dev = "cuda:0"
cfg = synthetic.CONFIGS["c2"]
params = synthetic.make_layer(cfg, device=dev)
x = synthetic.make_tokens(cfg, 1, device="cpu").to(dev)
# debug hook: expert 0's router logit is never published, so every CTA's bounded wait for it runs out
bad = MoELayer(cfg, params, max_tokens=8, fused=True, debug_withhold_logit=True)
bad(x)
torch.cuda.synchronize()  # the launch must end by itself (about a second)
status = bad.fused_status(1)
raised = False
try:
    bad.check_status()
except _lib.ZmoeError as e:
    raised = e.code == _lib.ERR_TIMEOUT
cleared = bad.fused_status(1) == 0
# the context is still usable, and a healthy layer on the same device still gives finite results
usable = bool((torch.arange(8, device=dev) + 1).sum().item() == 36)
good = MoELayer(cfg, params, max_tokens=8, fused=True)
out = good(x)
good.check_status()
print(json.dumps({{"status": status, "raised": raised, "cleared": cleared, "usable": usable,
                  "finite": bool(torch.isfinite(out.float()).all())}}))
"""


def test_a_wait_that_runs_out_ends_the_launch_with_the_status_word_set():
    res = subprocess.run([sys.executable, "-c", _CHILD.format(root=ROOT)], capture_output=True, text=True,
                         timeout=600)
    assert res.returncode == 0, res.stderr[-2000:]
    rec = json.loads(res.stdout.strip().splitlines()[-1])
    assert rec["status"] == 1
    assert rec["raised"], "check_status() must map the status word to ZMOE_ERR_TIMEOUT"
    assert rec["cleared"] and rec["usable"] and rec["finite"]


_MATMUL = r"""
import json, sys
sys.path.insert(0, {root!r})
import torch
from zmlx_b200 import _lib, ops, quant, synthetic
from zmlx_b200.layer import MoELayer

dev, E, N, K, rows = "cuda:0", 3, 200, 512, 40
g = torch.Generator(device=dev).manual_seed(1)
w, s, b = quant.quantize_affine(torch.randn((E, N, K), generator=g, device=dev) * 0.02, 64)
x = torch.randn((rows, K), generator=g, device=dev).to(torch.bfloat16)
ids = (torch.arange(rows, device=dev) % E).to(torch.int32)
plan = ops.build_plan(ids, E)
ws = ops.qmm_workspace(rows, E, K, rows_hint=rows, mode="affine", device=dev)
lib, p = _lib.load(), ops._ptr


def call(flags):
    out = torch.zeros((rows, N), dtype=torch.bfloat16, device=dev)
    _lib.check(lib.zmoe_gather_qmm_ws(p(x), rows, K, p(w), p(s), p(b), E, N, K, 64, 0, p(plan), rows, rows, 1 | flags,
                                      p(out), *ops._ws_args(ws), ops._stream()))
    torch.cuda.synchronize()
    return out


def raises(check):
    try:
        check()
    except _lib.ZmoeError as e:
        return e.code == _lib.ERR_TIMEOUT
    return False


good = call(0)
ops.check_plan(plan)
bad = call(_lib.DEBUG_WITHHOLD_TOKENS)  # no token tile ever arrives: ends by itself, after about a second
ops.build_plan(ids, E, out=plan)  # the word outlives the next build
rec = {{"void": bool(bad.isnan().all()), "raised": raises(lambda: ops.check_plan(plan)),
       "cleared": not raises(lambda: ops.check_plan(plan)), "same": bool(torch.equal(call(0), good))}}
# a layer reports what its plans say, once
cfg = synthetic.CONFIGS["c3"].scaled(d_model=256, d_ff=256, n_experts=16)
layer = MoELayer(cfg, synthetic.make_layer(cfg, device=dev), max_tokens=16)
tokens = synthetic.make_tokens(cfg, 12, device=dev)
layer(tokens)
layer.check_status()
word = 0x5a4d5457  # what the kernel leaves (kPlanTimeout in csrc/common.cuh)
for i, plan_of in enumerate((lambda: layer.plan, lambda: layer._shared_plans[12])):
    plan_of()[2] = word
    layer(tokens)
    rec["layer%d" % i] = raises(layer.check_status) and not raises(layer.check_status)
print(json.dumps(rec))
"""


def test_a_matmul_wait_that_runs_out_is_reported_by_the_plan():
    res = subprocess.run([sys.executable, "-c", _MATMUL.format(root=ROOT)], capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stderr[-2000:]
    rec = json.loads(res.stdout.strip().splitlines()[-1])
    assert len(rec) == 6 and all(rec.values()), rec
