"""The bounds-check build launches the kernels that the regular one launches, and its checks cover the V side's index lists
too: positions out of range are counted, their accesses left out, the other tokens' probabilities are what they would be."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, sys
import torch
from torch.profiler import ProfilerActivity, profile
sys.path.insert(0, {root!r})
from hqekv_b200 import _lib, synthetic
from hqekv_b200.quant.hqe_matmul import qkv_matmul_hqe_2
dev = torch.device("cuda:0")
checked = _lib.lib.hqkv_checks_enabled() == 1
def failures():
    n = ctypes.c_uint(0)
    _lib.check(_lib.lib.hqkv_check_failures(1, ctypes.byref(n)))
    return n.value
# query heads per kv head 4, 2, 1; groups 32, 64, 128; CTAs of one tier and of several
for batch, nh_q, nh_kv, ctx, group in ((1, 32, 8, 1064, 32), (2, 8, 4, 1320, 64), (1, 4, 1, 1320, 128), (1, 8, 8, 1064, 32),
                                       (80, 32, 8, 680, 32)):
    cfg = synthetic.CacheConfig("", batch, nh_q, nh_kv, 128, ctx, 40, (0.25, 0.5, 0.25), 0.0, group, True, 1, 0)
    cache, q = synthetic.build_cache(cfg, dev, seed=3)
    call = lambda c: qkv_matmul_hqe_2(q, c, None, 128, "uniform_group", group, group)
    weights, _ = call(cache)
    failures()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call(cache)
        torch.cuda.synchronize()
    names = sorted(e.key.split("(")[0] for e in p.key_averages() if "pass_kernel" in e.key)
    print("KERNELS", names)
    assert len(names) == 2 and failures() == 0
    if not checked:
        continue
    for bits, slot in ((8, 9), (4, 17), (2, 25)):       # positions of the V tiers
        bad, idx = list(cache), cache[slot].clone()
        lost = torch.cat((idx[:3], idx[-2:]))           # in a whole tile and in the last one
        idx[:3], idx[-2:] = 10 ** 6, cfg.context
        bad[slot] = idx
        w, out = call(tuple(bad))
        n = failures()
        assert n >= 5 * batch * nh_kv, (bits, n)
        keep = torch.ones(w.shape[-1], dtype=torch.bool, device=dev)
        keep[lost] = False
        assert torch.equal(w[..., keep], weights[..., keep]), bits
        assert torch.isfinite(out).all()
print("done")
"""


def child(library):
    env = dict(os.environ)
    if library:
        env["HQKV_LIB"] = library
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT)], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]
    return [line for line in r.stdout.splitlines() if line.startswith("KERNELS")]


def test_checked_build_runs_the_same_kernels(cuda_device):
    from hqekv_b200 import build
    lib = build.CHECKED_LIB_PATH
    if not os.path.exists(lib):
        lib = build.build(checks=True)
    assert child(lib) == child(None)
