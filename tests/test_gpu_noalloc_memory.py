"""The solve without allocation takes no device memory after its first call on a
device, whatever the later channels' lengths: loading a kernel takes some, so
the first call loads them all.  Measured in a process of its own, where no other
test has loaded them."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = r"""
import ctypes, sys
import torch, ekpnp
from ekpnp import EkParams, lib
ekpnp.set_device(0)
# every power of two, mixed lengths, and a column too tall for the partitioned solve
sizes = [(256, 64)] + [(1 << k, 40) for k in range(1, 14) if k != 8] + [(96, 61), (1000, 257), (1021, 30), (64, 8190), (8, 9000)]
bufs = {s: [torch.zeros((s[1], s[0]), dtype=torch.float64, device="cuda:0") for _ in range(5)] for s in sizes}
torch.cuda.synchronize()
def call(s, efield):
    p = EkParams.from_dict(ekpnp.channel_params(*s, kappa_h=4.0, zeta=-1.5))
    ptrs = [ctypes.c_void_p(b.data_ptr()) for b in bufs[s]]
    if not efield:
        ptrs[3:] = [None, None]
    assert lib().ek_poisson_noalloc(ctypes.byref(p), *ptrs, None) == 0, s
    torch.cuda.synchronize()
call(sizes[0], False)
free = torch.cuda.mem_get_info()[0]
for s in sizes:
    call(s, True)
    now = torch.cuda.mem_get_info()[0]
    assert now >= free, (s, free - now)
"""


def test_no_memory_after_the_first_call():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.path.join(root, "ek-pnp_b200"))
    r = subprocess.run([sys.executable, "-c", PROGRAM], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
