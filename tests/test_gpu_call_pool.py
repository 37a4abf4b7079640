"""Device memory that training and gradient calls leave behind: at most the
32 MiB that their pool keeps per device, whatever the size of the calls and
however many ran at once; and the calls work on after a device reset, which
takes the pool with its context."""
from __future__ import annotations

import subprocess
import sys
import threading

import numpy as np
import pytest

from icarion_b200 import ipm
from icarion_b200.sim import device_count

pytestmark = pytest.mark.gpu

KEEP = 32 << 20


@pytest.fixture(scope="module", autouse=True)
def _gpu():
    assert device_count() > 0, "these tests need a CUDA device"


def _free():
    import torch
    return torch.cuda.mem_get_info(0)[0]


def _call(n, gradients):
    x = np.zeros(2 * n, dtype=np.float32)
    y = np.zeros(n, dtype=np.float32)
    if gradients:
        ipm.gradients(ipm.init_params(3), x, y)
    else:
        ipm.train(x, y, params=ipm.init_params(3), epochs=1, batch=65536)


@pytest.mark.parametrize("gradients,n,threads", [(False, 16 << 20, 1), (False, 1 << 20, 6), (True, 1 << 20, 6)])
def test_large_calls_give_their_memory_back(gradients, n, threads):
    """(256 MB, 6 x 33 MB and 6 x 29 MB of workspace.)"""
    _call(65536, gradients)
    before = _free()
    ts = [threading.Thread(target=_call, args=(n, gradients)) for _ in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert before - _free() <= KEEP


def test_training_runs_after_a_device_reset():
    code = """
import ctypes, sys
import numpy as np
sys.path.insert(0, '.')
from icarion_b200 import ipm
rng = np.random.default_rng(1)
x = rng.uniform(-1, 1, (4096, 2)).astype(np.float32)
y = np.cos(x[:, 0]).astype(np.float32)
run = lambda: ipm.train(x.ravel(), y, params=ipm.init_params(3), epochs=3, batch=1024)[0]
cu = ctypes.CDLL('libcuda.so.1')
a = run()
for _ in range(2):
    assert cu.cuDevicePrimaryCtxReset_v2(0) == 0
    assert np.array_equal(a, run())
print('same')
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr
