"""The synchronous calls of the learned building blocks and what surrounds them:
several threads at a time, a thread that ends while another captures a graph, and
a device reset between two calls (an error, not a crash)."""
import glob
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from test_learned_gpu import C, _conv, _ints, _wgrad

pytestmark = pytest.mark.gpu


def _case(seed):
    rng = np.random.default_rng(seed)
    x, W = _ints(rng, (1, 9, 70, 32)), _ints(rng, (32, 9, 32), 0.2)
    b = rng.integers(-3, 4, 32).astype(np.float64)
    return x, W, b


def test_many_threads_at_a_time(pmhd_lib):
    cases = [_case(k) for k in range(6)]
    refs = [(C.conv3x3(x, W, b), C.conv3x3_backward_weight(x, x)) for x, W, b in cases]
    errors = []

    def work(k):
        try:
            x, W, b = cases[k % 6]
            for _ in range(5):
                z, _ = _conv(pmhd_lib, pmhd_lib.CONV_GELU, x, W, b, 32)
                np.testing.assert_array_equal(z, refs[k % 6][0])
                dw, db = _wgrad(pmhd_lib, x, x)
                np.testing.assert_array_equal(dw, refs[k % 6][1][0])
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(24)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors[0]


def test_a_thread_that_ends_does_not_break_a_capture(pmhd_lib):
    import torch

    x, W, b = _case(7)
    called, end = threading.Event(), threading.Event()

    def work():
        _conv(pmhd_lib, pmhd_lib.CONV_GELU, x, W, b, 32)
        called.set()
        end.wait(60)

    v = torch.zeros(16, device="cuda")
    t = threading.Thread(target=work)
    t.start()
    assert called.wait(60)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):  # global capture mode
        v += 1
        end.set()
        t.join()
    g.replay()
    torch.cuda.synchronize()
    assert v.tolist() == [1.0] * 16


RESET = """
import ctypes, sys
sys.path.insert(0, %r)
import pmhd
cu = ctypes.CDLL(%r)
fp = ctypes.POINTER(ctypes.c_float)

def call():
    bufs = []
    for n in (2 * 64 * 4 * 32, 2 * 32 * 9 * 32, 4 * 32, 2 * 64 * 4 * 32, 2 * 64 * 4 * 32):
        p = ctypes.c_void_p()
        assert cu.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(n)) == 0
        assert cu.cudaMemset(p, 0, ctypes.c_size_t(n)) == 0
        bufs.append(p.value)
    x, w, b, o0, o1 = bufs
    return pmhd.load().pmhd_conv3x3(pmhd.CONV_GELU, x, 1, 4, 64, 32, w, ctypes.cast(b, fp), 32, None, o0, o1, None)

assert call() == pmhd.OK
assert cu.cudaDeviceReset() == 0
print("RESET_OK", call() in (pmhd.OK, pmhd.ERR_CUDA))
"""


def test_a_device_reset_is_an_error_not_a_crash(pmhd_lib):
    import torch

    found = glob.glob(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib", "libcudart.so.*"))
    found += glob.glob("/usr/local/cuda/lib64/libcudart.so.*")
    if not found:
        pytest.skip("no shared CUDA runtime")
    pkg = os.path.dirname(os.path.dirname(os.path.abspath(pmhd_lib.__file__)))
    r = subprocess.run([sys.executable, "-c", RESET % (pkg, found[0])], capture_output=True, text=True, timeout=120)
    assert "RESET_OK True" in r.stdout, (r.returncode, r.stdout, r.stderr)
