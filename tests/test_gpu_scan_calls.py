"""The scan's calls and the host words in which they report an expired wait: many
threads at once, more than there are words, and calls before and after the device's
context was reset, which frees the words."""
import ctypes as C
import subprocess
import sys
import threading

import numpy as np
import pytest

from pbf_b200._lib import LIB_PATH, check, lib

pytestmark = pytest.mark.gpu

RESET = """
import ctypes as C, sys
rt, pbf = C.CDLL("libcudart.so.12"), C.CDLL(sys.argv[1])
pbf.pbf_scan_workspace_bytes.restype = C.c_size_t
m = 100003
for _ in range(3):
    src, out, ws, total = C.c_void_p(), C.c_void_p(), C.c_void_p(), C.c_int(-1)
    size = pbf.pbf_scan_workspace_bytes(m)
    ok = [rt.cudaMalloc(C.byref(src), C.c_size_t(4 * m)), rt.cudaMalloc(C.byref(out), C.c_size_t(4 * m + 4)),
          rt.cudaMalloc(C.byref(ws), C.c_size_t(size)), rt.cudaMemset(src, 1, C.c_size_t(4 * m)),
          rt.cudaDeviceSynchronize(), pbf.pbf_scan_exclusive_i32(src, out, m, ws, C.c_size_t(size), None),
          rt.cudaMemcpy(C.byref(total), C.c_void_p(out.value + 4 * m), C.c_size_t(4), 2)]
    assert ok == [0] * 7, ok
    assert total.value == ((0x01010101 * m + 2**31) % 2**32) - 2**31, total.value
    assert rt.cudaDeviceReset() == 0
print("done")
"""


def test_scan_after_a_context_reset():
    """A process of its own, whose context is reset between its calls."""
    p = subprocess.run([sys.executable, "-c", RESET, LIB_PATH], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout.strip() == "done", (p.returncode, p.stdout, p.stderr)


def test_scans_of_many_threads_at_once():
    import torch
    threads, m = 80, 50_000
    a = torch.randint(0, 9, (threads, m), dtype=torch.int32, device="cuda")
    out = torch.empty((threads, m + 1), dtype=torch.int32, device="cuda")
    size = int(lib().pbf_scan_workspace_bytes(m))
    ws = torch.empty((threads, (size + 255) // 256 * 256), dtype=torch.uint8, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(threads)]
    torch.cuda.synchronize()
    start, failed = threading.Barrier(threads), []

    def work(i):
        start.wait()
        try:
            for _ in range(20):
                check(lib().pbf_scan_exclusive_i32(a[i].data_ptr(), out[i].data_ptr(), m, ws[i].data_ptr(),
                                                   C.c_size_t(size), int(streams[i].cuda_stream)))
        except Exception as e:
            failed.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not failed
    want = np.zeros((threads, m + 1), np.int32)
    want[:, 1:] = np.cumsum(a.cpu().numpy(), axis=1, dtype=np.int32)
    assert np.array_equal(out.cpu().numpy(), want)
