"""Downloads: through the context's pinned memory, straight to the caller's, and from several threads at once."""
import ctypes
import threading
import time

import numpy as np
import pytest

import hologram_b200 as hb
from hologram_b200 import kernel_call as kc
from hologram_b200.backend import lib

pytestmark = pytest.mark.gpu


def download(ws, host_ptr, nbytes):
    assert lib.holo_b200_workspace_download(ws._h, kc.rb(0), ctypes.c_void_p(host_ptr), nbytes) == 0


@pytest.mark.parametrize("nbytes", [1, 4099, 1 << 20, (1 << 20) + 1])
def test_threads_download_side_by_side(backend, nbytes):
    # the last size that passes through the context's memory and the first that does not; a thread that finds it taken does without
    def run(seed):
        try:
            data = np.random.default_rng(seed).integers(0, 256, nbytes, dtype=np.uint8)
            ws = hb.DeviceWorkspace(backend, 1)
            ws.put(0, data)
            for _ in range(100):
                got = np.empty(nbytes, np.uint8)
                download(ws, got.ctypes.data, nbytes)
                backend.synchronize()
                if not np.array_equal(got, data):
                    raise AssertionError(f"thread {seed}: other bytes")
            ws.close()
        except BaseException as e:       # noqa: B902 -- reported by the test's own thread
            wrong.append(e)

    wrong = []
    threads = [threading.Thread(target=run, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong


def test_pinned_memory_is_copied_to_as_it_is(backend):
    # 1 MiB: 35 us to pinned memory, 77 us to pageable memory; a detour through the context's own memory would cost the pinned one 75
    import torch
    nbytes = 1 << 20
    ws = hb.DeviceWorkspace(backend, 1)
    data = np.random.default_rng(0).integers(0, 256, nbytes, dtype=np.uint8)
    ws.put(0, data)
    best = {}
    for pinned in (False, True):
        host = torch.zeros(nbytes, dtype=torch.uint8, pin_memory=pinned)
        times = []
        for _ in range(100):
            t = time.perf_counter()
            download(ws, host.data_ptr(), nbytes)
            times.append(time.perf_counter() - t)
        assert np.array_equal(host.numpy(), data)
        best[pinned] = min(times)
    ws.close()
    assert best[True] < 0.75 * best[False], best
