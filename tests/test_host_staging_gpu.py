"""The staging area behind the host-buffer calls: its device workspace is given back when memory is short, and calls of several
threads take turns."""
import threading

import numpy as np
import pytest
import torch

import helix_b200 as hb
import oracle_lib as ol

pytestmark = pytest.mark.gpu


def _same(a, b):
    return np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_workspace_is_given_back_to_an_allocation_that_needs_it():
    w = np.random.default_rng(3).standard_normal((8192, 4096)).astype(np.float32)
    hb.quantize_host(w)                                     # leaves about 190 MB with the device
    free = torch.cuda.mem_get_info()[0]
    hog = torch.empty(free - (64 << 20), dtype=torch.uint8, device="cuda")
    buf = hb.DeviceBuffer(150 << 20)
    del hog, buf
    torch.cuda.empty_cache()
    small = w[:300, :1000]
    assert _same(hb.quantize_host(small), ol.quantize(np.ascontiguousarray(small)))


def test_calls_of_several_threads():
    rng = np.random.default_rng(4)
    ws = [(0.02 * rng.standard_normal((200 * (i + 1), 1000 + 4 * i))).astype(np.float32) for i in range(6)]
    want, bad = [ol.quantize(w) for w in ws], []

    def run(i):
        for _ in range(5):
            if not _same(hb.quantize_host(ws[i]), want[i]):
                bad.append(i)

    th = [threading.Thread(target=run, args=(i,)) for i in range(6)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
