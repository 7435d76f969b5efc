"""Reorders on several threads at once, each on a stream of its own, with different sizes: every call's sorted keys, values and
cell ranges are numpy's, and releasing the workspace between rounds changes nothing."""
import threading

import numpy as np
import pytest
import torch

from metakonga_gb300._lib import call, ptr

pytestmark = pytest.mark.gpu
NCELL = 4_096


@pytest.mark.parametrize("sizes", [(100, 8_192, 3_000, 77), (8_193, 60_000, 131_072, 131_073)])
def test_results_stay_with_their_call(cuda, sizes):
    wrong = []

    def work(t):
        rng = np.random.Generator(np.random.MT19937(t))
        stream = torch.cuda.Stream()
        for k in range(8):
            n = sizes[(t + k) % len(sizes)]
            keys = rng.integers(0, NCELL, n).astype(np.int32)
            with torch.cuda.stream(stream):
                dk = torch.from_numpy(keys).cuda()
                dv = torch.arange(n, dtype=torch.int32, device="cuda")
                cs, ce = (torch.zeros(NCELL, dtype=torch.int32, device="cuda") for _ in range(2))
                so = torch.zeros(n, dtype=torch.int32, device="cuda")
                call("xd_reorder_and_find_cell_start", ptr(dk), ptr(dv), ptr(cs), ptr(ce), ptr(so), n, NCELL,
                     stream.cuda_stream)
                got = [x.cpu().numpy() for x in (dk, so, cs, ce)]
            order = np.argsort(keys, kind="stable")
            first = np.searchsorted(keys[order], np.arange(NCELL))
            last = np.searchsorted(keys[order], np.arange(NCELL), side="right")
            want = [keys[order], order, np.where(last > first, first, -1), np.where(last > first, last, 0)]
            if not all(np.array_equal(a, b) for a, b in zip(got, want)):
                wrong.append((t, k, n))

    for _ in range(2):
        threads = [threading.Thread(target=work, args=(t,)) for t in range(8)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        call("xd_release_workspace")
    assert not wrong
