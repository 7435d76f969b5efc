"""The reorder's error word is the calling thread's: calls on several threads and streams at once, some with a hash value
out of range, fail exactly where they should, and a thread's next call is not told of its last one's error."""
import threading

import pytest
import torch

from metakonga_gb300._lib import XdemError, call, ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 100, 9_000])
def test_errors_stay_with_their_call(cuda, n):
    wrong = []

    def work(t):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            idx = torch.arange(n, dtype=torch.int32, device="cuda")
            cs, ce = (torch.zeros(64, dtype=torch.int32, device="cuda") for _ in range(2))
            so = torch.zeros(n, dtype=torch.int32, device="cuda")
            for k in range(12):
                bad = (t + k) % 3 == 0
                keys = torch.full((n,), 5, dtype=torch.int32, device="cuda")
                keys[n // 2] = 70 if bad else 63
                try:
                    call("xd_reorder_and_find_cell_start", ptr(keys), ptr(idx), ptr(cs), ptr(ce), ptr(so), n, 64,
                         stream.cuda_stream)
                    failed = False
                except XdemError:
                    failed = True
                if failed != bad:
                    wrong.append((t, k, failed))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
