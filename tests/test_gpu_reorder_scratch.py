"""The reorder's scratch and error word are kept from call to call, whatever thread makes it, and given back by
xd_release_workspace: the CUDA calls that a profiler sees."""
import threading

import pytest
import torch

from metakonga_gb300._lib import call, ptr

pytestmark = pytest.mark.gpu


def _reorder(n=20_000, ncell=4_096):
    keys = torch.randint(0, ncell, (n,), dtype=torch.int32, device="cuda")
    idx = torch.arange(n, dtype=torch.int32, device="cuda")
    cs, ce = (torch.zeros(ncell, dtype=torch.int32, device="cuda") for _ in range(2))
    so = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return lambda: call("xd_reorder_and_find_cell_start", ptr(keys), ptr(idx), ptr(cs), ptr(ce), ptr(so), n, ncell, 0)


def _calls(f, threads=1):
    """The CUDA runtime calls of f, made on as many threads in turn."""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        for _ in range(threads):
            t = threading.Thread(target=f)
            t.start()
            t.join()
        torch.cuda.synchronize()
    return [e.name for e in prof.events() if e.name.startswith("cuda")]


def test_kept_over_threads_and_given_back(cuda):
    work = _reorder()
    call("xd_release_workspace")
    first = _calls(work)
    assert any("cudaHostAlloc" in x for x in first) and any("cudaMalloc" in x for x in first), first
    later = _calls(work, threads=3)
    assert any("Launch" in x for x in later)
    assert not [x for x in later if "Alloc" in x or "Free" in x], later
    back = _calls(lambda: call("xd_release_workspace"))
    assert any(x == "cudaFree" for x in back) and any("cudaFreeHost" in x for x in back), back
