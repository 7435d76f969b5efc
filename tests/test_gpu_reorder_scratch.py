"""The reorder's scratch and error word are kept from call to call, whatever thread makes it, and given back by
xd_release_workspace: the CUDA calls that a profiler sees."""
import pytest
import torch

from metakonga_gb300._lib import call, ptr

from .cuda_calls import runtime_calls

pytestmark = pytest.mark.gpu


def _reorder(n=20_000, ncell=4_096):
    keys = torch.randint(0, ncell, (n,), dtype=torch.int32, device="cuda")
    idx = torch.arange(n, dtype=torch.int32, device="cuda")
    cs, ce = (torch.zeros(ncell, dtype=torch.int32, device="cuda") for _ in range(2))
    so = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return lambda: call("xd_reorder_and_find_cell_start", ptr(keys), ptr(idx), ptr(cs), ptr(ce), ptr(so), n, ncell, 0)


def test_kept_over_threads_and_given_back(cuda):
    work = _reorder()
    release = lambda: call("xd_release_workspace")
    first = runtime_calls(work, before=release)
    assert any("cudaHostAlloc" in x for x in first) and any("cudaMalloc" in x for x in first), first
    later = runtime_calls(work, threads=3)
    assert any("Launch" in x for x in later)
    assert not [x for x in later if "Alloc" in x or "Free" in x], later
    back = runtime_calls(release, before=work)
    assert any(x == "cudaFree" for x in back) and any("cudaFreeHost" in x for x in back), back
