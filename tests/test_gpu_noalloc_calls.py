"""The allocation-free reorder allocates nothing, page-locked host memory included, on a thread that has not called it
before as well: no CUDA allocation is among the runtime calls that a profiler sees it make."""
import pytest
import torch

from metakonga_gb300._lib import XdemError, call, ptr

from .cuda_calls import runtime_calls

pytestmark = pytest.mark.gpu
ALLOCATIONS = ("Alloc", "Free", "HostRegister")


@pytest.mark.parametrize("n,bad", [(1, False), (5_000, True), (60_000, False)])
def test_a_thread_s_first_call_allocates_nothing(cuda, n, bad):
    ncell = 4_096
    keys = torch.randint(0, ncell, (n,), dtype=torch.int32, device="cuda")
    if bad:
        keys[n // 3] = ncell
    idx = torch.arange(n, dtype=torch.int32, device="cuda")
    cs, ce = (torch.zeros(ncell, dtype=torch.int32, device="cuda") for _ in range(2))
    so = torch.zeros(n, dtype=torch.int32, device="cuda")
    entry = "xd_reorder_and_find_cell_start_noalloc"
    call(entry, None, None, ptr(cs), ptr(ce), None, 0, ncell, 0)   # the device's set-up call
    torch.cuda.synchronize()
    got = []

    def work():
        try:
            call(entry, ptr(keys), ptr(idx), ptr(cs), ptr(ce), ptr(so), n, ncell, 0)
            got.append(False)
        except XdemError:
            got.append(True)

    names = runtime_calls(work)
    assert got and set(got) == {bad}
    assert any("Launch" in x for x in names), names     # the call's launches are among them
    assert not [x for x in names if any(a in x for a in ALLOCATIONS)], names
