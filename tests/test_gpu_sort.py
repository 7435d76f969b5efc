"""The sort's variants at their edges: all-pairs ranking up to 8,192 pairs, and digits of up to 11 bits over tiles
of 1,024 to 8,192 keys.  Whole numbers: bit-exact against numpy's stable sort, by the low key_bits bits."""
import numpy as np
import pytest
import torch

from metakonga_gb300 import dem
from metakonga_gb300._lib import call, ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 32, 33, 255, 1_023, 8_191, 8_192, 8_193, 9_999, 131_072, 131_073, 262_145, 524_288,
                               524_289, 1_300_001])
@pytest.mark.parametrize("bits", [1, 5, 11, 12, 21, 22, 23, 32])
def test_sort_sizes_and_bits(cuda, n, bits):
    rng = np.random.Generator(np.random.MT19937(n * 64 + bits))
    keys = rng.integers(0, 1 << 32, size=n, dtype=np.uint64).astype(np.uint32)
    low = np.uint32((1 << bits) - 1)
    keys[rng.integers(0, n, n // 4)] = keys[0]      # ties
    keys[n // 2:n // 2 + n // 8] = 0xFFFFFFFF       # and the largest key
    vals = rng.integers(0, 1 << 31, size=n).astype(np.uint32)
    dk, dv = (torch.from_numpy(a.view(np.int32).copy()).cuda() for a in (keys, vals))
    call("xd_radix_sort_pairs", ptr(dk), ptr(dv), n, bits, dem.stream_handle())
    torch.cuda.synchronize()
    order = np.argsort(keys & low, kind="stable")
    assert np.array_equal(dk.cpu().numpy().view(np.uint32), keys[order])
    assert np.array_equal(dv.cpu().numpy().view(np.uint32), vals[order])


@pytest.mark.parametrize("n", [4_097, 8_192, 200_003])
def test_one_key(cuda, n):
    """Every key the same: the order stays."""
    dk = torch.full((n,), 12_345, dtype=torch.int32, device="cuda")
    dv = torch.randint(0, 1 << 30, (n,), dtype=torch.int32, device="cuda")
    want = dv.clone()
    call("xd_radix_sort_pairs", ptr(dk), ptr(dv), n, 21, dem.stream_handle())
    assert torch.equal(dv, want) and bool((dk == 12_345).all())


@pytest.mark.parametrize("n", [8_000, 8_193])
def test_unaligned_cell_arrays(cuda, n):
    """Cell arrays that do not start on 16 bytes take the plain fill, and the error word starts at zero."""
    nc = 4_096
    rng = np.random.Generator(np.random.MT19937(n))
    keys = rng.integers(0, nc, n).astype(np.uint32)
    dk = torch.from_numpy(keys.view(np.int32).copy()).cuda()
    dv = torch.arange(n, dtype=torch.int32, device="cuda")
    cs, ce = (torch.full((nc + 1,), 9, dtype=torch.int32, device="cuda")[1:] for _ in range(2))
    so = torch.zeros(n, dtype=torch.int32, device="cuda")
    call("xd_reorder_and_find_cell_start", ptr(dk), ptr(dv), ptr(cs), ptr(ce), ptr(so), n, nc, dem.stream_handle())
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(so.cpu().numpy(), order)
    s = keys[order]
    start, end = np.searchsorted(s, np.arange(nc)), np.searchsorted(s, np.arange(nc), side="right")
    has = end > start
    assert np.array_equal(cs.cpu().numpy(), np.where(has, start, -1))
    assert np.array_equal(ce.cpu().numpy(), np.where(has, end, 0))
