"""The sort's scratch never gets smaller with more keys: a scene makes it for all its particles and triangles, and sorts
fewer with an emitter, or the particles alone on a grid of their own."""
import ctypes

from metakonga_gb300 import _lib


def _bytes():
    f = getattr(_lib.lib(), "_ZN2xd24radix_sort_scratch_bytesEj")   # xd::radix_sort_scratch_bytes(unsigned)
    f.argtypes, f.restype = [ctypes.c_uint], ctypes.c_size_t
    return f


def _own(n):
    """What a sort of exactly n keys uses: two alternate arrays, 2,048 digit counts a tile, the digits' totals."""
    tile = 1024 if n <= 1 << 17 else 2048 if n <= 1 << 18 else 4096 if n <= 1 << 19 else 8192
    up = lambda b: (b + 255) // 256 * 256
    return 2 * up(4 * n) + 4 * 2048 * -(-n // tile) + 4 * 2048


def test_scratch_never_falls():
    f = _bytes()
    last = 0
    for n in range(1, (1 << 21) + 1):
        b = f(n)
        assert b >= last, n
        last = b
    assert f((1 << 32) - 1) >= f(1 << 31) >= last


def test_scratch_holds_every_smaller_sort():
    f = _bytes()
    edges = sorted({max(1, (1 << k) + d) for k in range(10, 22) for d in (-1, 0, 1)} | {112_641, 130_000, 150_000, 200_000})
    for n in edges:
        for m in edges:
            if m <= n:
                assert f(n) >= _own(m), (n, m)
