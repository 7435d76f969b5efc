"""The CUDA runtime calls that a function makes, as a profiler sees them."""
import threading

import pytest
import torch


def runtime_calls(f, before=lambda: None, threads=1):
    """Names of the runtime calls of f(), made on `threads` new threads in turn; before() comes ahead of the recording.
    A profiler's first sessions can come back empty, and the synchronisation at the end shows whether one has: it is
    taken again then."""
    for _ in range(6):
        before()
        torch.cuda.synchronize()
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            for _ in range(threads):
                t = threading.Thread(target=f)
                t.start()
                t.join()
            torch.cuda.synchronize()
        names = [e.name for e in prof.events() if e.name.startswith("cuda")]
        if "cudaDeviceSynchronize" in names:
            return names
    pytest.skip("the profiler recorded no CUDA runtime calls")
