"""What a call launches and allocates on the device, from a profiler's record."""
import time

import pytest


def names_during(call, repeats=3):
    """Names of the kernels and runtime calls of `repeats` calls.  The record
    leaves out what its clocks place outside the profiled span, so the calls keep
    away from both ends.  Skips where another profiler holds the device's records
    and this one sees not even its own first kernel."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    first = torch.ones(1, device="cuda")
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        first.add_(1)
        torch.cuda.synchronize()
        time.sleep(0.05)
        for _ in range(repeats):
            call()
        torch.cuda.synchronize()
        time.sleep(0.05)
    names = [e.name for e in prof.events()]
    if not any("elementwise_kernel" in n for n in names):
        pytest.skip("kernel launches are not recorded here")
    return names
