"""Which kernels a call launches: tests of a route check that it was taken."""

import torch


def kernels(fn):
    """What fn() returns, and the names of the kernels its second call launches."""
    fn()
    torch.cuda.synchronize()
    for _ in range(5):  # now and then a profile comes back without a single record: it is taken again
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            res = fn()
            torch.cuda.synchronize()
        names = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]
        if names:
            break
    return res, names
