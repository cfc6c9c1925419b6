"""Which kernels a call launches: tests of a route check that it was taken."""

import torch


def kernels(fn):
    """What fn() returns, and the names of the kernels its second call launches."""
    fn()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        res = fn()
        torch.cuda.synchronize()
    return res, [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]
