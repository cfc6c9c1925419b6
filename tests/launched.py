"""Which kernels a call launches: tests of a route check that it was taken."""

import torch


def kernels(fn):
    """What fn() returns, and the names of the kernels its second call launches."""
    fn()
    torch.cuda.synchronize()
    # Now and then the profiler hands back a trace without a single record, for reasons of its own.  Only such a trace is
    # taken again: one that has records, but not of the kernel the caller asks for, is returned as it is.
    for _ in range(5):
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            res = fn()
            torch.cuda.synchronize()
        names = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]
        if names:
            return res, names
    raise RuntimeError("five profiles in a row without a record")
