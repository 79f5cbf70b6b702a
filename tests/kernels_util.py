"""Names of the kernels that a call launches, so that a test of a family of kernels can say that it reached it."""
import re

import pytest
import torch
from torch.profiler import ProfilerActivity, profile


def kernels_of(fn):
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        out = fn()
        torch.cuda.synchronize()
    names = {e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA}
    if not names:
        pytest.skip("the profiler records no kernels here")
    return out, names


def launched(names, pattern):
    return any(re.search(pattern, n) for n in names)
