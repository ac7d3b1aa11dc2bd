"""The kernels a call launches, by name, as torch's profiler sees them."""
import time
from typing import Callable, List

import pytest


def kernels_of(call: Callable[[], object]) -> List[str]:
    """The names of the device's activities during `call`, which may run more than
    once: the profiler drops what its clock puts outside the session, so the call
    has room on both sides and is repeated where nothing was seen."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    for attempt in range(8):
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            time.sleep(0.05 * (attempt + 1))
            call()
            torch.cuda.synchronize()
            time.sleep(0.05 * (attempt + 1))
        names = [e.name for e in p.events() if e.device_type.name == "CUDA"]
        if names:
            return names
    pytest.skip("the profiler sees no kernels here")
