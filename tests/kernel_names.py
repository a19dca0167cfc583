"""Names of the kernels that a call launches (torch's profiler, CUPTI activity records)."""
import re
import time

import pytest


def launched(run, family: str = r"\baa_\w+_kernel\b", tries: int = 6) -> list[str]:
    """The names among `family` of the kernels that `run()` launches (it launches some).  Records
    get lost now and then, so where none of the family is there `run()` is traced again; a process
    that gets none at all (another tracing tool holds them) skips the test."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    for k in range(tries):
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            run()
            torch.cuda.synchronize()
            time.sleep(0.05 * k)
        names = [e.name for e in p.events() if re.search(family, e.name)]
        if names:
            return names
    pytest.skip("the profiler records no kernels in this process")
