"""Which kernels a call launches, from the profiler's activity records."""
import time


def launched(call, parts, tries=6):
    """Names of the kernels that `call` launches, recorded until one of them holds one of `parts`; None where the
    profiler records none.  Records close to the ends of its window may be lost, so the call has time before and
    after it and is repeated when its kernels are missing."""
    import torch
    for _ in range(tries):
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            torch.cuda.synchronize()
            time.sleep(0.03)
            call()
            torch.cuda.synchronize()
            time.sleep(0.03)
        names = {e.name for e in prof.events()}
        if any(p in n for p in parts for n in names):
            return names
    return None
