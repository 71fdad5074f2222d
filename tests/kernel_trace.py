"""Names of the kernels and copies a call launches (the CUDA activity trace of
torch.profiler).  In a process that has run for a while the tracer misses the
first launch of a region: kernels of torch's go before the call, and one after
it, and both have to show."""
import time
import warnings


def kernels(call):
    import torch
    from torch.profiler import ProfilerActivity, profile
    other = torch.zeros(1 << 20, device="cuda")
    torch.cuda.synchronize()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        with profile(activities=[ProfilerActivity.CUDA]) as trace:
            for work in (lambda: other.add_(1), lambda: other.add_(1), lambda: other.add_(1),
                         call, lambda: other.add_(1)):
                work()
                torch.cuda.synchronize()
                time.sleep(0.01)
    names = [e.name for e in trace.events() if "(" in e.name]
    assert sum("at::native" in n for n in names) >= 2, names
    return [n for n in names if "at::native" not in n]
