"""Names of the kernels a call launches (the CUDA activity trace of
torch.profiler)."""
import warnings


def kernels(call):
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        with profile(activities=[ProfilerActivity.CUDA]) as trace:
            call()
            torch.cuda.synchronize()
    return [e.name for e in trace.events() if "(" in e.name]
