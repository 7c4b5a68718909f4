"""Short device memory for the tests, without a context that runs out by itself."""
import contextlib

import torch


@contextlib.contextmanager
def memory_left(nbytes):
    """All but about nbytes of the device's free memory held by an allocation (not touched)."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = torch.empty(max(0, torch.cuda.mem_get_info()[0] - int(nbytes)), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()
