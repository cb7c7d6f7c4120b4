"""Tests of what happens where the device has little room left."""
import contextlib


@contextlib.contextmanager
def device_room(torch, nbytes):
    """Device memory taken so that nbytes are left."""
    torch.cuda.empty_cache()
    taken = torch.cuda.caching_allocator_alloc(max(torch.cuda.mem_get_info()[0] - nbytes, 1))
    try:
        yield
    finally:
        torch.cuda.caching_allocator_delete(taken)
        torch.cuda.empty_cache()
