"""A device memory pool of limited size, current for a while: stream-ordered allocations beyond it fail as they do on a
full device (driver API through ctypes)."""
import contextlib
import ctypes as C


class _Props(C.Structure):
    _fields_ = [("alloc_type", C.c_int), ("handle_types", C.c_int), ("location_type", C.c_int), ("location_id", C.c_int),
                ("security", C.c_void_p), ("max_size", C.c_size_t), ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


@contextlib.contextmanager
def limited_pool(max_bytes, full=False):
    """full: nothing of it is left for anybody."""
    import torch

    cu = C.CDLL("libcuda.so.1")

    def call(name, *args):
        status = getattr(cu, name)(*args)
        assert status == 0, (name, status)

    torch.cuda.synchronize()
    device, old, pool = C.c_int(), C.c_void_p(), C.c_void_p()
    call("cuDeviceGet", C.byref(device), torch.cuda.current_device())
    call("cuDeviceGetMemPool", C.byref(old), device)
    props = _Props(alloc_type=1, location_type=1, location_id=device.value, max_size=max_bytes)  # pinned, on the device
    call("cuMemPoolCreate", C.byref(pool), C.byref(props))
    held = []
    call("cuDeviceSetMemPool", device, pool)
    try:
        size = max_bytes if full else 0
        while size >= 256:
            p = C.c_uint64()
            if cu.cuMemAllocFromPoolAsync(C.byref(p), C.c_size_t(size), pool, None) == 0:
                held.append(p)
            else:
                size //= 2
        torch.cuda.synchronize()
        yield
    finally:
        torch.cuda.synchronize()
        call("cuDeviceSetMemPool", device, old)
        for p in held:
            call("cuMemFreeAsync", p, None)
        torch.cuda.synchronize()
        call("cuMemPoolDestroy", pool)
