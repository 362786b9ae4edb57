"""Takes a device's free memory for a while, so that a test can see what a
call does where an allocation fails (it fails in the allocator, with an error:
nothing is accessed)."""
import contextlib
import ctypes

import torch

CHUNK = 2 << 20


@contextlib.contextmanager
def short_of_memory(leave: int = 0):
    """Allocates all free device memory but about `leave` bytes (whole 2 MB chunks)."""
    torch.cuda.init()
    rt = ctypes.CDLL("libcudart.so.12")   # the runtime torch has loaded
    held = []

    def take(size):
        p = ctypes.c_void_p()
        ok = rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0
        if ok:
            held.append((p, size))
        else:
            rt.cudaGetLastError()
        return ok

    try:
        size = 64 << 30
        while size >= CHUNK:
            if not take(size):
                size //= 2
        freed = 0
        while freed < leave and held:
            p, size = held.pop()
            rt.cudaFree(p)
            freed += size
        yield
    finally:
        for p, _ in held:
            rt.cudaFree(p)
