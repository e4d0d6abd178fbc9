"""A device memory pool with little room: allocations beyond it fail as they do
on a full device, in this process only and without filling the device."""
import contextlib
import ctypes as C


class _Location(C.Structure):
    _fields_ = [("type", C.c_int), ("id", C.c_int)]


class _Props(C.Structure):
    _fields_ = [("allocType", C.c_int), ("handleTypes", C.c_int), ("location", _Location),
                ("security", C.c_void_p), ("maxSize", C.c_size_t), ("usage", C.c_ushort),
                ("reserved", C.c_ubyte * 54)]


class SmallPool:
    """The current device's pool, replaced while it is entered; room(chunks)
    leaves about that many chunks of `chunk` bytes free in it."""

    def __init__(self, chunk: int, total: int = 64 << 20):
        self.cu = C.CDLL("libcuda.so.1")
        self.chunk, self.held = chunk, []
        props = _Props(allocType=1, location=_Location(1, 0), maxSize=total)  # pinned, device 0
        self.pool, self.old, self.dev = C.c_void_p(), C.c_void_p(), C.c_int()
        self._ok(self.cu.cuDeviceGet(C.byref(self.dev), 0))
        self._ok(self.cu.cuMemPoolCreate(C.byref(self.pool), C.byref(props)))
        keep = C.c_uint64(1 << 40)  # release threshold: what was freed stays in the pool
        self._ok(self.cu.cuMemPoolSetAttribute(self.pool, 4, C.byref(keep)))

    @staticmethod
    def _ok(rc):
        assert rc == 0, f"CUDA driver error {rc}"

    def _take(self):
        p = C.c_uint64()
        if self.cu.cuMemAllocFromPoolAsync(C.byref(p), C.c_size_t(self.chunk), self.pool, None):
            return False
        self.held.append(p.value)
        return True

    def _give(self):
        self._ok(self.cu.cuMemFreeAsync(C.c_uint64(self.held.pop()), None))

    @contextlib.contextmanager
    def room(self, chunks: int):
        while self._take():
            pass
        for _ in range(min(chunks, len(self.held))):
            self._give()
        self._ok(self.cu.cuStreamSynchronize(None))
        self._ok(self.cu.cuDeviceGetMemPool(C.byref(self.old), self.dev))
        self._ok(self.cu.cuDeviceSetMemPool(self.dev, self.pool))
        try:
            yield
        finally:
            self._ok(self.cu.cuDeviceSetMemPool(self.dev, self.old))

    def leaked(self):
        """Bytes of the pool that are neither free nor taken here."""
        self._ok(self.cu.cuCtxSynchronize())
        used = C.c_uint64()
        self._ok(self.cu.cuMemPoolGetAttribute(self.pool, 7, C.byref(used)))
        return used.value - len(self.held) * self.chunk

    def close(self):
        self._ok(self.cu.cuCtxSynchronize())
        while self.held:
            self._give()
        self._ok(self.cu.cuStreamSynchronize(None))
        self._ok(self.cu.cuMemPoolDestroy(self.pool))
