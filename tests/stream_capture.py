"""Stream capture through the driver API, for calls that a capture refuses and
for graphs that are replayed after the captured call has returned
(torch.cuda.graph keeps its allocator's private pool behind a capture that
fails)."""
import ctypes as C

import torch


def driver(name, *args):
    return getattr(C.CDLL("libcuda.so.1"), name)(*args)


def clear_error():
    """The runtime's last error of this thread, which a refused call leaves set."""
    C.CDLL("libcudart.so.13").cudaGetLastError()


class Capture:
    """`with Capture(stream) as c:` captures what is queued on the stream;
    c.status is 0 when the capture ended well, and c.replay() runs its graph."""

    def __init__(self, stream):
        self.stream = C.c_void_p(stream.cuda_stream)
        self.graph = C.c_void_p()
        self.exe = C.c_void_p()
        self.status = None

    def __enter__(self):
        torch.cuda.synchronize()
        assert driver("cuStreamBeginCapture_v2", self.stream, 2) == 0   # relaxed: this stream only
        return self

    def __exit__(self, *exc):
        self.status = driver("cuStreamEndCapture", self.stream, C.byref(self.graph))

    def replay(self):
        if not self.exe:
            assert self.status == 0
            assert driver("cuGraphInstantiateWithFlags", C.byref(self.exe), self.graph, C.c_ulonglong(0)) == 0
        assert driver("cuGraphLaunch", self.exe, self.stream) == 0

    def close(self):
        torch.cuda.synchronize()
        if self.exe:
            driver("cuGraphExecDestroy", self.exe)
        if self.graph:
            driver("cuGraphDestroy", self.graph)
        self.exe = self.graph = C.c_void_p()
