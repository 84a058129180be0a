"""The library's host code on a CUDA runtime without a device (fake_cudart.cpp): the package's gpu module
over the compiled library object linked with the fake runtime, and the fake's log and failure plan.  No
kernel runs, so results mean nothing; what is tested is the order of the calls and what a failure leaves."""
import ctypes
import importlib.util
import os
import subprocess
import tempfile

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


class Fake:
    def __init__(self, lib):
        self.lib = lib
        lib.fake_fail.argtypes = [ctypes.c_char_p, ctypes.c_long, ctypes.c_int]
        lib.fake_log_size.restype = ctypes.c_long
        lib.fake_log_line.argtypes = [ctypes.c_long]
        lib.fake_log_line.restype = ctypes.c_char_p
        lib.fake_pin.argtypes = [ctypes.c_void_p, ctypes.c_size_t, ctypes.c_int]

    def reset(self):
        """Forget the log and every planned failure."""
        self.lib.fake_reset()

    def fail(self, call, nth, error=2):
        """The nth call from now on returns ``error`` (2: out of memory)."""
        self.lib.fake_fail(call.encode(), nth, error)

    def pin(self, address, size, read_only=False):
        """Memory that the device maps, one registration a call."""
        self.lib.fake_pin(address, size, int(read_only))

    def unpin_all(self):
        self.lib.fake_unpin_all()

    def log(self):
        return [self.lib.fake_log_line(i).decode() for i in range(self.lib.fake_log_size())]

    def calls(self, name):
        return [x for x in self.log() if x.split()[0] == name]


_loaded = None


def load():
    """(gpu module, Fake), built once per process."""
    global _loaded
    if _loaded is None:
        from nessi_b200 import build
        so = os.path.join(tempfile.mkdtemp(prefix="fake_cudart_"), "libnessi_fake.so")
        # -Bsymbolic: the library's calls stay inside, whatever CUDA runtime the process has loaded
        subprocess.check_call([build.CXX, "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", CUDA + "/include",
                               "-o", so, os.path.join(HERE, "fake_cudart.cpp"), build.build_object(), "-ldl", "-lpthread"])
        path = os.path.join(os.path.dirname(HERE), "nessi_b200", "gpu.py")
        spec = importlib.util.spec_from_file_location("nessi_b200._gpu_on_fake_runtime", path)
        mod = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(mod)
        mod.load_library(so)
        _loaded = mod, Fake(ctypes.CDLL(so))
    return _loaded
