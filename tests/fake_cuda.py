"""The library's host code on tests/cpp/fake_cudart.cpp: a copy of the library linked from its own objects, for tests of
allocations, error exits and fallbacks that no GPU has to fail for."""
import ctypes as C
import os
import subprocess

from sirius_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
OUT_OF_MEMORY, INVALID_VALUE, NOT_SUPPORTED = 2, 1, 801  # cudaError_t


def link(folder):
    """The path of the library linked with the fake runtime, in `folder`."""
    objs = [os.path.join(build.HERE, "_build", os.path.basename(s) + ".o") for s in build.sources()]
    build.build(force=not all(os.path.exists(o) and os.path.getmtime(o) >= os.path.getmtime(s)
                              for o, s in zip(objs, build.sources())))
    lib = os.path.join(folder, "libsirius_fake.so")
    # (bound to its own runtime, whatever else the process has loaded)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", "/usr/local/cuda/include",
                    os.path.join(HERE, "cpp", "fake_cudart.cpp"), *objs, "-o", lib, "-lz"], check=True)
    return lib


class Fake:
    """The fake runtime's controls and counts."""

    def __init__(self, path):
        self.lib = C.CDLL(path)
        for n in ("calls", "launches"):
            getattr(self.lib, "fake_" + n).argtypes = [C.c_char_p]
        for n in ("calls", "launches", "device_bytes", "pinned", "streams", "events", "pending", "pending_own"):
            getattr(self.lib, "fake_" + n).restype = C.c_long
        self.lib.fake_fail.argtypes = [C.c_char_p, C.c_long, C.c_int]
        self.lib.fake_hook.argtypes = [C.c_char_p, C.c_int, C.c_int]

    def reset(self):
        self.lib.fake_reset()

    def fail(self, name, nth=1, error=OUT_OF_MEMORY):
        self.lib.fake_fail(name.encode(), nth, error)

    def hook(self, kernel, arg, value):
        self.lib.fake_hook(kernel.encode(), arg, value)

    def sync_ms(self, ms):
        self.lib.fake_sync_ms(ms)

    def major(self, version):
        """The device's compute capability, first number."""
        self.lib.fake_major(version)

    def wait(self):
        """As a caller that waits for its own (the legacy default) stream."""
        self.lib.cudaStreamSynchronize(None)

    def calls(self, name):
        return self.lib.fake_calls(name.encode())

    def launches(self, part):
        return self.lib.fake_launches(part.encode())

    def __getattr__(self, name):  # device_bytes, pinned, streams, events, pending, pending_own
        return getattr(self.lib, "fake_" + name)()


def link_without_tensor_maps(folder):
    """The library on the real runtime, but as on a driver that encodes no tensor maps; None where it cannot be linked."""
    objs = [os.path.join(build.HERE, "_build", os.path.basename(s) + ".o") for s in build.sources()]
    runtime = "/usr/local/cuda/lib64/libcudart_static.a"
    if not all(os.path.exists(p) for p in objs + [runtime]):
        return None
    stub, lib = os.path.join(folder, "no_maps.cpp"), os.path.join(folder, "libsirius_no_maps.so")
    with open(stub, "w") as f:
        f.write('extern "C" int __wrap_cudaGetDriverEntryPoint(const char*, void**, unsigned long long, void*) '
                "{ return %d; }\n" % NOT_SUPPORTED)
    subprocess.run(["g++", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-Wl,--wrap=cudaGetDriverEntryPoint", stub, *objs,
                    runtime, "-o", lib, "-lz", "-ldl", "-lrt", "-lpthread"], check=True)
    return lib
