"""The library's host code on a CPU: its objects linked with fake_cudart.cpp in
the CUDA runtime's place.  Images are not rendered; allocations, launches and
errors are what the host code makes of the device it is shown."""
import ctypes as C
import subprocess
from pathlib import Path

from cpp_volume_rendering_gb300 import abi, build, scene

HERE = Path(__file__).resolve().parent
CUDA = Path(build.NVCC).resolve().parents[1]


def load():
    lib = build.build()
    out = build.BUILD / "libcvr_fake.so"
    src = HERE / "fake_cudart.cpp"
    cu, cpp, _ = build._sources()
    objs = [build.BUILD / (s.stem + ".cu.o") for s in cu] + [build.BUILD / (s.stem + ".o") for s in cpp]
    if build._stale(out, [src, lib] + objs):
        build._run([build.CXX, "-O1", "-fPIC", "-std=c++17", "-shared", f"-I{CUDA / 'include'}", str(src)] +
                   [str(o) for o in objs] + ["-fopenmp", "-Wl,-Bsymbolic", "-o", str(out)])
    fake = abi.load(out)
    fake.fake_reset.argtypes, fake.fake_reset.restype = [C.c_size_t, C.c_size_t], None
    fake.fake_used.argtypes, fake.fake_used.restype = [], C.c_size_t
    fake.fake_refused.argtypes, fake.fake_refused.restype = [], C.c_int
    fake.fake_launches.argtypes, fake.fake_launches.restype = [C.c_char_p], C.c_int
    return fake


class Context(scene.Context):
    """A context on a device of `capacity` bytes."""

    def __init__(self, lib, capacity=280 << 30):
        lib.fake_reset(capacity, 1 << 62)
        self.lib = lib
        self.h = C.c_void_p()
        assert lib.cvr_create(C.byref(self.h), 0) == abi.CVR_OK
        self.dims = self.dtype = self.spacing = None

    def resize(self, capacity, largest=1 << 62):
        """Another capacity and largest free block; the counts of launches and
        refusals start over."""
        self.lib.fake_reset(capacity, largest)

    def launches(self, part):
        return self.lib.fake_launches(part.encode())
