"""The library's host code without a GPU: its object files linked with a stand-in for the CUDA runtime
(fake_cuda_runtime.cpp) that records launches.  For tests of what the dispatch chooses, refuses and asks for."""
import ctypes
import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HERE = os.path.dirname(os.path.abspath(__file__))
OBJ_DIR = os.path.join(ROOT, "appmult-aware-retraining_b200", "build")

OK, E_BADARG, E_BITS, E_SCRATCH, E_TOOLARGE = 0, -1, -2, -4, -5
CODES_GIVEN, LEAST = 1, 2


def build(out_dir) -> str:
    import build_ext
    build_ext.build()
    if len(glob.glob(os.path.join(OBJ_DIR, "*.o"))) < len(build_ext._sources()):
        build_ext.build(force=True)
    path = os.path.join(str(out_dir), "host_dispatch.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-o", path, *sorted(glob.glob(os.path.join(OBJ_DIR, "*.o"))),
                    os.path.join(HERE, "fake_cuda_runtime.cpp"), "-I", os.path.join(cuda, "include"), "-Wl,-Bsymbolic"],
                   check=True)
    return path


class Library:
    """ctypes view of the linked library; `p` stands for any valid device pointer."""

    p = ctypes.c_void_p(1 << 40)

    def __init__(self, path):
        self.lib = ctypes.CDLL(path)
        self.lib.fake_name.restype = ctypes.c_char_p
        self.lib.fake_size.restype = ctypes.c_ulonglong
        for name in re.findall(r"size_t (lutgemm_\w+)\(", open(os.path.join(ROOT, "include", "lutgemm.h")).read()):
            getattr(self.lib, name).restype = ctypes.c_size_t

    def call(self, name, *args):
        """(status, [(kernel or "memset", grid x or bytes), ...]) of one entry point; ints above 32 bits are sizes."""
        self.lib.fake_reset()
        conv = [ctypes.c_size_t(a) if isinstance(a, Size) else ctypes.c_float(a) if isinstance(a, float) else a for a in args]
        rc = getattr(self.lib, name)(*conv)
        names = []
        for i in range(self.lib.fake_calls()):
            mangled = self.lib.fake_name(i).decode()
            words = re.findall(r"\d+([a-z_]+_kernel)", mangled)
            names.append((words[0] if words else mangled, self.lib.fake_size(i, 0)))
        return rc, names

    def query(self, name, *args):
        return getattr(self.lib, name)(*args)


class Size(int):
    """An argument of type size_t."""
