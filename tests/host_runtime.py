"""The library's host code on a stand-in for the CUDA runtime (no GPU).

`FakeRuntime` is the package's api module on a library made of librmd's objects
and tests/c_abi/fake_cudart.cpp: device memory is host memory and kernels do
nothing, so a test can follow the host's calls (`on`), make one fail, play the
device's part in the counters and see which work nobody has waited for."""
import contextlib
import ctypes as C
import gc
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
HOOK = C.CFUNCTYPE(C.c_int, C.c_char_p, C.c_void_p, C.c_size_t, C.c_void_p)
COUNTERS_SIZE, ERRORS, NUM_PATHS, PATHS_DONE, NUM_SAMPLES = range(5)
OUT_OF_MEMORY = 2  # cudaErrorMemoryAllocation


def build_fake(out_dir: Path) -> Path:
    from raymond_b200 import build as b

    nvcc = Path(b.NVCC)
    if not nvcc.exists() or shutil.which("g++") is None:
        pytest.skip("no CUDA toolkit or C++ compiler")
    b.build()
    objs = [str(o) for o in sorted(b.BUILD.glob("*.o"))]
    c_abi = ROOT / "tests" / "c_abi"
    fake, layout, lib = out_dir / "fake_cudart.o", out_dir / "counters_layout.o", out_dir / "librmd_host.so"
    inc = ["-I", str(b.CUDA / "include"), "-I", str(b.CSRC)]
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", *inc, "-c", str(c_abi / "fake_cudart.cpp"), "-o", str(fake)], check=True)
    subprocess.run([str(nvcc), *b.NVCC_FLAGS, "-c", str(c_abi / "counters_layout.cu"), "-o", str(layout)], check=True)
    subprocess.run(["g++", "-shared", "-o", str(lib), *objs, str(layout), str(fake), "-L", str(b.CUDA / "lib64"), "-lnvrtc", "-lz",
                    "-fopenmp", f"-Wl,-rpath,{b.CUDA / 'lib64'}", "-Wl,-Bsymbolic", "-Wl,--no-undefined"], check=True)
    return lib


class FakeRuntime:
    def __init__(self, path: Path):
        from raymond_b200 import api

        self.api, self.path = api, path
        self._saved = api._lib, api.LIB_PATH
        api._lib, api.LIB_PATH = None, path
        self.lib = api.lib()
        L = self.lib
        L.fake_allocated.restype = C.c_size_t
        L.fake_pending.restype, L.fake_pending.argtypes = C.c_ulonglong, [C.c_void_p]
        L.fake_set_capacity.argtypes = [C.c_size_t]
        L.fake_set_capturing.argtypes = [C.c_void_p, C.c_int]
        L.fake_counters_layout.restype, L.fake_counters_layout.argtypes = C.c_size_t, [C.c_int]
        L.fake_set_hook.argtypes = [C.c_void_p]
        L.fake_clear_arrays()
        self.layout = [L.fake_counters_layout(k) for k in range(5)]

    @contextlib.contextmanager
    def on(self, see):
        """Calls see(name, ptr, size, stream) before every runtime call; what it returns (an error code) fails the call."""
        hook = HOOK(lambda name, ptr, size, stream: see(name.decode(), ptr, size, stream) or 0)
        self.lib.fake_set_hook(C.cast(hook, C.c_void_p))
        try:
            yield
        finally:
            self.lib.fake_set_hook(None)

    def is_counters(self, name, size):
        return name == "cudaMemcpyAsync" and size == self.layout[COUNTERS_SIZE]

    def counter(self, base, field, bits=64):
        return (C.c_uint32 if bits == 32 else C.c_uint64).from_address(base + self.layout[field])

    def close(self):
        gc.collect()
        self.lib.fake_set_hook(None)
        self.lib.fake_set_capacity(180 << 30)
        self.api._lib, self.api.LIB_PATH = self._saved


_lib_path = None


@pytest.fixture
def fake(tmp_path_factory):
    """The api module on the stand-in runtime, for one test (its objects must not outlive it)."""
    global _lib_path
    if _lib_path is None:
        _lib_path = build_fake(tmp_path_factory.mktemp("host_runtime"))
    rt = FakeRuntime(_lib_path)
    yield rt
    rt.close()
