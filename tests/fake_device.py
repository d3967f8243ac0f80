"""The library's host code on a machine without a GPU: its objects linked with
fake_cudart.c, whose kernel launches are counted and do nothing.  Tests use
it for what the host decides: which launches a call makes, what is allocated
and uploaded, and what a failed allocation leaves behind."""
import contextlib
import ctypes as C
import functools
import os
import shutil
import subprocess
import tempfile

import pytest

from seismod_b200 import _lib as L

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "seismod_b200")


def build(out_dir):
    """The library linked with the fake runtime; only its own entry points and
    the fake's are visible, so nothing is shared with the real library."""
    if not shutil.which("make") or not os.path.exists(os.path.join(PKG, "Makefile")):
        pytest.skip("no build tools")
    made = subprocess.run(["make", "-s", "-C", PKG, os.path.join(PKG, "libseismod_gpu.so")],
                          capture_output=True, text=True)
    if made.returncode:
        pytest.skip("library objects cannot be built here")
    objs = sorted(os.path.join(PKG, "_build", f) for f in os.listdir(os.path.join(PKG, "_build"))
                  if f.endswith(".o"))
    script = os.path.join(out_dir, "visible.map")
    with open(script, "w") as f:
        f.write("{ global: sm_*; fake_*; local: *; };\n")
    fake = os.path.join(out_dir, "fake.o")
    lib = os.path.join(out_dir, "libseismod_fake.so")
    cuda = os.environ.get("CUDA", "/usr/local/cuda")
    subprocess.run(["gcc", "-O1", "-fPIC", "-I" + os.path.join(cuda, "include"), "-c",
                    os.path.join(HERE, "fake_cudart.c"), "-o", fake], check=True)
    subprocess.run(["g++", "-shared", "-o", lib, *objs, fake, "-Wl,--version-script=" + script,
                    "-lm", "-lpthread"], check=True)
    return lib


@functools.lru_cache(maxsize=None)
def _loaded():
    with tempfile.TemporaryDirectory() as d:
        return Fake(build(d))   # (a loaded library outlives its file)


@pytest.fixture
def fake():
    """The library on a fake CUDA runtime, loaded once (import it into the
    module that uses it)."""
    return _loaded()


class Fake:
    def __init__(self, path):
        self.lib = lib = C.CDLL(path)
        for name, (res, args) in L._SIGS.items():
            fn = getattr(lib, name)
            fn.restype, fn.argtypes = res, args
        lib.fake_launch.restype = C.c_char_p
        for f in (lib.fake_mallocs, lib.fake_uploads, lib.fake_upload_bytes, lib.fake_live_bytes):
            f.restype = C.c_long

    @contextlib.contextmanager
    def device(self):
        """The api module's handles come from the fake library inside."""
        old, L._LIB = L._LIB, self.lib
        self.lib.sm_pool_set_limit(0, C.c_size_t(0))   # no cached blocks: every handle allocates
        try:
            yield self
        finally:
            self.lib.fake_fail_malloc(0, 0)
            L._LIB = old

    def clear(self):
        self.lib.fake_clear()

    def fail_malloc(self, skip, count=1):
        self.lib.fake_fail_malloc(skip, count)

    def launches(self):
        """[(kernel name, grid x y z, block x y z)] since clear()"""
        out = []
        for k in range(self.lib.fake_launches()):
            gb = (C.c_uint * 6)()
            name = self.lib.fake_launch(k, gb)
            out.append((name.decode(),) + tuple(gb))
        return out

    def watch(self, name, arg):
        self.lib.fake_watch(name.encode(), arg)

    def watched(self):
        buf = (C.c_uint64 * 16)()
        self.lib.fake_watched(buf)
        return list(buf)
