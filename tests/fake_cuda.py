"""The engine's library linked against a CUDA runtime without a device (fake_cudart.cpp), for tests
of what the host does: which buffers it makes, which graphs it captures, what it refuses."""
import ctypes as C
import os
import subprocess
import sys

import es_sieve
from conftest import PKG, ROOT

OBJECTS = [os.path.join(PKG, "_build", o) for o in ("es_engine.o", "es_noalloc.o", "es_wheel.o", "es_digest.o")]


class FakeCuda:
    def __init__(self, folder):
        if not all(os.path.exists(o) for o in OBJECTS):
            sys.path.insert(0, ROOT)
            import __graft_entry__
            __graft_entry__.build()
        so = os.path.join(str(folder), "libes_fake.so")
        cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
        subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I" + cuda, "-o", so,
                        os.path.join(os.path.dirname(__file__), "fake_cudart.cpp")] + OBJECTS + ["-ldl", "-pthread"],
                       check=True)
        keep, es_sieve._lib = es_sieve._lib, None
        try:
            self.lib = es_sieve.load_library(so)
        finally:
            es_sieve._lib = keep
        self.lib.fake_log.restype = self.lib.fake_bytes.restype = C.c_size_t
        self.lib.fake_rates.argtypes = [C.c_double, C.c_double]
        self.lib.fake_counts.argtypes = [C.c_ulonglong, C.c_ulonglong]
        self.lib.fake_fail.argtypes = [C.c_long, C.c_long]

    def engine(self, monkeypatch, rates=(0.0, 0.0), **kw):
        monkeypatch.setattr(es_sieve, "load_library", lambda *a: self.lib)
        self.lib.fake_rates(*rates)
        e = es_sieve.Engine(**kw)
        self.log()
        return e

    def log(self):
        """The runtime's calls since the last look, a line each."""
        buf = C.create_string_buffer(1 << 20)
        out = ""
        while True:
            n = self.lib.fake_log(buf, len(buf))
            out += buf.raw[:n].decode()
            if n < len(buf):
                return out.splitlines()

    def fail(self, alloc=0, instantiate=0):
        self.lib.fake_fail(alloc, instantiate)

    def counts(self, surv=0, chunks=0):
        """What the next run is to report."""
        self.lib.fake_counts(surv, chunks)

    def bytes(self):
        return self.lib.fake_bytes()

    def bad(self):
        return self.lib.fake_bad()
