"""The library's host code over a CUDA runtime that runs nothing (fake_cudart.c): what a call would launch, with which
arguments, and what it does when a runtime call fails."""
import ctypes as C
import importlib.util
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
HOOK = C.CFUNCTYPE(C.c_int, C.c_char_p, C.c_char_p, C.c_void_p, C.c_void_p, C.c_size_t, C.c_void_p)


def load(directory):
    """Links the library's archive with the fake runtime and loads the result with the ABI's argument types."""
    from kairos_engine_b200 import _lib, build
    build.build()
    so = os.path.join(str(directory), "libsp_moe_fake.so")
    rt = os.path.join(str(directory), "fake_cudart.o")
    subprocess.run(["gcc", "-O1", "-fPIC", "-std=gnu11", "-I/usr/local/cuda/include", "-c", os.path.join(HERE, "fake_cudart.c"), "-o", rt], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-Wl,-z,defs", "-o", so, "-Wl,--whole-archive", build.ARCHIVE, "-Wl,--no-whole-archive", rt, "-ldl", "-lpthread"], check=True)
    spec = importlib.util.spec_from_file_location("fake_abi", _lib.__file__)      # a second copy of the loader, with its own path
    abi = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(abi)
    abi.LIB_PATH = so
    return Fake(abi)


class Launch:
    def __init__(self, name, grid, stream, words):
        self.name, self.grid, self.stream, self.words = name, grid, stream, words


class Fake:
    """L: the library. log: launches (Launch), copies ("memcpy", dst, src, bytes) and synchronisations ("sync", ...) in order.
    read: part of a kernel's name -> (argument, count): that many 8-byte words of the argument are kept as Launch.words, for
    as many launches. on_launch(launch) -> the error code the launch answers with."""

    def __init__(self, abi):
        self.abi, self.L, self.log, self.read, self.on_launch = abi, abi.lib(), [], {}, None
        self._hook = HOOK(self._told)                       # kept alive for as long as the library may call it
        self.L.fake_set_hook(self._hook)

    def _told(self, what, name, a, b, n, stream):
        if what != b"launch":
            self.log.append((what.decode(), a, b, n))
            return 0
        name, words = name.decode(), []
        for part, (arg, count) in self.read.items():
            if part in name:
                p = C.cast(a, C.POINTER(C.c_void_p))[arg]
                words = list(C.cast(p, C.POINTER(C.c_uint64 * count)).contents)
        launch = Launch(name, n, stream, words)
        self.log.append(launch)
        return int(self.on_launch(launch) or 0) if self.on_launch else 0

    def launches(self, part=""):
        return [x for x in self.log if isinstance(x, Launch) and part in x.name]

    def engine(self, cfg, n_layers=1, max_tokens=1, **kw):
        """An open handle whose layers count as uploaded (their bytes are never looked at)."""
        c = self.abi.SpMoeConfig(n_layers=n_layers, max_tokens=max_tokens, **cfg, **kw)
        h = C.c_void_p()
        assert self.L.sp_moe_open(C.byref(c), C.byref(h)) == 0, self.L.sp_last_error()
        E, NE, FFE, FFS = cfg["E"], cfg["NE"], cfg["FFE"], cfg["FFS"]
        blob = C.create_string_buffer(max(4 * NE * E, NE * 2 * FFE * E // 2, FFS * E // 2, 4 * FFS, 4096))
        w = self.abi.SpMoeLayerWeights(**{f: C.addressof(blob) for f, _ in self.abi.SpMoeLayerWeights._fields_})
        for layer in range(n_layers):
            assert self.L.sp_moe_upload_layer(h, layer, C.byref(w)) == 0
        self.log.clear()
        return h
