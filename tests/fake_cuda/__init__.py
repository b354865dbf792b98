"""The library's host code over a CUDA runtime that launches nothing: its
objects linked with fake_cudart.cpp in place of the CUDA runtime."""
import importlib.util
import pathlib
import subprocess

HERE = pathlib.Path(__file__).resolve().parent
LIB_DIR = HERE.parent.parent / "cl-ops_gb300"


def load(out_dir):
    """A copy of the clops module bound to such a library, built in out_dir."""
    spec = importlib.util.spec_from_file_location("build_lib_fake", LIB_DIR / "build_lib.py")
    build_lib = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build_lib)
    build_lib.build()
    cuda = pathlib.Path(build_lib.nvcc()).resolve().parent.parent / "include"
    so = pathlib.Path(out_dir) / "libclops_fake.so"
    objects = [str(build_lib.BUILD / (s.name + ".o")) for s in build_lib.sources()]
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", f"-I{cuda}", "-o", str(so),
                    str(HERE / "fake_cudart.cpp"), *objects, "-ldl", "-lpthread", "-lrt",
                    "-Wl,-z,defs", "-Wl,-Bsymbolic"],
                   check=True, capture_output=True, text=True)
    text = (LIB_DIR / "clops.py").read_text()
    mod = type(importlib)("clops_fake")
    mod.__file__ = str(LIB_DIR / "clops.py")
    exec(compile(text.replace('LIB_PATH = HERE / "libclops.so"', f"LIB_PATH = pathlib.Path({str(so)!r})"),
                 mod.__file__, "exec"), mod.__dict__)
    return mod


def launches(mod):
    """(kernel name, grid, current device, the stream's device) of each
    launch since the last reset."""
    import ctypes as C
    mod.lib.fake_name.restype = C.c_char_p
    return [(mod.lib.fake_name(i).decode(), mod.lib.fake_grid(i), mod.lib.fake_device(i),
             mod.lib.fake_stream_device(i)) for i in range(mod.lib.fake_launches())]
