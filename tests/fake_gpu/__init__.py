"""The library's host code (front end, contexts, batches, serving) over stand-ins for the CUDA
runtime and the kernel launches: what the host does when an allocation fails or a pass does not
fit, without a GPU."""
import ctypes
import importlib
import os
import subprocess

from mytinygl_gb300 import gl as G

B = importlib.import_module("mytinygl_gb300.build")  # the package's `build` is its function
HERE = os.path.dirname(os.path.abspath(__file__))


def load():
    """(library, its controls): fake_totals, fake_log, fake_log_clear, fake_alloc_limit, fake_allocs."""
    B.build()
    out = os.path.join(HERE, "_build")
    os.makedirs(out, exist_ok=True)
    objs = [os.path.join(B.OBJ_DIR, f) for f in sorted(os.listdir(B.OBJ_DIR))
            if f.endswith(".c.o") or f in ("dev_runtime.cu.o", "dev_pipeline.cu.o", "dev_batch.cu.o")]
    for src in ("cudart.c", "kernels.cu"):
        obj = os.path.join(out, src + ".o")
        subprocess.run([B.nvcc_path()] + B.ARCH + ["-O1", "-Xcompiler", "-fPIC", f"-I{B.INCLUDE}", f"-I{B.DEV_DIR}", "-c",
                        os.path.join(HERE, src), "-o", obj], check=True, capture_output=True)
        objs.append(obj)
    path = os.path.join(out, "libmtgl_fake_gpu.so")
    subprocess.run(["g++", "-shared", "-o", path + ".tmp"] + objs + ["-Wl,-Bsymbolic", "-lm", "-lpthread"], check=True,
                   capture_output=True)
    os.replace(path + ".tmp", path)
    c = ctypes.CDLL(path)
    c.fake_log.restype = ctypes.c_char_p
    c.fake_allocs.restype = ctypes.c_long
    c.fake_alloc_limit.argtypes = [ctypes.c_size_t]
    c.fake_totals.argtypes = [ctypes.c_uint32, ctypes.c_uint32]
    return G.load(path), c
