"""Builds librtp_b200.so (all CUDA kernels of the package) for sm_100a with nvcc.

The library exposes a plain C ABI (see api.h) and is loaded with ctypes, so it does not link
against libtorch and cross-compiles on a machine without a GPU in a few seconds.
"""
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_DIR = os.path.join(os.path.dirname(HERE), "lib")
LIB_PATH = os.path.join(LIB_DIR, "librtp_b200.so")
SOURCES = ["gemm.cu", "gemm_local.cu", "kernels.cu", "attn_tc.cu", "flash_attn.cu", "ring_shift.cu", "gate_rope.cu", "im2col.cu", "noalloc.cu"]
# sources with many variants of a kernel, compiled in parts side by side: the macro that names a part, their number
PARTS = {"flash_attn.cu": ("RTP_FLASH_PART", 4)}
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--use_fast_math", "-Xcompiler", "-fPIC", "-Xcompiler", "-O3",
]


def _nvcc():
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found")
    return cand


def sources():
    return [os.path.join(HERE, s) for s in SOURCES if os.path.exists(os.path.join(HERE, s))]


def needs_build():
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    deps = [os.path.join(HERE, f) for f in os.listdir(HERE) if f.endswith((".cu", ".cuh", ".h"))]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    """Compile every .cu of the package into one shared library. Returns the library path."""
    if not force and not needs_build():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    nvcc = _nvcc()
    objs = []
    procs = []
    for src in sources():
        name = os.path.basename(src)
        macro, parts = PARTS.get(name, (None, 1))
        for part in range(parts):
            obj = os.path.join(LIB_DIR, f"{name}.{part}.o" if macro else name + ".o")
            cmd = [nvcc, *NVCC_FLAGS, *([f"-D{macro}={part}", "-diag-suppress", "177"] if macro else []), "-c", src, "-o", obj]
            if verbose:
                cmd[1:1] = ["-Xptxas", "-v"]
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
            objs.append(obj)
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode:
            sys.stderr.write(out)
        if p.returncode:
            raise RuntimeError(f"nvcc failed on {src}")
    cmd = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB_PATH, *objs, "-lcudart"]
    subprocess.check_call(cmd)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
