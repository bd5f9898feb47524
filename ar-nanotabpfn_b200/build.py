"""Build libartab_b200.so (sm_100a only) next to this file.

    python ar-nanotabpfn_b200/build.py [--force]

nvcc cross-compiles without a GPU.  The library has no torch dependency: it is a
plain C-ABI shared object (see include/artab.h) loaded with ctypes.
"""
from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "libartab_b200.so")
# (source, object name, extra defines)
SOURCES = [(f, f[:-3], []) for f in ("api.cu", "dense_simt.cu", "attn_simt.cu", "attn_fma.cu", "attn_tc.cu", "buf_mma.cu", "noalloc.cu",
                                     "dense_tc.cu", "dense_fma.cu", "dense_mma.cu", "seq.cu")]
# the whole-sequence kernel has many variants: one compiler process per cache type and head size
SOURCES += [("seq_simt.cu", f"seq_simt_{'bf16' if b else 'f32'}_{dh}", [f"-DARTAB_SEQ_BF16={b}", f"-DARTAB_SEQ_DH={dh}"])
            for b in (0, 1) for dh in (16, 32, 64)]
FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "-I", os.path.join(ROOT, "include"), "-I", CSRC,
]


def _stale() -> bool:
    if not os.path.exists(OUT):
        return True
    t = os.path.getmtime(OUT)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(ROOT, "include", "artab.h"), __file__]
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return OUT
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    objs = []
    procs = []
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    newest = max(map(os.path.getmtime, [*headers, os.path.join(ROOT, "include", "artab.h"), __file__]))
    for src, name, defines in SOURCES:
        obj = os.path.join(HERE, "build", name + ".o")
        if not force and os.path.exists(obj) and os.path.getmtime(obj) > max(
                newest, os.path.getmtime(os.path.join(CSRC, src))):
            objs.append(obj)
            continue
        cmd = [nvcc, *FLAGS, *defines, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode:
            sys.stderr.write(out)
        if p.returncode:
            raise RuntimeError(f"nvcc failed on {src}")
    cmd = [nvcc, "-shared", "-o", OUT, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"]
    subprocess.check_call(cmd)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
