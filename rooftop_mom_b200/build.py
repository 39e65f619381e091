"""Builds librtm.so in-tree for sm_100a (nvcc; no JIT cache).

    python -m rooftop_mom_b200.build          # or: from rooftop_mom_b200.build import build; build()
"""
from __future__ import annotations

import concurrent.futures
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "librtm.so")
OBJ = os.path.join(HERE, "_build")
SOURCES = ["runtime.cpp", "capi.cpp", "server.cpp", "grid.cu", "grid_fast.cu", "assembly.cu", "krylov.cu", "strip_solve.cu", "ops.cu", "excitation.cu", "fixed_scratch.cu", "fault.cu", "tune.cpp", "batch.cu"]
# Sources compiled once for each form, so that their kernels compile side by side: object name -> (source, defines).
# Without -lineinfo: a kernel's first launch in a process loads its whole unit, and the line tables of the unrolled
# codelets are three quarters of these (first product on 250 x 139 faces 27 ms with them, 7 without; librtm.so 84 MB, 41).
FORMS = {**{f"grid_reg.{k}": ("grid_reg.cu", [f"-DRTM_REG_FORM={k}"]) for k in range(8)},
         **{f"gen_reg.{k}": ("gen_reg.cu", [f"-DRTM_GEN_FORM={k}"]) for k in range(4)}}
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-std=c++17", "-O3", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
         "-Wno-deprecated-gpu-targets"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _stale(obj: str, deps: list[str]) -> bool:
    if not os.path.exists(obj):
        return True
    t = os.path.getmtime(obj)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    nvcc = _nvcc()
    os.makedirs(OBJ, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    headers.append(os.path.join(HERE, "..", "include", "rtm.h"))
    jobs = []
    units = {**FORMS, **{src: (src, []) for src in SOURCES}}
    for name, (src, defines) in units.items():
        path = os.path.join(CSRC, src)
        obj = os.path.join(OBJ, name + ".o")
        if force or _stale(obj, [path] + headers):
            flags = [f for f in FLAGS if f != "-lineinfo" or name not in FORMS]
            cmd = [nvcc, *flags, *ARCH, *defines, "-c", path, "-o", obj]
            jobs.append((name, cmd))

    def run(job):
        src, cmd = job
        p = subprocess.run(cmd, capture_output=True, text=True)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{p.stderr}")
        if verbose:
            print(src, "ok", file=sys.stderr)
        return src

    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 2)) as ex:
        list(ex.map(run, jobs))
    objs = [os.path.join(OBJ, s + ".o") for s in units]
    if force or jobs or not os.path.exists(OUT) or _stale(OUT, objs):
        cmd = [nvcc, *ARCH, "-shared", "-o", OUT + ".tmp", *objs, "-lcudart", "-Xcompiler", "-fPIC"]
        p = subprocess.run(cmd, capture_output=True, text=True)
        if p.returncode != 0:
            raise RuntimeError(f"link failed:\n{p.stderr}")
        os.replace(OUT + ".tmp", OUT)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose=True))
