"""Build the sm_100a shared library libhammerhead_b200.so in-tree.

Each csrc/*.cu is compiled with nvcc for sm_100a (in parallel), then linked
into hammerhead_b200/libhammerhead_b200.so next to the Python host layer that
loads it. Objects go to _build/ (not committed). Usage:

    python hammerhead.jl_b200/build.py [--force] [--verbose]
"""
import argparse
import concurrent.futures as cf
import os
import re
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(HERE, "_build")
OUT = os.path.join(HERE, "hammerhead_b200", "libhammerhead_b200.so")

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-lineinfo", "-std=c++17", "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC",
         "-I", os.path.join(ROOT, "include"), "-I", CSRC]


def nvcc():
    path = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(path):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build hammerhead_b200")
    return path


def _includes(path, seen):
    """The project headers that `path` includes, directly or through others."""
    with open(path) as f:
        for name in re.findall(r'^\s*#include "([^"]+)"', f.read(), re.M):
            for d in (CSRC, os.path.join(ROOT, "include")):
                p = os.path.join(d, name)
                if os.path.exists(p) and p not in seen:
                    seen.add(p)
                    _includes(p, seen)
    return seen


def _stale(src, obj, deps):
    if not os.path.exists(obj):
        return True
    t = os.path.getmtime(obj)
    return any(os.path.getmtime(d) > t for d in [src] + deps)


def build(force=False, verbose=False, jobs=None):
    os.makedirs(BUILD, exist_ok=True)
    sources = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
    cc = nvcc()
    todo = []
    objs = []
    for s in sources:
        src = os.path.join(CSRC, s)
        obj = os.path.join(BUILD, s.replace(".cu", ".o"))
        objs.append(obj)
        if force or _stale(src, obj, list(_includes(src, set()))):
            todo.append((src, obj))

    def compile_one(item):
        src, obj = item
        cmd = [cc] + ARCH + FLAGS + ["-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, r.returncode, r.stdout + r.stderr

    if todo:
        with cf.ThreadPoolExecutor(max_workers=jobs or min(8, os.cpu_count() or 4)) as ex:
            for src, rc, log in ex.map(compile_one, todo):
                if verbose and log:
                    print(log)
                if rc != 0:
                    sys.stderr.write(log)
                    raise RuntimeError(f"nvcc failed on {os.path.basename(src)}")
    if force or todo or not os.path.exists(OUT) or any(os.path.getmtime(o) > os.path.getmtime(OUT) for o in objs):
        cmd = [cc] + ARCH + ["-shared", "-o", OUT] + objs + ["-lcudart_static", "-lrt", "-lpthread", "-ldl"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("linking libhammerhead_b200.so failed")
    return OUT


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(force=a.force, verbose=a.verbose))
