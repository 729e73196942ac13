"""Builds the fftb CUDA library in-tree for sm_100a.

``python -m fftm_b200.build`` compiles every ``.cu`` source under
``fftm_b200/csrc`` with nvcc (``-gencode arch=compute_100a,code=sm_100a``) into
objects under ``fftm_b200/_build`` and links ``fftm_b200/libfftb_b200.so``
(CUDA runtime linked statically, so the library does not depend on the runtime
version that other libraries in the process load).  The pass and line kernels are
instantiated in parts so the compiler runs in parallel.
"""
from __future__ import annotations

import concurrent.futures as cf
import hashlib
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libfftb_b200.so")
NPARTS = 8        # objects of the pass kernel's instantiations
LINE_NPARTS = 64  # objects per precision of the line kernel's

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-Xcompiler", "-O2",
              "--expt-relaxed-constexpr", f"-DFFTB_NPARTS={NPARTS}", f"-DFFTB_LINE_NPARTS={LINE_NPARTS}"]
# An object's device code is one module, which the runtime unpacks and loads whole when the first of
# its kernels is asked for: the first call of a process on a length pays for that.  The line
# kernels' (1200 of them) are therefore kept small: 64 objects per precision, about five lengths each,
# and without -lineinfo, whose records of the inlined stages are 70% of a module (21.3 against
# 6.0 MB for a sixteenth of the lengths).  Loading one module on a B200: 30 ms in 16 objects with line
# records, 8.5 ms in 64 with them, 2.4 ms in 64 without; the first 192^3 gradient of a process (two
# modules and its allocations): 58 ms in 16 objects with records, 6.1 so.
LINE_FLAGS = ["-Xfatbin=--compress-mode=size"]
OTHER_FLAGS = ["-lineinfo"]


def nvcc() -> str:
    cand = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return cand if os.path.exists(cand) else (shutil.which("nvcc") or "nvcc")


def _headers_digest() -> str:
    h = hashlib.sha256()
    for d in (CSRC, os.path.join(ROOT, "include")):
        for root, _, files in os.walk(d):
            for f in sorted(files):
                if f.endswith((".h", ".cuh", ".hpp")):
                    with open(os.path.join(root, f), "rb") as fh:
                        h.update(f.encode())
                        h.update(fh.read())
    return h.hexdigest()


def source_digest() -> str:
    """SHA-256 over every source the library is compiled from (csrc/ and include/, names and
    contents).  The build compiles it into the library (fftb_build_digest()), so a process can
    check that the library it loaded was built from the tree beside it."""
    h = hashlib.sha256()
    for d in (CSRC, os.path.join(ROOT, "include")):
        for root, _, files in sorted(os.walk(d)):
            for f in sorted(files):
                if f.endswith((".cu", ".cuh", ".h", ".hpp")):
                    with open(os.path.join(root, f), "rb") as fh:
                        h.update(os.path.relpath(os.path.join(root, f), ROOT).encode())
                        h.update(b"\0")
                        h.update(fh.read())
    return h.hexdigest()


def _digest_source(digest: str) -> str:
    """Writes _build/fftb_digest.cu (only when the digest changed, so its object is reused)."""
    path = os.path.join(BUILD, "fftb_digest.cu")
    text = ('// generated by fftm_b200/build.py: digest of the sources this library is built from\n'
            f'extern "C" const char *fftb_build_digest(void) {{ return "{digest}"; }}\n')
    if not os.path.exists(path) or open(path).read() != text:
        with open(path, "w") as fh:
            fh.write(text)
    return path


def _jobs():
    jobs = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith(".cu"):
            continue
        src = os.path.join(CSRC, f)
        if f == "fftb_pass_inst.cu":
            for k in range(NPARTS):
                jobs.append((src, os.path.join(BUILD, f"pass_float_{k}.o"),
                             OTHER_FLAGS + ["-DFFTB_REAL=float", f"-DFFTB_PART={k}"]))
        elif f == "fftb_line_inst.cu":
            for real in ("float", "double"):
                for k in range(LINE_NPARTS):
                    obj = os.path.join(BUILD, f"line_{real}_{k}.o")
                    jobs.append((src, obj, LINE_FLAGS + [f"-DFFTB_REAL={real}", f"-DFFTB_PART={k}"]))
        else:
            jobs.append((src, os.path.join(BUILD, f[:-3] + ".o"), OTHER_FLAGS))
    jobs.append((_digest_source(source_digest()), os.path.join(BUILD, "fftb_digest.o"), OTHER_FLAGS))
    return jobs


def _compile(job, digest):
    src, obj, extra = job
    stamp = obj + ".stamp"
    with open(src, "rb") as fh:  # by content: a copied tree keeps its objects
        key = digest + "|" + " ".join(NVCC_FLAGS + extra) + "|" + hashlib.sha256(fh.read()).hexdigest()
    if os.path.exists(obj) and os.path.exists(stamp) and open(stamp).read() == key:
        return obj, None
    cmd = [nvcc()] + ARCH + NVCC_FLAGS + extra + ["-c", src, "-o", obj]
    p = subprocess.run(cmd, capture_output=True, text=True)
    if p.returncode != 0:
        return obj, " ".join(cmd) + "\n" + p.stdout + p.stderr
    with open(stamp, "w") as fh:
        fh.write(key)
    return obj, None


def build(verbose: bool = False) -> str:
    os.makedirs(BUILD, exist_ok=True)
    digest = _headers_digest()
    jobs = _jobs()
    errors = []
    objs = []
    with cf.ThreadPoolExecutor(max_workers=max(2, os.cpu_count() or 2)) as ex:
        for obj, err in ex.map(lambda j: _compile(j, digest), jobs):
            objs.append(obj)
            if err:
                errors.append(err)
    if errors:
        raise RuntimeError("nvcc failed:\n" + "\n".join(errors))
    newest = max(os.path.getmtime(o) for o in objs)
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < newest:
        tmp = LIB + ".tmp"
        cmd = [nvcc()] + ARCH + ["-shared", "-Xcompiler", "-fPIC", "-o", tmp] + objs + ["-lcuda"]
        subprocess.check_call(cmd)
        os.replace(tmp, LIB)
    if verbose:
        print(LIB)
    return LIB


if __name__ == "__main__":
    build(verbose=True)
    sys.exit(0)
