"""Builds the native library in-tree: map_b200/libmap_b200.so.

Steps:
  1. embed the hand-written skeleton headers (csrc/skeleton/*.cuh) into
     csrc/skeleton_embed.inc so NVRTC can compile generated kernels against them;
  2. compile the host runtime (csrc/*.cpp) and the hand-written kernels that are
     built ahead of time (csrc/*.cu, nvcc for sm_100a), and link them with the
     static CUDA runtime and NVRTC;
  3. compile csrc/skeleton/selfcheck.cu with nvcc for sm_100a (the skeleton
     building blocks must build under nvcc as well as NVRTC).

Usage: python -m map_b200.build [--force]
"""
import concurrent.futures as cf
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
SKEL = os.path.join(CSRC, "skeleton")
BUILD = os.path.join(HERE, "_build")
LIB = os.path.join(HERE, "libmap_b200.so")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
NVCC = os.path.join(CUDA, "bin", "nvcc")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]

# name under which each header is visible to NVRTC-compiled kernels
HEADERS = [("common.cuh", "map_common.cuh"), ("scan.cuh", "map_scan.cuh"), ("rule.cuh", "map_rule.cuh"),
           ("flow.cuh", "map_flow.cuh")]


def _run(cmd):
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError("command failed: %s\n%s" % (" ".join(cmd), r.stdout))
    return r.stdout


def embed_headers():
    out = os.path.join(CSRC, "skeleton_embed.inc")
    parts = ["// generated by map_b200/build.py from csrc/skeleton/*.cuh -- do not edit\n",
             "struct EmbeddedHeader { const char *name; const char *source; };\n",
             "static const EmbeddedHeader kSkeletonHeaders[] = {\n"]
    for fname, vname in HEADERS:
        path = os.path.join(SKEL, fname)
        if not os.path.exists(path):
            continue
        text = open(path).read()
        chunks = [text[i:i + 8000] for i in range(0, len(text), 8000)]
        lit = "\n".join('R"MAPB(%s)MAPB"' % c for c in chunks)
        parts.append('  {"%s", %s},\n' % (vname, lit))
    parts.append("};\n")
    new = "".join(parts)
    if not os.path.exists(out) or open(out).read() != new:
        with open(out, "w") as f:
            f.write(new)


def _obj(src):
    return os.path.join(BUILD, os.path.basename(src) + ".o")


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    os.makedirs(BUILD, exist_ok=True)
    embed_headers()
    srcs = sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cpp"))
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".hpp", ".inc"))]
    headers.append(os.path.join(HERE, "..", "include", "map_b200.h"))
    cflags = ["-O2", "-g", "-fPIC", "-std=c++17", "-Wall", "-Wno-unused-function", "-fvisibility=hidden",
              "-I" + os.path.join(CUDA, "include"), "-I" + CSRC]
    jobs = []
    for s in srcs:
        o = _obj(s)
        if force or _stale(o, [s] + headers):
            jobs.append(["g++", "-c", s, "-o", o] + cflags)
    with cf.ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
        for out in ex.map(_run, jobs):
            if verbose and out:
                print(out)
    cu_srcs = sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))
    cu_jobs = []
    for s in cu_srcs:
        o = _obj(s)
        if force or _stale(o, [s] + headers):
            cu_jobs.append([NVCC, "-c", s, "-o", o, "-std=c++17", "-O3", "-lineinfo", "--fmad=false"] + ARCH +
                           ["-Xcompiler", "-fPIC,-fvisibility=hidden", "-I" + CSRC])
    with cf.ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
        for out in ex.map(_run, cu_jobs):
            if verbose and out:
                print(out)
    objs = [_obj(s) for s in srcs + cu_srcs]
    if force or _stale(LIB, objs):
        _run(["g++", "-shared", "-o", LIB] + objs +
             ["-L" + os.path.join(CUDA, "lib64"), "-Wl,--exclude-libs,ALL", "-lcudart_static", "-lnvrtc",
              "-ldl", "-lpthread", "-lrt", "-Wl,-rpath," + os.path.join(CUDA, "lib64")])
    # nvcc self-check of the skeleton building blocks for sm_100a
    sc = os.path.join(SKEL, "selfcheck.cu")
    cubin = os.path.join(BUILD, "selfcheck.cubin")
    if os.path.exists(sc) and (force or _stale(cubin, [sc] + [os.path.join(SKEL, h) for h, _ in HEADERS
                                                            if os.path.exists(os.path.join(SKEL, h))])):
        _run([NVCC, "-cubin", "-std=c++17", "--fmad=false", "-lineinfo", "-O3"] + ARCH +
             ["-I" + SKEL, "-o", cubin, sc])
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(LIB)
