"""Build libfmta_b200.so (sm_100a only) in-tree with nvcc.

    python flash-multi-token-attention_b200/build.py [--force] [--verbose]

Every translation unit under csrc/ is compiled with
``-gencode arch=compute_100a,code=sm_100a -lineinfo`` (cross-compiles without a GPU) and
linked into ``fmta_b200/libfmta_b200.so`` next to the Python layer, so the library
travels with the source tree; ``csrc_torch/`` (the operators' host side, C++ against torch) becomes ``fmta_b200/_native.so``.  A unit is rebuilt when it or any header is newer than its
object file, the host side also when torch, the interpreter or the command has changed.
"""
import argparse
import concurrent.futures as cf
import glob
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "fmta_b200", "libfmta_b200.so")
NATIVE = os.path.join(HERE, "fmta_b200", "_native.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--use_fast_math", "-Xcompiler", "-fPIC", "-Xptxas", "-v",
]


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libfmta_b200.so cannot be built")
    return exe


def _newest_header():
    hs = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + \
        glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    return max(os.path.getmtime(h) for h in hs)


def _compile(src, obj, verbose):
    cmd = [_nvcc()] + NVCC_FLAGS + os.environ.get("FMTA_NVCC_EXTRA", "").split() + ["-c", src, "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    log = r.stdout + r.stderr
    with open(obj + ".log", "w") as f:
        f.write(" ".join(cmd) + "\n" + log)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed for %s:\n%s" % (src, log[-4000:]))
    if verbose:
        print(log)
    return obj


def build(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    hdr_t = _newest_header()
    jobs, objs = [], []
    for s in srcs:
        o = os.path.join(OBJ, os.path.basename(s)[:-3] + ".o")
        objs.append(o)
        if force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), hdr_t):
            jobs.append((s, o))
    if jobs:
        with cf.ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            list(ex.map(lambda a: _compile(a[0], a[1], verbose), jobs))
    if jobs or not os.path.exists(LIB):
        cmd = [_nvcc(), "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n" + r.stdout + r.stderr)
    _build_host_layer(force, verbose)
    return LIB


def _build_host_layer(force=False, verbose=False):
    """fmta_b200/_native.so: the operators' host side in C++ (csrc_torch/), linked against torch and LIB."""
    import sysconfig
    import torch
    src = os.path.join(HERE, "csrc_torch", "fmta_torch.cpp")
    hdr = os.path.join(HERE, "..", "include", "fmta_b200.h")
    tdir = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    inc = [os.path.join(tdir, "include"), os.path.join(tdir, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    cmd = [os.environ.get("CXX", "g++"), "-shared", "-fPIC", "-O2", "-std=c++17", src, "-o", NATIVE, "-DTORCH_EXTENSION_NAME=_native",
           "-DTORCH_API_INCLUDE_EXTENSION_H", "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI)]
    for i in inc:
        cmd += ["-isystem", i]
    cmd += ["-L" + os.path.join(tdir, "lib"), "-L" + os.path.dirname(LIB), "-l:libfmta_b200.so", "-lc10", "-lc10_cuda", "-ltorch",
            "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    # it is bound to the torch (and the interpreter) that it was compiled against
    stamp, key = os.path.join(OBJ, "_native.stamp"), "\n".join([torch.__version__, sys.version] + cmd)
    built = open(stamp).read() if os.path.exists(stamp) else None
    if not force and built == key and os.path.exists(NATIVE) and os.path.getmtime(NATIVE) > max(os.path.getmtime(src), os.path.getmtime(hdr)):
        return NATIVE
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("host layer failed:\n%s" % (r.stdout + r.stderr)[-4000:])
    if verbose:
        print(r.stdout + r.stderr)
    with open(stamp, "w") as f:
        f.write(key)
    return NATIVE


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
