"""In-tree build of libTHC.so (nvcc, sm_100a only) and of the Python call module _calls.so.

    python -m mcw_cppamp_torch_b200.build [--force] [--verbose]

Objects go to csrc/build/, the library to mcw_cppamp_torch_b200/libTHC.so.  A file is recompiled
when it or any header in csrc/ or include/ is newer than its object."""
import concurrent.futures
import glob
import os
import subprocess
import sys
import sysconfig

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(CSRC, "build")
LIB = os.path.join(PKG, "libTHC.so")
CALLS = os.path.join(PKG, "_calls.so")

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
         "-Xcompiler", "-fPIC", "--use_fast_math=false", "-I", os.path.join(ROOT, "include"), "-I", CSRC]
FLAGS = [f for f in FLAGS if f != "--use_fast_math=false"] + os.environ.get("THC_EXTRA_NVCC_FLAGS", "").split()


def _newest_header():
    hs = glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh")) + \
        glob.glob(os.path.join(ROOT, "include", "*.h"))
    return max(os.path.getmtime(h) for h in hs)


def build(force=False, verbose=False):
    os.makedirs(OBJ, exist_ok=True)
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    hdr = _newest_header()
    jobs = []
    objs = []
    for s in srcs:
        o = os.path.join(OBJ, os.path.basename(s)[:-3] + ".o")
        objs.append(o)
        if force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), hdr):
            jobs.append((s, o))

    def cc(job):
        s, o = job
        cmd = [NVCC] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
        r = subprocess.run(cmd, capture_output=True, text=True)
        return s, r

    failed = False
    with concurrent.futures.ThreadPoolExecutor(max_workers=8) as ex:
        for s, r in ex.map(cc, jobs):
            if verbose or r.returncode != 0:
                sys.stderr.write("== %s\n%s%s" % (os.path.basename(s), r.stdout, r.stderr))
            failed = failed or r.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    if jobs or not os.path.exists(LIB):
        cmd = [NVCC, "-shared", "-o", LIB] + objs + ["-lcudart"]
        subprocess.check_call(cmd)
    build_calls(force)
    return LIB


def build_calls(force=False):
    """_calls.so: the CPython module behind lib()'s functions (csrc/py_calls.cpp), compiled by the host compiler."""
    src, hdr = os.path.join(CSRC, "py_calls.cpp"), os.path.join(ROOT, "include", "THC.h")
    if not force and os.path.exists(CALLS) and os.path.getmtime(CALLS) > max(os.path.getmtime(src), os.path.getmtime(hdr)):
        return CALLS
    subprocess.check_call([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
                           "-I", os.path.join(ROOT, "include"), "-I", sysconfig.get_paths()["include"], src, "-o", CALLS])
    return CALLS


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
