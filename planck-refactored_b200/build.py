"""Build libplanck_fock.so (sm_100a) in-tree.

nvcc compiles pfk_classes.cu once per quartet class (55 translation units), the
setup kernels and the C ABI in parallel into _build/, then links the shared
library next to this file.  Objects are rebuilt when any source under csrc/
or include/ is newer than they are.  nvcc writes under another name, and what it
wrote becomes the object when it is complete, with the time at which the
compilation began: an interrupted build, or a source edited during one, leaves
nothing that looks current.

    python build.py [-j N] [--force]
"""
import argparse
import concurrent.futures as cf
import os
import subprocess
import sys
import time

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(REPO, "_build", "pfk")
LIB = os.path.join(HERE, "libplanck_fock.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-lineinfo", "-std=c++17", "-Xcompiler", "-fPIC", "-I" + CSRC,
         "-I" + os.path.join(REPO, "include")]


DEVICE_DEPS = ["pfk_device.cuh", "pfk_internal.h", "rys_table_data.inc", "../../include/planck_fock.h"]
DEPS = {
    "pfk_classes.cu": DEVICE_DEPS + ["pfk_kernels.cuh", "pfk_os.cuh", "boys_table_data.inc"],
    "pfk_setup.cu": DEVICE_DEPS + ["pfk_kernels.cuh", "pfk_setup.h"],
    "pfk_api.cu": DEVICE_DEPS + ["pfk_setup.h", "../../include/planck_fock.h"],
    "pfk_onee.cu": DEVICE_DEPS + ["pfk_kernels.cuh", "pfk_os.cuh", "boys_table_data.inc"],
    "pfk_mlp.cu": ["../../include/planck_fock.h"],
    "pfk_checkpoint.cu": ["../../include/planck_fock.h"],
    "pfk_scf.cu": ["../../include/planck_fock.h", "pfk_internal.h", "pfk_device.cuh"],
}


# Class ranges per translation unit (class c = X(X+1)/2 + Y for bra pair
# class X >= ket pair class Y): one unit per class, so the 55 classes compile
# in parallel.
CLASS_UNITS = [(c, c + 1) for c in range(55)]
# Those that take longest to compile (4 to 12 minutes of one core), which begin
# first: (dp|dp) alone, begun among the last, had the others wait for 4 minutes.
LONGEST = [14, 17, 5, 20, 13, 12, 11]


def _units():
    units = [("pfk_classes.cu", f"classes_{b}_{e}.o", [f"-DPFK_CLASS_BEGIN={b}", f"-DPFK_CLASS_END={e}"])
             for b, e in [CLASS_UNITS[c] for c in LONGEST] + [u for u in reversed(CLASS_UNITS) if u[0] not in LONGEST]]
    units += [("pfk_setup.cu", "setup.o", []), ("pfk_api.cu", "api.o", []), ("pfk_onee.cu", "onee.o", []),
              ("pfk_mlp.cu", "mlp.o", []), ("pfk_checkpoint.cu", "checkpoint.o", []), ("pfk_scf.cu", "scf.o", [])]
    return units


def _newest(src):
    files = [os.path.join(CSRC, src)] + [os.path.join(CSRC, d) for d in DEPS[src]] + [os.path.abspath(__file__)]
    return max(os.path.getmtime(f) for f in files)


def _compile(src, obj, extra, verbose):
    part = f"{obj}.{os.getpid()}.part"
    cmd = [NVCC] + ARCH + FLAGS + extra + ["-c", os.path.join(CSRC, src), "-o", part]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
    began = time.time()
    try:
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src} {extra}:\n{r.stderr[-6000:]}")
        os.utime(part, (began, began))
        os.replace(part, obj)
    finally:
        if os.path.exists(part):
            os.remove(part)
    return r.stderr


def build(jobs=None, force=False, verbose=False):
    os.makedirs(BUILD, exist_ok=True)
    todo = []
    for src, obj, extra in _units():
        path = os.path.join(BUILD, obj)
        if force or not os.path.exists(path) or os.path.getmtime(path) < _newest(src):
            todo.append((src, path, extra))
    logs = {}
    if todo:
        with cf.ThreadPoolExecutor(max_workers=jobs or os.cpu_count()) as ex:
            futs = {ex.submit(_compile, s, o, e, verbose): (s, o) for s, o, e in todo}
            for f in cf.as_completed(futs):
                logs[futs[f][1]] = f.result()
    objs = [os.path.join(BUILD, o) for _, o, _ in _units()]
    if todo or not os.path.exists(LIB) or os.path.getmtime(LIB) < max(os.path.getmtime(o) for o in objs):
        part = f"{LIB}.{os.getpid()}.part"
        try:
            subprocess.check_call([NVCC] + ARCH + ["-shared", "-o", part] + objs + ["-lcudart", "-lcublas", "-lcusolver"])
            os.replace(part, LIB)
        finally:
            if os.path.exists(part):
                os.remove(part)
    return LIB, logs


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("-j", type=int, default=None)
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true", help="print ptxas register/spill report")
    a = ap.parse_args()
    lib, logs = build(a.j, a.force, a.verbose)
    if a.verbose:
        for k, v in logs.items():
            print("==", k)
            print(v)
    print(lib)
    sys.exit(0)
