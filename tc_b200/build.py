"""Build step of the CUDA library libtcg_b200.so (in-tree, sm_100a).

api.cu (C-ABI, orchestration, generic kernels), cube.cu (on-chip hf2x), subspace.cu
(the dense Davidson subspace step), any_inst.cu per precision (run-time shapes) and
one instance of fast_inst.cu per compiled cubic grid size and precision are compiled in
parallel into tc_b200/_build/ and linked into tc_b200/libtcg_b200.so, the device code
compressed for size (173 MB otherwise).
"""
import concurrent.futures as cf
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
SO = os.path.join(HERE, "libtcg_b200.so")
SRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "_build")
FAST_SIZES = (12, 15, 16, 18, 20, 24, 25, 27, 30, 32, 36, 40, 45, 48)     # ctx.cuh: TCG_FAST_SIZES
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
CFLAGS = ARCH + ["-O3", "-lineinfo", "-compress-mode=size", "-std=c++17", "-Xcompiler", "-fPIC"]


def sources():
    return [os.path.join(SRC, f) for f in sorted(os.listdir(SRC)) if f.endswith((".cu", ".cuh"))] + \
        [os.path.join(HERE, "..", "include", "tcg.h")]


def stale():
    if not os.path.exists(SO):
        return True
    t = os.path.getmtime(SO)
    return any(os.path.getmtime(s) > t for s in sources())


def _units():
    units = [(os.path.join(SRC, "api.cu"), os.path.join(OBJ, "api.o"), []),
             (os.path.join(SRC, "cube.cu"), os.path.join(OBJ, "cube.o"), []),
             (os.path.join(SRC, "subspace.cu"), os.path.join(OBJ, "subspace.o"), [])]
    for t in ("double", "float"):                 # the longest units first
        units.append((os.path.join(SRC, "any_inst.cu"), os.path.join(OBJ, f"any_{t}.o"), [f"-DTCG_FAST_T={t}"]))
        for n in reversed(FAST_SIZES):
            units.append((os.path.join(SRC, "fast_inst.cu"), os.path.join(OBJ, f"fast_{n}_{t}.o"),
                          [f"-DTCG_FAST_N={n}", f"-DTCG_FAST_T={t}"]))
    return units


def build(force=False, verbose=False, jobs=None):
    if not force and not stale():
        return SO
    nvcc = os.environ.get("NVCC", "nvcc")
    os.makedirs(OBJ, exist_ok=True)

    def compile_one(u):
        src, obj, extra = u
        cmd = [nvcc, *CFLAGS, *extra, "-c", "-o", obj, src]
        if verbose:
            print(" ".join(cmd), file=sys.stderr)
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src} {extra}:\n{r.stderr}")
        return obj

    units = _units()
    jobs = jobs or min(len(units), os.cpu_count() or 4)
    with cf.ThreadPoolExecutor(jobs) as ex:
        objs = list(ex.map(compile_one, units))
    cmd = [nvcc, *ARCH, "-shared", "-o", SO + ".tmp", *objs, "-lcublas", "-lcusolver"]
    if verbose:
        print(" ".join(cmd), file=sys.stderr)
    subprocess.run(cmd, check=True)
    os.replace(SO + ".tmp", SO)
    return SO


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
    print(SO)
