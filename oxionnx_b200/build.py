"""Builds oxionnx_b200/_lib/liboxb200.so: the CUDA kernels (sm_100a only) plus the C++ host
runtime behind the C ABI of include/oxb200.h.

nvcc cross-compiles without a GPU.  The CUDA runtime is linked statically and the driver's
tensor-map encoders are resolved at run time, so the library loads (and its symbols can be
checked) on a host that has no GPU driver.
"""
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT_DIR = os.path.join(HERE, "_lib")
OBJ_DIR = os.path.join(OUT_DIR, "obj")
LIB = os.path.join(OUT_DIR, "liboxb200.so")

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-std=c++17", "-O3", "-lineinfo", "-Xcompiler", "-fPIC,-ffp-contract=off,-fno-fast-math", "--fmad=false"]
# --fmad=false everywhere except the tensor-core kernel file, whose float epilogue is one add
KERNEL = [f for f in COMMON if f != "--fmad=false"]
# object -> (source, flags); the integer contraction kernel is compiled once per tile width, side by side
OBJECTS = {
    "kernels_glue": ("kernels_glue.cu", COMMON),
    **{name: (name + ".cu", KERNEL) for name in ("kernels_simt", "kernels_umma", "umma_i8", "umma_tf32", "umma_f16", "umma_small_i8", "umma_small_float",
                                                  "umma_probe", "umma_chain", "umma_attention")},
    **{f"umma_i8_{tile}": ("umma_i8_tile.cu", KERNEL + [f"-DOXB_TILE={bn}", f"-DOXB_PAIR={pair}"])
       for tile, bn, pair in (("32", 32, "false"), ("64", 64, "false"), ("128", 128, "false"), ("256", 256, "false"), ("pair", 256, "true"))},
    **{name: (name + ".cpp", COMMON) for name in ("runtime", "planner", "abi", "onnx_model", "model_abi")},
}
HEADERS = ["common.hpp", "kernels.hpp", "runtime.hpp", "umma_kernel.cuh", "umma_epilogue8.cuh", "umma_launch.cuh", "umma_small.cuh", "pdl.cuh", "umma_chain.cuh", "model.hpp", "abi_internal.hpp", os.path.join("..", "..", "include", "oxb200.h")]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = [os.path.join(CSRC, h) for h in HEADERS]
    nvcc = _nvcc()
    jobs = []
    objs = []
    for name, (src, flags) in OBJECTS.items():
        path = os.path.join(CSRC, src)
        obj = os.path.join(OBJ_DIR, name + ".o")
        objs.append(obj)
        if force or _stale(obj, [path] + headers):
            cmd = [nvcc] + ARCH + flags + ["-x", "cu", "-c", path, "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("build failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stderr

    if jobs:
        with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as ex:
            for log in ex.map(run, jobs):
                if verbose and log:
                    print(log)
    if force or jobs or _stale(LIB, objs):
        run([nvcc] + ARCH + ["-shared", "-o", LIB] + objs + ["-cudart", "static", "-Xlinker", "--no-undefined", "-lpthread", "-ldl", "-lrt"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
