"""Builds libzinc_b200.so (CUDA kernels + C ABI) in-tree with nvcc for sm_100a."""
from __future__ import annotations

import os
import re
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
SO = os.path.join(HERE, "libzinc_b200.so")
CALL_SO = os.path.join(HERE, "_call.so")   # Python module: calls into the library without ctypes
SOURCES = ["api.cu", "dmmv.cu", "dmmv_warp.cu", "dmmv_q6k.cu", "dmmv_row.cu", "misc.cu", "gemm_simple.cu", "gemm_tc.cu", "gemm_cut.cu",
           "dmmv_static_scratch.cu", "comm.cu", "dmmv_mxfp4.cu", "program.cu", "moe_program.cu", "moe_gemm_tc.cu", "moe_gemm_pair.cu", "gemm_mx.cu", "gemm_exact.cu",
           "gemm_exact_q4k.cu", "gemm_exact_q5k.cu", "gemm_exact_q6k.cu", "gemm_exact_q8.cu", "gemm_exact_mxfp4.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--use_fast_math=false", "-Xptxas", "-v",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.exists(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def _torch_spec():
    import importlib.util

    return importlib.util.find_spec("torch")


def _call_command():
    """g++ on call.cpp, against the headers and libraries of the installed torch (found without importing it); None
    where there is no torch: the library does not need it."""
    import sysconfig

    spec = _torch_spec()
    if spec is None or not spec.origin:
        return None
    torch_dir = os.path.dirname(spec.origin)
    inc = os.path.join(torch_dir, "include")
    lib = os.path.join(torch_dir, "lib")
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", os.path.join(CSRC, "call.cpp"), "-o", CALL_SO,
            "-isystem", inc, "-isystem", os.path.join(inc, "torch", "csrc", "api", "include"),
            "-I", sysconfig.get_paths()["include"], "-L", lib, "-Wl,-rpath," + lib, "-ltorch_python", "-ltorch_cpu", "-lc10"]


def stale() -> bool:
    built = [SO] if _call_command() is None else [SO, CALL_SO]
    if not all(os.path.exists(f) for f in built):
        return True
    t = min(os.path.getmtime(f) for f in built)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [
        os.path.join(HERE, "..", "include", "zinc_cuda.h")]
    return any(os.path.getmtime(d) > t for d in deps)


def check_registers(log: str) -> int:
    """Raises where a kernel of the f32-accurate GEMM got another number of registers than gemm_exact.cuh counts on: the launch would be
    refused then (its promoting warps would wait for registers that nobody gives back), and the product left to a kernel some thirty
    times slower. Returns the number of kernels."""
    with open(os.path.join(CSRC, "gemm_exact.cuh")) as f:
        widest, few, many = map(int, re.search(r"kLaunchRegs = BN <= (\d+) \? (\d+) : (\d+)", f.read()).groups())
    found = re.findall(r"entry function '(\w*gemm_exact_kernelILi\d+ELi(\d+)E\w*)'(?:(?!entry function).)*?Used (\d+) registers", log, re.S)
    for name, width, used in found:
        want = few if int(width) <= widest else many
        if int(used) != want:
            raise RuntimeError(f"{name}: {used} registers, not {want}")
    if not found:
        raise RuntimeError("no kernel of the f32-accurate GEMM among the compiled ones")
    return len(found)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu into objects (in parallel) and link the shared library."""
    if not force and not stale():
        return SO
    nvcc = _nvcc()
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    procs = []
    command = _call_command()
    call = command and subprocess.Popen(command, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    for src in SOURCES:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        cmd = [nvcc, *[f for f in NVCC_FLAGS if f != "--use_fast_math=false"], "-c",
               os.path.join(CSRC, src), "-o", obj]
        procs.append((src, obj, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    objs = []
    log = []
    for src, obj, p in procs:
        out, _ = p.communicate()
        log.append(f"==== {src}\n{out}")
        if p.returncode != 0:
            sys.stderr.write(out)
            raise RuntimeError(f"nvcc failed on {src}")
        objs.append(obj)
    if call is not None:
        out, _ = call.communicate()
        if call.returncode != 0:
            sys.stderr.write(out)
            raise RuntimeError("g++ failed on call.cpp")
    with open(os.path.join(objdir, "ptxas.log"), "w") as f:
        f.write("\n".join(log))
    if verbose:
        print("\n".join(log))
    check_registers("\n".join(log))
    subprocess.check_call([nvcc, "-shared", "-o", SO, *objs, "-gencode", "arch=compute_100a,code=sm_100a"])
    return SO


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
