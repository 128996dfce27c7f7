"""In-tree build of the package's native libraries.

* ``libyule_cuda.so``  — the CUDA backend (``csrc/*.cu``), nvcc, sm_100a only.
* ``_calls*.so``        — the per-op entry points as a CPython extension module (``csrc/calls.c``) over ``libyule_cuda.so``, gcc.
* ``libyule_synth.so`` — the host-side synthetic tensor generator / quantiser (``csrc/synth.cpp``), g++.

``python -m yule_b200.build`` builds all (``--force`` rebuilds; ``--verbose`` adds ``-Xptxas -v``).
nvcc cross-compiles without a GPU present.
"""

from __future__ import annotations

import glob
import os
import re
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
CUDA_SO = os.path.join(HERE, "libyule_cuda.so")
SYNTH_SO = os.path.join(HERE, "libyule_synth.so")
CALLS_SO = os.path.join(HERE, "_calls" + sysconfig.get_config_var("EXT_SUFFIX"))

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "--use_fast_math=false", "-Xcompiler", "-fPIC", "-Xcompiler", "-O2", "-shared",
]


def _nvcc() -> str:
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found: the CUDA backend cannot be built")
    return cand


def _stale(target: str, sources: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(s) > t for s in sources)


# The 128-row kernels of the GEMMs move registers between its warps (setmaxnreg) out of what their launch brings, and would wait for ever if the compiler had
# given it fewer than the split adds up to: that is a matter of the compiler, so it is checked where the compiler runs.
REGISTER_FLOORS = {"qgemm_tc.cu": (r"qgemm_tc_kernelILi128E", r"kLaunchRegs = (\d+);"),
                   "qgemm_int.cu": (r"qgemm_int_kernelI", r"kLaunchRegs = (\d+);"),
                   "attn_prefill.cu": (r"attn_prefill_kernelI", r"kLaunchRegs = (\d+);")}


def check_registers(report: str, kernel: str, at_least: int) -> None:
    """Raises unless ``report`` (ptxas -v) gives every instantiation of ``kernel`` (a pattern) at least so many registers."""
    counts = {}
    for name, rest in re.findall(r"Compiling entry function '(\S+)'(.*?)(?=Compiling entry function|\Z)", report, re.S):
        used = re.search(r"Used (\d+) registers", rest)
        if re.search(kernel, name) and used:
            counts[name] = int(used.group(1))
    if not counts:
        raise RuntimeError(f"the compiler's report names no kernel {kernel}")
    for name, n in counts.items():
        if n < at_least:
            raise RuntimeError(f"{name} was compiled to {n} registers; its register split is made for a launch with {at_least}")


def _compile(job: list[str]) -> None:
    src = job[job.index("-c") + 1]
    floor = REGISTER_FLOORS.get(os.path.basename(src))
    if floor is None:
        subprocess.check_call(job)
        return
    done = subprocess.run(job if "-v" in job else job[:1] + ["-Xptxas", "-v"] + job[1:], stderr=subprocess.PIPE, text=True)
    all_of_it = done.returncode or "-v" in job
    sys.stderr.write("".join(line for line in done.stderr.splitlines(True) if all_of_it or not line.startswith(("ptxas info", "    "))))
    if done.returncode:
        raise subprocess.CalledProcessError(done.returncode, job)
    try:
        with open(src) as f:
            check_registers(done.stderr, floor[0], int(re.search(floor[1], f.read()).group(1)))
    except RuntimeError:
        os.remove(job[job.index("-o") + 1])
        raise


def build_cuda(force: bool = False, verbose: bool = False) -> str:
    """One nvcc process per source file (in parallel), objects under ``csrc/build/``, then one link."""
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    common = glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.cuh")) + [
        os.path.join(os.path.dirname(HERE), "include", "yule_cuda.h"), os.path.abspath(__file__)]
    objdir = os.path.join(CSRC, "build")
    os.makedirs(objdir, exist_ok=True)
    flags = [f for f in NVCC_FLAGS if f not in ("--use_fast_math=false", "-shared")]
    jobs = []
    for src in srcs:
        obj = os.path.join(objdir, os.path.basename(src)[:-3] + ".o")
        if force or _stale(obj, [src] + common):
            jobs.append([_nvcc()] + flags + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj])
    if jobs:
        from concurrent.futures import ThreadPoolExecutor
        with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as pool:
            list(pool.map(_compile, jobs))
    objs = [os.path.join(objdir, os.path.basename(s)[:-3] + ".o") for s in srcs]
    if force or jobs or _stale(CUDA_SO, objs):
        subprocess.check_call([_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC"] + objs +
                              ["-ldl", "-o", CUDA_SO])
    build_calls(force)
    return CUDA_SO


def build_calls(force: bool = False) -> str:
    """The extension module finds ``libyule_cuda.so`` beside itself."""
    src, include = os.path.join(CSRC, "calls.c"), os.path.join(os.path.dirname(HERE), "include")
    if force or _stale(CALLS_SO, [src, os.path.join(include, "yule_cuda.h"), os.path.abspath(__file__)]):
        subprocess.check_call(["gcc", "-O2", "-std=c11", "-fPIC", "-shared", "-I", sysconfig.get_paths()["include"], "-I", include, src,
                               "-L", HERE, "-l:libyule_cuda.so", "-Wl,-rpath,$ORIGIN", "-o", CALLS_SO])
    return CALLS_SO


def build_synth(force: bool = False) -> str:
    src = os.path.join(CSRC, "synth.cpp")
    if force or _stale(SYNTH_SO, [src, os.path.abspath(__file__)]):
        subprocess.check_call(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-pthread", "-ffp-contract=off",
                               src, "-o", SYNTH_SO])
    return SYNTH_SO


def main(argv: list[str]) -> int:
    force, verbose = "--force" in argv, "--verbose" in argv
    print(build_synth(force))
    print(build_cuda(force, verbose))
    return 0


if __name__ == "__main__":
    sys.exit(main(sys.argv[1:]))
