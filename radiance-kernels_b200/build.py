"""Builds librk_mx_attn.so (the C-ABI library) in-tree with nvcc for sm_100a, and _rk_front.so (the Python package's
native front end over it) with the host compiler.

    python radiance-kernels_b200/build.py [--force]

nvcc cross-compiles without a GPU; the .so files sit beside this file so they travel
with the source tree to the machine that has the GPU.
"""
import importlib.util
import os
import pathlib
import subprocess
import sys
import sysconfig

HERE = pathlib.Path(__file__).resolve().parent
CSRC = HERE / "csrc"
SOURCES = ["rk_api.cu", "rk_quant.cu", "rk_prefill.cu", "rk_prefill1.cu", "rk_prefill2c.cu", "rk_peak.cu", "rk_mxgemm.cu", "rk_decode.cu"]
HEADERS = ["rk_common.cuh", "rk_internal.h", "rk_rebase.cuh", "rk_prefill.cuh", "rk_decode_tc.cuh"]
LIB = HERE / "librk_mx_attn.so"
FRONT_SRC = CSRC / "rk_front.cpp"
FRONT = HERE / "_rk_front.so"
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-lineinfo",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--use_fast_math=false"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def needs_build():
    if not LIB.exists():
        return True
    t = LIB.stat().st_mtime
    deps = [CSRC / s for s in SOURCES + HEADERS] + [HERE.parent / "include" / "rk_mx_attn.h"]
    return any(p.stat().st_mtime > t for p in deps)


def front_needs_build():
    deps = [FRONT_SRC, HERE.parent / "include" / "rk_mx_attn.h"]
    return not FRONT.exists() or any(p.stat().st_mtime > FRONT.stat().st_mtime for p in deps)


def front_object():
    return CSRC / "rk_front.o"


def front_compile_command():
    """Host compiler call for the front end.  torch is located, not imported: its headers give the tensor class, its
    libraries are in the process before the module is."""
    torch_dir = pathlib.Path(importlib.util.find_spec("torch").submodule_search_locations[0])
    cuda = pathlib.Path(_nvcc()).resolve().parent.parent if os.path.isabs(_nvcc()) else pathlib.Path("/usr/local/cuda")
    inc = [torch_dir / "include", torch_dir / "include" / "torch" / "csrc" / "api" / "include", sysconfig.get_paths()["include"], cuda / "include"]
    return (["g++", "-std=c++17", "-O2", "-fPIC", "-fvisibility=hidden", "-c", str(FRONT_SRC), "-o", str(front_object())] +
            [f for i in inc for f in ("-isystem", str(i))])


def front_link_command():
    torch_lib = pathlib.Path(importlib.util.find_spec("torch").submodule_search_locations[0]) / "lib"
    return ["g++", "-shared", str(front_object()), "-o", str(FRONT), f"-L{HERE}", "-l:" + LIB.name, f"-L{torch_lib}", "-ltorch_python",
            "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10", "-Wl,-rpath,$ORIGIN"]


def build(force=False, verbose=False):
    lib_stale, front_stale = force or needs_build(), force or front_needs_build()
    procs = []
    objs = [str(CSRC / (s[:-3] + ".o")) for s in SOURCES]
    if front_stale:
        procs.append((FRONT_SRC.name, subprocess.Popen(front_compile_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    if lib_stale:
        for s, o in zip(SOURCES, objs):
            cmd = [_nvcc()] + [f for f in NVCC_FLAGS if f != "--use_fast_math=false"] + ["-c", str(CSRC / s), "-o", o]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            procs.append((s, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = []
    for s, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        if p.returncode != 0:
            failed.append(s)
    if failed:
        raise RuntimeError("compiler failed on " + ", ".join(failed))
    if lib_stale:
        subprocess.run([_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(LIB)] + objs, check=True)
    if front_stale:
        subprocess.run(front_link_command(), check=True)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
