"""Build libflare_b200.so (sm_100a) from csrc/ with nvcc and the native host layer with g++.  Objects are cached by content hash."""

from __future__ import annotations

import concurrent.futures as cf
import hashlib
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build", "obj")
LIB = os.path.join(HERE, "libflare_b200.so")
HOST = os.path.join(HERE, "causal_flare", "_host.so")  # native host layer of the Python package (host_ext.cpp)

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
    "--compress-mode=size",  # (line tables are most of the code's size: a sixth of the library)
    *os.environ.get("FLARE_B200_NVCC_FLAGS", "").split(),  # extra flags for experiments (e.g. -DNAME)
]

# (source file, extra defines, object name)
UNITS = [
    ("flare_abi.cu", [], "flare_abi"),
    ("walk_exact.cu", [], "walk_exact_dispatch"),
    *[("walk_exact.cu", [f"-DFLARE_WALK_MM={mm}"], f"walk_exact_mm{mm}") for mm in (2, 8, 16, 32, 64)],
    ("narrow_exact.cu", [], "narrow_exact"),
    ("narrow_mma.cu", [], "narrow_mma"),
    ("decode_step.cu", [], "decode_step"),
    ("state_ops.cu", [], "state_ops"),
    ("prefill_tc.cu", [], "prefill_tc_host"),
    *[("prefill_tc.cu", [f"-DFLARE_TC_UNIT={u}", f"-DFLARE_TC_MODE={m}"], f"prefill_tc_unit{u}_mode{m}") for u in range(8) for m in range(3)],
    ("noalloc.cu", [], "noalloc"),
    ("bwd_tc.cu", [], "bwd_tc_host"),
    *[("bwd_tc.cu", [f"-DFLARE_BT_UNIT={u}"], f"bwd_tc_unit{u}") for u in range(6)],
    ("bwd_exact.cu", [], "bwd_exact_dispatch"),
    *[("bwd_exact.cu", [f"-DFLARE_WALK_MM={mm}"], f"bwd_exact_mm{mm}") for mm in (2, 8, 16, 32, 64)],
    *[("bwd_standby.cu", [f"-DFLARE_WALK_MM={mm}"], f"bwd_standby_mm{mm}") for mm in (64, 32, 16, 8, 2)],
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; libflare_b200.so cannot be built")


def _digest(src: str, defines: list[str]) -> str:
    h = hashlib.sha256()
    h.update(" ".join(NVCC_FLAGS + defines).encode())
    with open(os.path.join(CSRC, src), "rb") as f:
        h.update(f.read())
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cuh", ".h")):
            with open(os.path.join(CSRC, name), "rb") as f:
                h.update(f.read())
    with open(os.path.join(HERE, "..", "include", "flare_b200.h"), "rb") as f:
        h.update(f.read())
    return h.hexdigest()


def _compile(unit, verbose: bool) -> tuple[str, bool]:
    src, defines, name = unit
    obj = os.path.join(OBJ, name + ".o")
    stamp = obj + ".sha"
    dig = _digest(src, defines)
    if os.path.exists(obj) and os.path.exists(stamp) and open(stamp).read() == dig:
        return obj, False
    cmd = [_nvcc(), *NVCC_FLAGS, *defines, "-c", os.path.join(CSRC, src), "-o", obj]
    if verbose:
        cmd.insert(1, "-Xptxas=-v")
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {name}:\n{res.stdout}\n{res.stderr}")
    if verbose:
        sys.stderr.write(f"--- {name}\n{res.stderr}\n")
    with open(stamp, "w") as f:
        f.write(dig)
    return obj, True


def build(verbose: bool = False, jobs: int | None = None) -> str:
    os.makedirs(OBJ, exist_ok=True)
    jobs = jobs or min(len(UNITS), os.cpu_count() or 4)
    with cf.ThreadPoolExecutor(jobs) as pool:
        results = list(pool.map(lambda u: _compile(u, verbose), UNITS))
    objs = [o for o, _ in results]
    if any(changed for _, changed in results) or not os.path.exists(LIB):
        cmd = [_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB, *objs]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    _build_host()
    return LIB


def _build_host() -> None:
    """The native host layer: plain C++ against torch's headers (no CUDA code in it)."""
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths

    stamp = os.path.join(OBJ, "host_ext.sha")
    dig = _digest("host_ext.cpp", [torch.__version__, sys.version])  # (an extension module of this interpreter)
    if os.path.exists(HOST) and os.path.exists(stamp) and open(stamp).read() == dig:
        return
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           *(f"-isystem{p}" for p in (*include_paths(), sysconfig.get_paths()["include"], os.path.join(cuda, "include"))),
           os.path.join(CSRC, "host_ext.cpp"), "-o", HOST,
           f"-L{lib}", f"-Wl,-rpath,{lib}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for host_ext.cpp:\n{res.stdout}\n{res.stderr}")
    with open(stamp, "w") as f:
        f.write(dig)


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv))
