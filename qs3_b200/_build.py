"""In-tree build of ``libqs3moe.so`` (CUDA, sm_100a only).

``python -m qs3_b200._build`` compiles every translation unit under
``qs3_b200/csrc`` with nvcc for ``sm_100a`` and links them into
``qs3_b200/libqs3moe.so``, and the descriptor-marshalling extension ``qs3_b200/_marshal.so``
with g++. nvcc cross-compiles without a GPU, so this also runs
on a CPU-only machine; the shared object is what a GPU machine loads.
"""
from __future__ import annotations

import concurrent.futures as cf
import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
SRC_DIR = os.path.join(PKG_DIR, "csrc")
OBJ_DIR = os.path.join(SRC_DIR, "build")
LIB_PATH = os.path.join(PKG_DIR, "libqs3moe.so")
MARSHAL_PATH = os.path.join(PKG_DIR, "_marshal.so")
MARSHAL_TAG_PATH = os.path.join(OBJ_DIR, "marshal.tag")
CHECKED_LIB_PATH = os.path.join(PKG_DIR, "libqs3moe_checked.so")

SOURCES = ["context.cu", "router.cu", "routing.cu", "gemm.cu", "gemm_api.cu", "nvfp4.cu", "moe.cu",
           "peak_probe.cu", "fp8.cu", "fp8_rows.cu", "fp8_stream.cu", "bf16_stream.cu", "gemv.cu", "norm.cu", "loader.cu", "nvfp4_decode.cu", "gemm_dense.cu", "gemm_splitk.cu", "gemm_pair.cu", "failure.cu"]
HEADERS = ["common.cuh", "nvfp4.cuh", "tcgen05.cuh", "topk.cuh", "route_sort.cuh", "fp8.cuh", os.path.join("..", "..", "include", "qs3_moe.h")]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-std=c++17", "-O3", "-lineinfo",
    "-Xcompiler", "-fPIC",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or install the CUDA toolkit")


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def marshal_tag() -> str:
    """What the marshalling extension is built against beside its sources: torch's C++ interface and Python's."""
    import importlib.metadata
    import sysconfig
    return f"{importlib.metadata.version('torch')} {sysconfig.get_config_var('SOABI')}"


def _marshal_stale() -> bool:
    if _stale(MARSHAL_PATH, [os.path.join(SRC_DIR, "marshal.cpp"), os.path.join(SRC_DIR, HEADERS[-1])]):
        return True
    if not os.path.exists(MARSHAL_TAG_PATH):
        return True
    with open(MARSHAL_TAG_PATH) as f:
        return f.read() != marshal_tag()


def build_marshal(force: bool = False) -> str:
    """Compile the Python extension that fills descriptors from torch tensors (``csrc/marshal.cpp``)."""
    if force or _marshal_stale():
        import sysconfig

        import torch
        src = os.path.join(SRC_DIR, "marshal.cpp")
        base = os.path.dirname(torch.__file__)
        cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", src, "-o", MARSHAL_PATH,
               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
               f'-DQS3_TORCH_VERSION="{torch.__version__}"',
               *(f"-I{d}" for d in (os.path.join(base, "include"),
                                    os.path.join(base, "include", "torch", "csrc", "api", "include"),
                                    sysconfig.get_paths()["include"])),
               f"-L{os.path.join(base, 'lib')}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"g++ failed on {src}:\n{r.stdout}\n{r.stderr}")
        os.makedirs(OBJ_DIR, exist_ok=True)
        with open(MARSHAL_TAG_PATH, "w") as f:
            f.write(marshal_tag())
    return MARSHAL_PATH


def build(force: bool = False, verbose: bool = False, checked: bool = False) -> str:
    """Compile the library in-tree. ``checked`` builds the variant with device-side input
    validation (``-DQSFI_ENABLE_CHECKED_VALIDATION=1``, as upstream's checked test binary):
    ``libqs3moe_checked.so`` next to the release ``libqs3moe.so``."""
    nvcc = _nvcc()
    obj_dir = OBJ_DIR + ("_checked" if checked else "")
    lib_path = CHECKED_LIB_PATH if checked else LIB_PATH
    flags = NVCC_FLAGS + (["-DQSFI_ENABLE_CHECKED_VALIDATION=1"] if checked else [])
    os.makedirs(obj_dir, exist_ok=True)
    headers = [os.path.join(SRC_DIR, h) for h in HEADERS]
    jobs = []
    for src in SOURCES:
        s = os.path.join(SRC_DIR, src)
        o = os.path.join(obj_dir, src.replace(".cu", ".o"))
        if force or _stale(o, [s] + headers):
            jobs.append((s, o))

    def compile_one(job):
        s, o = job
        cmd = [nvcc, *flags, "-c", s, "-o", o]
        if verbose:
            cmd[1:1] = ["-Xptxas", "-v"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        return s, r

    with cf.ThreadPoolExecutor(max_workers=min(8, len(jobs) + 1)) as pool:
        marshal = pool.submit(build_marshal, force)
        for s, r in pool.map(compile_one, jobs):
            if verbose and r.stderr:
                sys.stderr.write(r.stderr)
            if r.returncode != 0:
                raise RuntimeError(f"nvcc failed on {s}:\n{r.stdout}\n{r.stderr}")
        marshal.result()
    objs = [os.path.join(obj_dir, s.replace(".cu", ".o")) for s in SOURCES]
    if force or jobs or _stale(lib_path, objs):
        cmd = [nvcc, "-shared", "-o", lib_path, *objs, "-Xcompiler", "-fPIC"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return lib_path


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv, checked=True))
