"""In-tree build of the CUDA library (nvcc, sm_100a only) and of its torch binding (g++).

`python -m sharq_b200._build` compiles sharq_b200/csrc/*.cu into
sharq_b200/lib/libsharq_b200.so (nvcc cross-compiles without a GPU) and sharq_b200/csrc/torch_bind.cpp
into sharq_b200/lib/sharq_native.so.  Each is built when its own sources are newer.  Callers of the C ABI need only the first: where
torch is not installed the binding is left out.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB_DIR = PKG / "lib"
LIB_PATH = LIB_DIR / "libsharq_b200.so"
BIND_PATH = LIB_DIR / "sharq_native.so"
BIND_TAG_PATH = LIB_DIR / "sharq_native.tag"  # what the binding was built against
BIND_SOURCE = CSRC / "torch_bind.cpp"
HEADER = PKG.parent / "include" / "sharq_b200.h"
SOURCES = ["prepare.cu", "prepare_static.cu", "sp_transition.cu", "quant.cu", "gemm.cu", "allreduce.cu", "decoder_ops.cu",
           "c_api.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
]


def find_nvcc() -> str:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        raise RuntimeError("nvcc not found; the sharq_b200 kernels cannot be built")
    return nvcc


def _older(target: Path, sources: list[Path]) -> bool:
    return not target.exists() or any(s.stat().st_mtime > target.stat().st_mtime for s in sources)


def binding_tag() -> str:
    """The torch and Python that the binding is good for: its C++ ABI is theirs, so another one may load and misbehave."""
    import torch

    return f"torch {torch.__version__} cxx11abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)} python {sysconfig.get_config_var('EXT_SUFFIX')}"


def binding_matches() -> bool:
    """Whether the binding was built against the torch and Python that are running."""
    return BIND_TAG_PATH.exists() and BIND_TAG_PATH.read_text() == binding_tag()


def _bind_command(out: Path) -> list[str]:
    import torch

    root = Path(torch.__file__).resolve().parent
    cuda = Path(find_nvcc()).resolve().parent.parent / "include"
    includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", sysconfig.get_paths()["include"], cuda]
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            *[a for i in includes for a in ("-isystem", str(i))], str(BIND_SOURCE), "-o", str(out),
            f"-L{root / 'lib'}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", f"-L{LIB_DIR}", "-l:" + LIB_PATH.name,
            "-Wl,-rpath,$ORIGIN"]


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile the library and the binding, each if it is missing or older than its sources."""
    if force or _older(LIB_PATH, [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh"), HEADER]):
        _build_library(verbose)
    try:
        import torch  # noqa: F401
    except ImportError:
        print("torch is not installed: built the C library without its torch binding", file=sys.stderr)
        return LIB_PATH
    if force or _older(BIND_PATH, [BIND_SOURCE, HEADER]) or not binding_matches():
        _build_binding()
    return LIB_PATH


def _build_library(verbose: bool) -> None:
    nvcc = find_nvcc()
    LIB_DIR.mkdir(exist_ok=True)
    obj_dir = LIB_DIR / "obj"
    obj_dir.mkdir(exist_ok=True)
    procs = []
    for src in SOURCES:
        cmd = [nvcc, *NVCC_FLAGS, "-c", str(CSRC / src), "-o", str(obj_dir / (src + ".o"))]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}")
    tmp = LIB_PATH.with_suffix(".so.tmp")  # linked beside the target and moved into place, so a reader never sees half a file
    cmd = [nvcc, "-shared", "-o", str(tmp)] + [str(obj_dir / (s + ".o")) for s in SOURCES]
    subprocess.run(cmd, check=True)
    os.replace(tmp, LIB_PATH)


def _build_binding() -> None:
    tmp = BIND_PATH.with_suffix(".so.tmp")
    subprocess.run(_bind_command(tmp), check=True)
    BIND_TAG_PATH.unlink(missing_ok=True)  # no moment with this binding and another one's tag
    os.replace(tmp, BIND_PATH)
    BIND_TAG_PATH.write_text(binding_tag())


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
