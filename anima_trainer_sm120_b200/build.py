"""In-tree build of ``libanima_b200.so`` (sm_100a only, plain ``nvcc``) and of the
native host path ``_host.so`` (``g++`` against this torch, linked to the library).

``python -m anima_trainer_sm120_b200.build`` compiles every ``csrc/*.cu`` and
``csrc/host/*.cpp`` to an object file (in parallel) and links them into the two
shared objects beside this file. nvcc cross-compiles without a GPU, so this also
runs on a CPU-only box. Objects are rebuilt only when a source or header is newer.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG_DIR = Path(__file__).resolve().parent
CSRC = PKG_DIR / "csrc"
INCLUDE = PKG_DIR.parent / "include"
HOST_SRC = CSRC / "host"
LIB_PATH = PKG_DIR / "libanima_b200.so"
HOST_PATH = PKG_DIR / "_host.so"
OBJ_DIR = PKG_DIR / "build"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libanima_b200.so cannot be built")
    return exe


def _newest(*patterns: tuple[Path, str]) -> float:
    return max((h.stat().st_mtime for d, pat in patterns for h in d.glob(pat)), default=0.0)


def _run(cmd: list[str], what: str, verbose: bool = False) -> None:
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode:
        sys.stderr.write(res.stdout + res.stderr)
    if res.returncode:
        raise RuntimeError(f"{what} failed")


def _host_flags() -> tuple[list[str], list[str]]:
    """Compile and link flags of the host path: torch's headers and libraries, the library beside it."""
    import torch
    root = Path(torch.__file__).resolve().parent
    cuda = Path(_nvcc()).resolve().parents[1]
    inc = [root / "include", root / "include/torch/csrc/api/include", cuda / "include",
           Path(sysconfig.get_paths()["include"])]
    compile_flags = ["-std=c++17", "-O2", "-fPIC", "-DTORCH_EXTENSION_NAME=_host",
                     f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
                     *(f for i in inc for f in ("-isystem", str(i)))]
    link_flags = [f"-L{root / 'lib'}", "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10",
                  f"-L{PKG_DIR}", f"-l:{LIB_PATH.name}", "-Wl,-rpath,$ORIGIN"]
    return compile_flags, link_flags


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile and link the library and the host path; returns the library's path."""
    nvcc = _nvcc()
    OBJ_DIR.mkdir(exist_ok=True)
    sources = sorted(CSRC.glob("*.cu"))
    host_sources = sorted(HOST_SRC.glob("*.cpp"))
    if not sources or not host_sources:
        raise RuntimeError(f"no sources under {CSRC}")
    cu_headers = _newest((CSRC, "*.cuh"), (CSRC, "*.h"), (INCLUDE, "*.h"))
    host_headers = _newest((HOST_SRC, "*.h"), (INCLUDE, "*.h"))
    host_compile, host_link = _host_flags()

    def compile_one(src: Path) -> tuple[Path, bool]:
        host = src.suffix == ".cpp"
        obj = OBJ_DIR / (("host_" if host else "") + src.stem + ".o")
        newest = max(src.stat().st_mtime, host_headers if host else cu_headers)
        stale = force or not obj.exists() or obj.stat().st_mtime < newest
        if stale and host:
            _run(["g++", *host_compile, "-c", str(src), "-o", str(obj)], f"g++ on {src.name}")
        elif stale:
            cmd = [nvcc, *NVCC_FLAGS, "-I", str(INCLUDE), "-c", str(src), "-o", str(obj)]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            _run(cmd, f"nvcc on {src.name}", verbose)
        return obj, stale

    with ThreadPoolExecutor(max_workers=8) as pool:
        results = dict(zip(sources + host_sources, pool.map(compile_one, sources + host_sources)))
    for path, srcs, cmd in ((LIB_PATH, sources, [nvcc, "-shared"]), (HOST_PATH, host_sources, ["g++", "-shared"])):
        if force or not path.exists() or any(results[s][1] for s in srcs):
            flags = ["-cudart", "static", "-ldl"] if path is LIB_PATH else host_link
            _run([*cmd, "-o", str(path), *(str(results[s][0]) for s in srcs), *flags], f"link of {path.name}")
    return LIB_PATH


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
