"""Builds libtessiq_b200.so, in tree, for sm_100a, and the Python module beside it that launches from it.

    python -m tessiq_b200.build [--force] [--verbose]

Each `csrc/*.cu` is compiled to an object with nvcc (in parallel) and the objects are linked into
`tessiq_b200/libtessiq_b200.so` with the CUDA runtime linked statically; `csrc/launcher.cpp` becomes
`tessiq_b200/_launcher.so` (torch's headers, the host compiler). NVRTC (used to instantiate
fused elementwise kernels) is opened at run time, so the library loads on a machine without a GPU
or a driver. Objects are rebuilt only when a source or header is newer.
"""

from __future__ import annotations

import argparse
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PACKAGE = Path(__file__).resolve().parent
ROOT = PACKAGE.parent
CSRC = PACKAGE / "csrc"
OBJECTS = CSRC / "build"
LIBRARY = PACKAGE / "libtessiq_b200.so"
LAUNCHER = PACKAGE / "_launcher.so"

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = [
    "-O3",
    "-std=c++17",
    "-lineinfo",
    "--expt-relaxed-constexpr",
    "--extended-lambda",
    "-Xcompiler",
    "-fPIC,-Wall,-Wno-unknown-pragmas",
    f"-I{ROOT / 'include'}",
    f"-I{CSRC}",
]


def nvcc() -> str:
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(found):
        raise RuntimeError("nvcc not found; tessiq_b200 has no CPU build")
    return found


def _newest_header() -> float:
    headers = list(CSRC.glob("*.h")) + list((ROOT / "include").glob("*.h"))
    return max(h.stat().st_mtime for h in headers)


def _compile(source: Path, force: bool, verbose: bool) -> Path:
    target = OBJECTS / (source.stem + ".o")
    stamp = max(source.stat().st_mtime, _newest_header(), Path(__file__).stat().st_mtime)
    if not force and target.exists() and target.stat().st_mtime >= stamp:
        return target
    command = [nvcc(), *ARCH, *COMMON, "-c", str(source), "-o", str(target)]
    if verbose:
        command.insert(1, "-Xptxas=-v")
        print(" ".join(command), flush=True)
    result = subprocess.run(command, capture_output=True, text=True)
    if result.returncode != 0:
        raise RuntimeError(f"nvcc failed on {source.name}:\n{result.stdout}\n{result.stderr}")
    if verbose or result.stderr.strip():
        sys.stderr.write(result.stderr)
    return target


def build(force: bool = False, verbose: bool = False) -> Path:
    OBJECTS.mkdir(parents=True, exist_ok=True)
    sources = sorted(CSRC.glob("*.cu"))
    if not sources:
        raise RuntimeError(f"no CUDA sources under {CSRC}")
    with ThreadPoolExecutor(max_workers=min(8, len(sources))) as pool:
        objects = list(pool.map(lambda s: _compile(s, force, verbose), sources))
    newest = max(o.stat().st_mtime for o in objects)
    if force or not LIBRARY.exists() or LIBRARY.stat().st_mtime < newest:
        command = [
            nvcc(), *ARCH, "-shared", "-o", str(LIBRARY), *map(str, objects),
            "-cudart", "static", "-Xcompiler", "-fPIC", "-ldl", "-lpthread",
        ]
        result = subprocess.run(command, capture_output=True, text=True)
        if result.returncode != 0:
            raise RuntimeError(f"linking {LIBRARY.name} failed:\n{result.stdout}\n{result.stderr}")
    build_launcher(force, verbose)
    return LIBRARY


def launcher_is_current(built_for: str) -> bool:
    """Whether the module is newer than its sources and was built for this torch and Python."""
    sources = (CSRC / "launcher.cpp", ROOT / "include" / "tessiq_b200.h", Path(__file__))
    noted = OBJECTS / "launcher.built_for"
    return (LAUNCHER.exists() and LAUNCHER.stat().st_mtime >= max(s.stat().st_mtime for s in sources)
            and noted.exists() and noted.read_text() == built_for)


def build_launcher(force: bool = False, verbose: bool = False) -> Path:
    import sysconfig

    import torch

    built_for = f"torch {torch.__version__}, Python {sys.version_info.major}.{sys.version_info.minor}"
    if not force and launcher_is_current(built_for):
        return LAUNCHER
    OBJECTS.mkdir(parents=True, exist_ok=True)
    home = Path(torch.__file__).resolve().parent
    cuda = Path(nvcc()).resolve().parent.parent
    command = [
        os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
        f'-DTQ_BUILT_FOR="{built_for}"',
        *[f"-I{path}" for path in (home / "include", home / "include" / "torch" / "csrc" / "api" / "include", cuda / "include",
                                   sysconfig.get_paths()["include"], ROOT / "include")],
        str(CSRC / "launcher.cpp"), "-o", str(LAUNCHER), f"-L{home / 'lib'}", "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10", "-ldl",
    ]
    if verbose:
        print(" ".join(command), flush=True)
    result = subprocess.run(command, capture_output=True, text=True)
    if result.returncode != 0:
        raise RuntimeError(f"building {LAUNCHER.name} failed:\n{result.stdout}\n{result.stderr}")
    (OBJECTS / "launcher.built_for").write_text(built_for)
    return LAUNCHER


def main() -> None:
    parser = argparse.ArgumentParser(description=__doc__)
    parser.add_argument("--force", action="store_true")
    parser.add_argument("--verbose", action="store_true", help="print commands and ptxas -v output")
    arguments = parser.parse_args()
    print(build(arguments.force, arguments.verbose))


if __name__ == "__main__":
    main()
