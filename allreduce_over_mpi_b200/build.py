"""In-tree build of libflextree.so (host planner + sm_100a kernels + runtime).

`python -m allreduce_over_mpi_b200.build` compiles every source under csrc/ with nvcc for
sm_100a only (`-gencode arch=compute_100a,code=sm_100a -lineinfo`) and links one shared
library next to the package.  nvcc cross-compiles without a GPU.  The CUDA runtime is
linked statically and the driver API is resolved at run time, so the library also loads
on a machine without a driver (the planner, cost model and CPU executors work there).

Counterpart of the reference's three separate builds (allreduce_over_mpi/CMakeLists.txt,
cost_model/CMakeLists.txt, vector_add/Makefile, which targets sm_35..sm_86 only).
"""
from __future__ import annotations

import concurrent.futures as cf
import contextlib
import fcntl
import hashlib
import os
import shutil
import subprocess
import sys
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
OBJ = PKG / "csrc" / "build"
LIB = PKG / "lib" / "libflextree.so"
EXT_SOURCES = (CSRC / "python" / "ft_torch.cpp", CSRC / "api" / "ft_types.h")

NVCC = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC,-fopenmp,-Wall,-Wno-unknown-pragmas",
          "-I", str(CSRC), "--expt-relaxed-constexpr"]


def sources() -> list[Path]:
    out = []
    for sub in ("api", "kernels", "runtime"):
        d = CSRC / sub
        if d.is_dir():
            out += sorted(p for p in d.iterdir() if p.suffix in (".cu", ".cpp"))
    return out


def headers_mtime() -> float:
    m = 0.0
    for p in CSRC.rglob("*"):
        if p.suffix in (".h", ".hpp", ".cuh"):
            m = max(m, p.stat().st_mtime)
    return max(m, Path(__file__).stat().st_mtime)


def compile_one(src: Path, verbose: bool, obj_dir: Path = OBJ, defines: tuple = ()) -> tuple[Path, str]:
    obj = obj_dir / (src.stem + ".o")
    cmd = [NVCC, *ARCH, *COMMON, *defines, "-c", str(src), "-o", str(obj)]
    if verbose:
        cmd += ["-Xptxas", "-v"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src.name}:\n{r.stdout}\n{r.stderr}")
    return obj, r.stderr


@contextlib.contextmanager
def _lock():
    """One build at a time in this tree, whatever the number of ranks that find something missing."""
    LIB.parent.mkdir(parents=True, exist_ok=True)
    with open(LIB.parent / ".build.lock", "w") as f:
        fcntl.flock(f, fcntl.LOCK_EX)
        yield


def _produce(cmd: list, out: Path, what: str) -> Path:
    """Run a compiler or linker on a file of its own and put the result in place whole: a process that finds `out` may
    load it at once, and one that has the file before it in use keeps that."""
    part = out.with_name(f".{out.name}.{os.getpid()}")
    try:
        r = subprocess.run([*cmd, "-o", str(part)], capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"{what} failed:\n{r.stdout}\n{r.stderr}")
        os.replace(part, out)
    finally:
        part.unlink(missing_ok=True)
    return out


def build(force: bool = False, verbose: bool = False) -> Path:
    """Compile what changed and link, with the tools and the native call path; returns the path of the shared library."""
    build_lib(force, verbose)
    build_ext(force)
    return LIB


def build_lib(force: bool = False, verbose: bool = False) -> Path:
    """libflextree.so and the tools."""
    with _lock():
        return _build_lib(force, verbose)


def _build_lib(force: bool, verbose: bool) -> Path:
    OBJ.mkdir(parents=True, exist_ok=True)
    hm = headers_mtime()
    srcs = sources()
    todo = []
    for s in srcs:
        o = OBJ / (s.stem + ".o")
        if force or not o.exists() or o.stat().st_mtime < max(s.stat().st_mtime, hm):
            todo.append(s)
    logs = []
    if todo:
        with cf.ThreadPoolExecutor(max_workers=min(len(todo), os.cpu_count() or 4)) as ex:
            for obj, log in ex.map(lambda s: compile_one(s, verbose), todo):
                logs.append(log)
    objs = [OBJ / (s.stem + ".o") for s in srcs]
    if todo or not LIB.exists() or any(o.stat().st_mtime > LIB.stat().st_mtime for o in objs):
        _produce([NVCC, *ARCH, "-shared", "-cudart", "static", *map(str, objs), "-Xcompiler", "-fopenmp", "-lpthread", "-ldl", "-lrt"], LIB, "link")
    build_tools()
    if verbose:
        print("\n".join(logs))
    return LIB


BOUNDS_LIB = PKG / "lib" / "libflextree_bounds.so"


def build_bounds(force: bool = False) -> Path:
    """The debugging build: the same sources with -DFT_BOUNDS, linked as lib/libflextree_bounds.so.  Its collective
    kernels test every run of heap bytes against the heap size before touching it (csrc/kernels/comm_bounds.h);
    select it with FT_LIB=bounds in the environment of the process that loads the library."""
    with _lock():
        return _build_bounds(force)


def _build_bounds(force: bool) -> Path:
    obj_dir = PKG / "csrc" / "build_bounds"
    obj_dir.mkdir(parents=True, exist_ok=True)
    hm = headers_mtime()
    srcs = sources()
    todo = [s for s in srcs if force or not (obj_dir / (s.stem + ".o")).exists()
            or (obj_dir / (s.stem + ".o")).stat().st_mtime < max(s.stat().st_mtime, hm)]
    if todo:
        with cf.ThreadPoolExecutor(max_workers=min(len(todo), os.cpu_count() or 4)) as ex:
            list(ex.map(lambda s: compile_one(s, False, obj_dir, ("-DFT_BOUNDS",)), todo))
    objs = [obj_dir / (s.stem + ".o") for s in srcs]
    if todo or not BOUNDS_LIB.exists():
        _produce([NVCC, *ARCH, "-shared", "-cudart", "static", *map(str, objs), "-Xcompiler", "-fopenmp", "-lpthread", "-ldl", "-lrt"],
                 BOUNDS_LIB, "link")
    return BOUNDS_LIB


def build_tools() -> list[Path]:
    """Native command-line tools next to the library: ft_bench, planner_dump, cost_model_sweep."""
    out = []
    tools = CSRC / "tools"
    hm = headers_mtime()
    for src in sorted(tools.glob("*.cpp")):
        exe = LIB.parent / src.stem
        if exe.exists() and exe.stat().st_mtime >= max(src.stat().st_mtime, hm, LIB.stat().st_mtime):
            out.append(exe)
            continue
        cmd = [NVCC, *ARCH, "-O2", "-std=c++17", "-I", str(CSRC), str(src), "-o", str(exe), "-Xcompiler", "-fopenmp",
               "-L", str(LIB.parent), "-lflextree", "-Xlinker", "-rpath", "-Xlinker", "$ORIGIN", "-lpthread"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"tool build failed for {src.name}:\n{r.stdout}\n{r.stderr}")
        out.append(exe)
    return out


def ext_path() -> Path:
    """Where the native call path for this interpreter, this torch and these sources lies.  The name says what it was
    compiled from and for: an edit, or another torch beside this one, looks for another file."""
    import torch
    h = hashlib.sha256(str(torch.version.git_version).encode())
    for p in EXT_SOURCES:
        h.update(p.read_bytes())
    return LIB.with_name(f"_ft_torch-{sys.implementation.cache_tag}-torch{torch.__version__}-{h.hexdigest()[:16]}.so")


def build_ext(force: bool = False) -> Path:
    """The native call path of the Python entry points (csrc/python/ft_torch.cpp), a CPython module on torch's C++
    headers.  It holds no kernels and does not link libflextree: the loader hands it the entry points."""
    import sysconfig
    import torch
    ext = ext_path()
    if ext.exists() and not force:
        return ext
    root = Path(torch.__file__).resolve().parent
    cuda = Path(NVCC).resolve().parent.parent
    src = EXT_SOURCES[0]
    with _lock():
        if ext.exists() and not force:   # built by the process that had the lock before
            return ext
        cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-w", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
               "-isystem", str(root / "include"), "-isystem", str(root / "include" / "torch" / "csrc" / "api" / "include"),
               "-isystem", str(cuda / "include"), "-isystem", sysconfig.get_paths()["include"], str(src),
               "-L", str(root / "lib"), f"-Wl,-rpath,{root / 'lib'}", "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10"]
        _produce(cmd, ext, src.name)
        for old in ext.parent.glob(ext.name.rpartition("-")[0] + "-*.so"):   # of earlier sources, for the same torch
            if old != ext:
                old.unlink(missing_ok=True)
        return ext


def ensure_built() -> Path:
    """Build the library if it is missing or older than its sources (needs nvcc).  The native call path is looked for,
    and built, where it is loaded (``_lib.native``)."""
    if LIB.exists():
        newest = max([s.stat().st_mtime for s in sources()] + [headers_mtime()])
        if LIB.stat().st_mtime >= newest:
            return LIB
        if not os.path.exists(NVCC):
            return LIB
    return build_lib()


if __name__ == "__main__":
    p = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(p)
    if "--bounds" in sys.argv:
        print(build_bounds(force="--force" in sys.argv))
