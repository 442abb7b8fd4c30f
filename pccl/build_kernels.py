"""Build and load the native extension ``pccl._C`` for sm_100a.

Counterpart of ``pccl/build_kernels.py:22-116`` in the reference (a JIT
``torch.utils.cpp_extension.load`` of four sources with an sm_70..sm_90 gencode list and
the mpi4py include path).  Differences:

* one target, ``-gencode arch=compute_100a,code=sm_100a``; no MPI, no HIP branch;
* the shared object is kept inside the package (``pccl/_build/pccl_C.so``) together with
  a digest of the sources, and is imported directly when the digest matches, so a
  machine that received a built tree never runs the compiler;
* one process compiles at a time, under a lock that the system releases when its holder
  ends, however it ends; a build that was interrupted is begun again by the next call, and a wait for
  another process has a limit;
* the module is called ``pccl_C`` and is reachable as ``pccl._C``: it does not shadow the
  Python package the way the reference's extension named ``pccl`` does.

``build()`` is idempotent.  The compiler works in ``pccl/_build/obj`` and the finished shared
object is moved into place, followed by its digest, so no other process ever sees half of one.
Callers that start one process per GPU should let rank 0 build
first (``build_rank0_first``), as the reference's callers do with an MPI barrier
(``benchmark_raw_collectives/all_gather.py:45-51``).
"""
from __future__ import annotations

import contextlib
import fcntl
import hashlib
import importlib.machinery
import importlib.util
import os
import shutil
import sys
import time
from pathlib import Path
from typing import List

_HERE = Path(__file__).resolve().parent
CSRC = _HERE / "csrc"
BUILD_DIR = _HERE / "_build"
MODULE_NAME = "pccl_C"
_SO = BUILD_DIR / f"{MODULE_NAME}.so"
_DIGEST = BUILD_DIR / f"{MODULE_NAME}.digest"
_LOCK = BUILD_DIR / f"{MODULE_NAME}.lock"
WAIT_S = 1200.0                  # for another process that is compiling (PCCL_BUILD_WAIT_S)

SOURCES = [
    "bindings.cpp",
    "gemm_bindings.cpp",
    "optim_bindings.cpp",
    "comm.cpp",
    "segments.cpp",
    "collectives.cu",
    "all_reduce_two_phase_bf16.cu",
    "all_reduce_two_phase_f16.cu",
    "all_reduce_two_phase_f32.cu",
    "reduce_scatter_bf16.cu",
    "reduce_scatter_f16.cu",
    "reduce_scatter_f32.cu",
    "gemm_sm100.cu",
    "optim.cu",
    "train_ops.cu",
    "noalloc.cu",
]

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "--expt-relaxed-constexpr", "--expt-extended-lambda",
    "-Xptxas", "-v",
    "-U__CUDA_NO_HALF_OPERATORS__", "-U__CUDA_NO_HALF_CONVERSIONS__",
    "-U__CUDA_NO_BFLOAT16_CONVERSIONS__", "-U__CUDA_NO_HALF2_OPERATORS__",
]
CXX_FLAGS = ["-O3", "-std=c++17", "-Wall", "-Wno-unused-function"]

BUILT = False
_module = None


def _existing_sources() -> List[Path]:
    return [CSRC / s for s in SOURCES if (CSRC / s).exists()]


def source_digest() -> str:
    h = hashlib.sha256()
    files = sorted(p for p in CSRC.iterdir() if p.suffix in (".cpp", ".cu", ".cuh", ".h"))
    for p in files:
        h.update(p.name.encode())
        h.update(p.read_bytes())
    h.update(" ".join(NVCC_FLAGS + CXX_FLAGS).encode())
    return h.hexdigest()


def is_built() -> bool:
    return _SO.exists() and _DIGEST.exists() and _DIGEST.read_text().strip() == source_digest()


def _import_so():
    global _module
    if _module is not None:
        return _module
    import torch  # noqa: F401  (the extension links against libtorch)

    loader = importlib.machinery.ExtensionFileLoader(MODULE_NAME, str(_SO))
    spec = importlib.util.spec_from_file_location(MODULE_NAME, str(_SO), loader=loader)
    mod = importlib.util.module_from_spec(spec)
    loader.exec_module(mod)
    sys.modules[MODULE_NAME] = mod
    _module = mod
    return mod


@contextlib.contextmanager
def _build_lock():
    """Held by the one process that compiles.  An ``flock`` goes away with its holder, so the file that a killed
    build leaves behind (or that travelled here with a copy of the tree) locks nothing."""
    limit = float(os.environ.get("PCCL_BUILD_WAIT_S", WAIT_S))
    with open(_LOCK, "a+") as f:
        deadline = time.monotonic() + limit
        while True:
            try:
                fcntl.flock(f, fcntl.LOCK_EX | fcntl.LOCK_NB)
                break
            except OSError:
                if time.monotonic() >= deadline:
                    f.seek(0)
                    raise TimeoutError(
                        f"pccl: another process ({f.read().strip() or 'unknown'}) has held {_LOCK} for {limit:.0f} s; "
                        "the native extension was not built"
                    ) from None
                time.sleep(0.1)
        f.seek(0)
        f.truncate()
        f.write(f"pid {os.getpid()}")
        f.flush()
        yield


def _publish(src: Path, digest: str) -> None:
    """Move the finished shared object into place; the digest that vouches for it comes last."""
    _DIGEST.unlink(missing_ok=True)
    for dst, put in ((_SO, lambda t: shutil.copy2(src, t)), (_DIGEST, lambda t: t.write_text(digest))):
        tmp = dst.with_name(f"{dst.name}.{os.getpid()}")
        put(tmp)
        os.replace(tmp, dst)


def build(verbose: bool = False, force: bool = False):
    """Compile the extension if the shared object is missing or stale, then import it."""
    global BUILT, _module
    if BUILT and not force and _module is not None:
        return _module
    if force or not is_built():
        BUILD_DIR.mkdir(exist_ok=True)
        with _build_lock():
            if force or not is_built():          # not finished by somebody else while we waited
                _compile(verbose)
    mod = _import_so()
    BUILT = True
    return mod


def _compile(verbose: bool) -> None:
    global _module
    from torch.utils import cpp_extension

    # A toolchain that only ships a static libstdc++ gives the extension its own,
    # never-initialised copy of the iostream locale (integer formatting then crashes).
    # The distribution compiler links the shared libstdc++ that torch itself uses.
    for var, path in (("CXX", "/usr/bin/g++"), ("CC", "/usr/bin/gcc")):
        if os.path.exists(path) and os.environ.get("PCCL_KEEP_COMPILER") != "1":
            os.environ[var] = path
    cuda_home = cpp_extension.CUDA_HOME
    if cuda_home is None or not (Path(cuda_home) / "bin" / "nvcc").exists():
        raise RuntimeError("pccl: nvcc not found; the native extension cannot be built on this machine")
    obj = BUILD_DIR / "obj"
    if (obj / "lock").exists():
        # Nobody else compiles here now, so this belongs to a build that was killed.  cpp_extension would wait without a
        # limit for it to go away; and a compiler that outlived its parent may still be writing to that directory.
        dead = BUILD_DIR / f"obj.{os.getpid()}"
        os.replace(obj, dead)
        shutil.rmtree(dead, ignore_errors=True)
    obj.mkdir(exist_ok=True)
    digest = source_digest()
    mod = cpp_extension.load(
        name=MODULE_NAME,
        sources=[str(p) for p in _existing_sources()],
        extra_cflags=CXX_FLAGS,
        extra_cuda_cflags=NVCC_FLAGS,
        extra_include_paths=[str(CSRC)],
        build_directory=str(obj),
        with_cuda=True,
        verbose=verbose,
    )
    _publish(obj / f"{MODULE_NAME}.so", digest)
    if _module is None:
        _module = mod
        sys.modules[MODULE_NAME] = mod


def load(allow_build: bool = True):
    """Import ``pccl._C``; build it first when that is needed and possible."""
    if _module is not None:
        return _module
    if is_built():
        return _import_so()
    if not allow_build or os.environ.get("PCCL_NO_BUILD") == "1":
        raise ImportError(
            "pccl native extension is missing or stale; run `python -m pccl.build_kernels` on a machine with nvcc"
        )
    return build()


def build_rank0_first(barrier) -> None:
    """Rank 0 compiles, the others wait at ``barrier()`` and then load the result."""
    rank = int(os.environ.get("RANK", os.environ.get("SLURM_PROCID", "0")))
    if rank == 0:
        build()
        barrier()
    else:
        barrier()
        build()


if __name__ == "__main__":
    m = build(verbose="-v" in sys.argv, force="--force" in sys.argv)
    print(f"built {m.__name__} -> {_SO}")
