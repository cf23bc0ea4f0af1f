"""In-tree build of the native code.

These artefacts are produced under ``hetu_galvatron_b200/_lib``:

* ``libhg_sm100.so``  -- every ``csrc/sm100/*.cu`` kernel, compiled by ``nvcc`` for sm_100a only
  (``-gencode arch=compute_100a,code=sm_100a``) and loaded from Python through ``ctypes``.
* ``hg_dp_core*.so`` / ``hg_dataset_helpers*.so`` / ``hg_torch_ops*.so`` -- the host-side C++ modules (pybind11): the
  strategy-search dynamic program, the dataset index builders and the autograd nodes of the layers' operations.

Objects are rebuilt only when a source or header is newer than the object.  ``nvcc`` cross-compiles
without a GPU, so the build also serves as the "does it compile" check on a CPU-only machine.
"""
from __future__ import annotations

import contextlib
import fcntl
import os
import re
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

CSRC = Path(__file__).resolve().parent
PKG = CSRC.parent
LIB_DIR = PKG / "_lib"
OBJ_DIR = CSRC / "build"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--expt-relaxed-constexpr", "--expt-extended-lambda",
    "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _newer(src_paths, target: Path) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(Path(s).stat().st_mtime > t for s in src_paths)


def _run(cmd, log: Path | None = None):
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if log is not None:
        log.write_text(proc.stdout + proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError("command failed: %s\n%s\n%s" % (" ".join(map(str, cmd)), proc.stdout, proc.stderr))
    return proc


def _produce(cmd, target: Path, log: Path | None = None):
    """Run a compiler whose output is ``target``.  The file appears whole or not at all: other processes may be loading it."""
    part = target.with_name(".%s.%d" % (target.name, os.getpid()))
    try:
        _run([*cmd, "-o", str(part)], log)
        os.replace(part, target)
    finally:
        part.unlink(missing_ok=True)


@contextlib.contextmanager
def _one_builder():
    """The ranks of a job that start without the native code build it once: the first one does, the others wait and find it.
    A tree that cannot be written to has no lock, and nothing is built there."""
    with contextlib.ExitStack() as stack:
        with contextlib.suppress(OSError):
            OBJ_DIR.mkdir(exist_ok=True)
            fcntl.flock(stack.enter_context(open(OBJ_DIR / ".lock", "w")), fcntl.LOCK_EX)
        yield


def build_cuda(verbose: bool = False, jobs: int | None = None, debug: bool = False, half: bool = False) -> Path:
    """The kernel library, or one of its variants built from the same sources:

    * ``debug=True``  ``libhg_sm100_debug.so`` (``-DHG_DEBUG_BOUNDS``: index checks that record a status code instead of
      touching memory; see ``HG_BOUNDS_OK`` in sm100_common.cuh), loaded when ``HG_DEBUG_KERNELS=1``;
    * ``half=True``   ``libhg_sm100_fp16.so`` (``-DHG_HALF``: IEEE half as the 16-bit storage type instead of bfloat16;
      see ``hg_lp_t`` in sm100_common.cuh), loaded for ``mixed_precision: fp16`` models."""
    if debug and half:
        raise ValueError("one variant at a time")
    with _one_builder():
        if debug:
            return _build_cuda_variant(OBJ_DIR / "debug", "libhg_sm100_debug.so", ["-DHG_DEBUG_BOUNDS=1"], verbose, jobs)
        if half:
            return _build_cuda_variant(OBJ_DIR / "fp16", "libhg_sm100_fp16.so", ["-DHG_HALF=1"], verbose, jobs)
        return _build_cuda_variant(OBJ_DIR, "libhg_sm100.so", [], verbose, jobs)


def _build_cuda_variant(obj_dir: Path, lib_name: str, extra_flags, verbose: bool, jobs) -> Path:
    src_dir = CSRC / "sm100"
    sources = sorted(src_dir.glob("*.cu"))
    headers = sorted(src_dir.glob("*.cuh")) + sorted(src_dir.glob("*.h"))
    obj_dir.mkdir(exist_ok=True)
    LIB_DIR.mkdir(exist_ok=True)
    nvcc = _nvcc()
    todo = []
    objs = []
    for s in sources:
        o = obj_dir / (s.stem + ".o")
        objs.append(o)
        if _newer([s, *headers], o):
            todo.append((s, o))

    def compile_one(pair):
        s, o = pair
        _produce([nvcc, *NVCC_FLAGS, *extra_flags, "-I", str(src_dir), "-c", str(s)], o, log=obj_dir / (s.stem + ".log"))
        if verbose:
            print("[build] nvcc", s.name)

    with ThreadPoolExecutor(max_workers=jobs or os.cpu_count() or 4) as ex:
        list(ex.map(compile_one, todo))
    lib = LIB_DIR / lib_name
    if todo or _newer(objs, lib):
        _produce([nvcc, "-shared", *map(str, objs), "-lcudart"], lib)
        if verbose:
            print("[build] link", lib.name)
    return lib


def build_host(verbose: bool = False):
    """The modules that need neither CUDA nor torch: the search's dynamic program and the dataset index builders."""
    import pybind11

    LIB_DIR.mkdir(exist_ok=True)
    ext = sysconfig.get_config_var("EXT_SUFFIX")
    inc = ["-I", pybind11.get_include(), "-I", sysconfig.get_paths()["include"]]
    out = []
    with _one_builder():
        for name, src in (("hg_dp_core", "dp_core.cpp"), ("hg_dataset_helpers", "dataset_helpers.cpp")):
            s = CSRC / "host" / src
            if not s.exists():
                continue
            target = LIB_DIR / (name + ext)
            if _newer([s], target):
                _produce(["g++", "-O3", "-std=c++17", "-shared", "-fPIC", "-pthread", *inc, str(s)], target)
                if verbose:
                    print("[build] g++", src)
            out.append(target)
    return out


def _torch_ops() -> Path:
    return LIB_DIR / ("hg_torch_ops" + sysconfig.get_config_var("EXT_SUFFIX"))


def _torch_ops_mark(interface: int) -> str:
    import torch

    return "torch %s, interface %d" % (torch.__version__, interface)


def torch_ops_current(interface: int, unmarked: bool = False) -> bool:
    """Whether the module that is there was built against this interpreter's torch and for this version of the kernel library's
    entry points (``native_interface.h``); ``unmarked``: the answer for one that nothing is known about."""
    mark = _torch_ops().with_suffix(".stamp")
    if not _torch_ops().exists():
        return False
    return mark.read_text() == _torch_ops_mark(interface) if mark.exists() else unmarked


def build_torch_ops(verbose: bool = False) -> Path:
    """``hg_torch_ops``: the autograd nodes of the layers' operations, against this interpreter's torch."""
    from torch.utils.cpp_extension import include_paths, library_paths

    s = CSRC / "host" / "torch_ops.cpp"
    headers = [CSRC / "sm100" / h for h in ("attn_tensor.h", "decoder_step.h", "native_interface.h")]
    interface = int(re.search(r"kHgNativeInterface = (\d+)", headers[-1].read_text()).group(1))
    target = _torch_ops()
    with _one_builder():
        if _newer([s, *headers], target) or not torch_ops_current(interface):
            LIB_DIR.mkdir(exist_ok=True)
            cuda = Path(_nvcc()).resolve().parent.parent / "include"
            inc = [f for p in (*include_paths(), str(cuda), sysconfig.get_paths()["include"]) for f in ("-I", p)]
            libs = ["-L" + p for p in library_paths()]
            _produce(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-DTORCH_EXTENSION_NAME=hg_torch_ops", *inc, str(s), *libs,
                      "-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10", "-lc10_cuda"], target)
            target.with_suffix(".stamp").write_text(_torch_ops_mark(interface))
            if verbose:
                print("[build] g++", s.name)
    return target


def build_all(verbose: bool = False, variants: bool = True):
    host = [*build_host(verbose), build_torch_ops(verbose)]
    cuda = build_cuda(verbose)
    out = [cuda, *host]
    if variants:
        out.append(build_cuda(verbose, debug=True))
        out.append(build_cuda(verbose, half=True))
    return out


def ptxas_report() -> str:
    """Registers / spills / shared memory per kernel, as printed by ``-Xptxas -v`` at build time."""
    parts = []
    for log in sorted(OBJ_DIR.glob("*.log")):
        parts.append("== %s ==\n%s" % (log.stem, log.read_text()))
    return "\n".join(parts)


if __name__ == "__main__":
    built = build_all(verbose=True)
    for b in built:
        print(b)
    if "--report" in sys.argv:
        print(ptxas_report())
