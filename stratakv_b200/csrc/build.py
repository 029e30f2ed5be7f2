"""Compiles the sm_100a kernel library with nvcc and returns the path of the .so.

One library serves one compute dtype and one head size (the attention kernels
keep a head in registers, so the head size is a compile-time constant).  It
holds the attention kernels alone; everything that does not depend on the head
size is in a library of the dtype, which it names as a needed library beside it
(so whoever loads the first has the symbols of both).  With one library of
everything per dtype and head size the sixteen that the tests use were 441 MB.
An engine therefore compiles only what its model needs, at first use, in a build
folder inside the package (or, if that is not writable, under the system's
temporary folder).  The file names carry a hash of the sources and flags, so
a stale library is never loaded.
"""
from __future__ import annotations

import fcntl
import hashlib
import os
import shutil
import subprocess
import sys
import tempfile
import threading
import time
from pathlib import Path
from typing import Optional

CSRC = Path(__file__).resolve().parent
HEAD_SOURCES = ("attention.cu", "attention_decode.cu", "attention_decode_fused.cu", "attention_prefill.cu", "attention_prefill_tc.cu")
COMMON_SOURCES = ("elementwise.cu", "linear.cu", "gemm_tcgen05.cu", "attention_general.cu", "sampling.cu", "stream_ops.cu",
                  "headwise_linear.cu", "recurrent.cu", "stream_mix.cu", "retention.cu", "latent_finish.cu", "routed_mlp.cu",
                  "short_conv.cu", "time_mix.cu", "normed_rotary.cu", "linear_state.cu", "channel_state.cu")
HEADERS = ("common.cuh", "head_size.cuh")
ARCH_FLAGS = ("-gencode", "arch=compute_100a,code=sm_100a")
COMMON_FLAGS = ("-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden")
DTYPE_CODES = {"float32": 0, "bfloat16": 1}


class BuildError(RuntimeError):
    pass


def find_nvcc() -> str:
    candidates = []
    for var in ("CUDA_HOME", "CUDA_PATH"):
        if os.environ.get(var):
            candidates.append(Path(os.environ[var]) / "bin" / "nvcc")
    found = shutil.which("nvcc")
    if found:
        candidates.append(Path(found))
    candidates.append(Path("/usr/local/cuda/bin/nvcc"))
    for candidate in candidates:
        if candidate.is_file():
            return str(candidate)
    raise BuildError("nvcc not found (looked in CUDA_HOME, PATH and /usr/local/cuda): "
                     "the kernel library cannot be compiled and there is no other backend")


def _source_hash(sources, flags) -> str:
    digest = hashlib.sha256()
    for name in HEADERS + sources:
        digest.update(name.encode())
        digest.update((CSRC / name).read_bytes())
    digest.update(" ".join(flags).encode())
    return digest.hexdigest()[:12]


def _build_dir() -> Path:
    preferred = CSRC / "_build"
    try:
        preferred.mkdir(exist_ok=True)
        probe = preferred / f".write_probe_{os.getpid()}"
        probe.write_text("")
        probe.unlink()
        return preferred
    except OSError:
        fallback = Path(tempfile.gettempdir()) / f"stratakv_b200_build_{os.getuid()}"
        fallback.mkdir(parents=True, exist_ok=True)
        return fallback


def _defines(dtype: str, head_dim: Optional[int] = None) -> tuple:
    return (f"-DSKV_DTYPE={DTYPE_CODES[dtype]}",) + ((f"-DSKV_HEAD_DIM={head_dim}",) if head_dim is not None else ())


def common_library_name(dtype: str) -> str:
    short = "f32" if dtype == "float32" else "bf16"
    return f"libstratakv_{short}_{_source_hash(COMMON_SOURCES, ARCH_FLAGS + COMMON_FLAGS + _defines(dtype))}.so"


def library_name(dtype: str, head_dim: int) -> str:
    flags = ARCH_FLAGS + COMMON_FLAGS + _defines(dtype, head_dim)
    short = "f32" if dtype == "float32" else "bf16"
    # (the common library's name among what is hashed: each names the very one that it was linked against)
    return f"libstratakv_{short}_hd{head_dim}_{_source_hash(HEAD_SOURCES, flags + (common_library_name(dtype),))}.so"


def find_built(dtype: str, head_dim: int):
    name, common = library_name(dtype, head_dim), common_library_name(dtype)
    for folder in (CSRC / "_build", Path(tempfile.gettempdir()) / f"stratakv_b200_build_{os.getuid()}"):
        if (folder / name).is_file() and (folder / common).is_file():
            return folder / name
    return None


def build_library(dtype: str, head_dim: int, verbose: bool = True) -> Path:
    """Path of the library for (dtype, head size); compiled now if it is not there yet."""
    if dtype not in DTYPE_CODES:
        raise BuildError(f"no kernels for dtype {dtype}")
    if head_dim <= 0 or head_dim % 16 != 0 or head_dim > 256:
        raise BuildError(f"head size {head_dim} is not supported: the kernels take multiples of 16 up to 256")
    built = find_built(dtype, head_dim)
    if built is not None:
        return built
    nvcc = find_nvcc()
    folder = _build_dir()
    common, target = folder / common_library_name(dtype), folder / library_name(dtype, head_dim)
    _build_once(common, lambda: _compile(nvcc, f"{dtype}", COMMON_SOURCES, _defines(dtype), (), common, verbose))
    # $ORIGIN: the common library is looked for in the folder of the one that needs it
    beside = ("-L", str(folder), f"-l:{common.name}", "-Xlinker", "-rpath=$ORIGIN")
    _build_once(target, lambda: _compile(nvcc, f"{dtype}, head size {head_dim}", HEAD_SOURCES, _defines(dtype, head_dim), beside,
                                         target, verbose))
    return target


def _build_once(target: Path, compile_it) -> None:
    """One process compiles ``target``, the others wait for it."""
    with open(target.parent / (target.name + ".lock"), "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        try:
            if not target.is_file():
                compile_it()
                drop_older(target)
        finally:
            fcntl.flock(lock, fcntl.LOCK_UN)


def drop_older(target: Path) -> None:
    """Libraries of the same dtype and head size, of other sources, go from the package's own folder: nothing loads them again, and
    some tens of megabytes for every change of a source add up.  The folder for temporary files is shared by every copy of the
    package, each of which may be of other sources, so there they stay."""
    if target.parent != CSRC / "_build":
        return
    stem = target.name.rsplit("_", 1)[0]
    for other in target.parent.glob(f"{stem}_*.so"):
        if other != target and other.name.rsplit("_", 1)[0] == stem:
            other.unlink(missing_ok=True)


def _compile(nvcc: str, what: str, sources, defines, link_flags, target: Path, verbose: bool) -> None:
    start = time.time()
    say = (lambda text: print(f"[stratakv_b200] {text}", file=sys.stderr, flush=True)) if verbose else (lambda text: None)
    say(f"compiling kernels for sm_100a ({what}); this happens once")
    done = threading.Event()

    def heartbeat():
        while not done.wait(5.0):
            say(f"still compiling ({time.time() - start:.0f} s)")

    ticker = threading.Thread(target=heartbeat, daemon=True)
    ticker.start()
    work = Path(tempfile.mkdtemp(prefix="skv_build_", dir=str(target.parent)))
    try:
        jobs = []
        for name in sources:
            obj = work / (name + ".o")
            cmd = [nvcc, *ARCH_FLAGS, *COMMON_FLAGS, *defines, "-I", str(CSRC), "-c", str(CSRC / name), "-o", str(obj)]
            jobs.append((name, obj, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objects = []
        for name, obj, proc in jobs:
            output, _ = proc.communicate()
            if proc.returncode != 0:
                raise BuildError(f"nvcc failed on {name}:\n{output}")
            objects.append(str(obj))
        staged = work / target.name
        link = subprocess.run([nvcc, *ARCH_FLAGS, "-shared", "-o", str(staged), *objects, *link_flags],
                              stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        if link.returncode != 0:
            raise BuildError(f"nvcc failed to link {target.name}:\n{link.stdout}")
        os.replace(staged, target)
    finally:
        done.set()
        shutil.rmtree(work, ignore_errors=True)
    say(f"kernels ready in {time.time() - start:.0f} s: {target.name}")
