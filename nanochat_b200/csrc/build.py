"""Build libnckv.so (all CUDA sources of this directory) for sm_100a with nvcc, and _native.so (binding.cpp: the most
repeated calls from torch tensors to the library) with the host compiler.

Usage:  python -m nanochat_b200.csrc.build [--verbose] [--force]
Both are written next to the package (nanochat_b200/); they are build artefacts and are not tracked.
"""
import fcntl
import os
import subprocess
import sys
import sysconfig
import tempfile
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.dirname(HERE)
OUT = os.path.join(PKG, "libnckv.so")
NATIVE = os.path.join(PKG, "_native.so")
NATIVE_FOR = NATIVE + ".for"  # beside it: what it was built for
BINDING = os.path.join(HERE, "binding.cpp")
SOURCES = ["host.cu", "append.cu", "decode_attn.cu", "decode_small.cu", "prefill_broadcast.cu", "lse_combine.cu",
           "prefill_attn.cu", "p2p_exchange.cu", "glue.cu", "flash_attn_bwd.cu", "host_step.cu",
           "recurrent.cu", "recurrent_f32.cu", "norm_mix.cu", "window_attn.cu", "hyper_norm.cu",
           "gated_linear.cu", "delta.cu", "delta_chunk.cu", "experts.cu", "experts_tc.cu", "experts_pair.cu", "linear_cap.cu"]
HEADERS = ["nckv_common.cuh", "vec_io.cuh", "tc05.cuh", "rope_row.cuh", "recurrent.cuh", "experts.cuh", os.path.join("..", "..", "include", "nckv.h")]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def up_to_date():
    return _library_current() and _native_current()


def _library_current():
    return _newer(OUT, [os.path.join(HERE, s) for s in SOURCES + HEADERS])


def _native_current():
    return native_wanted() is None or (_newer(NATIVE, [BINDING, os.path.join(HERE, HEADERS[-1])]) and native_built_for() == native_wanted())


def native_wanted():
    """The torch and interpreter that _native.so has to be built for: it holds their tensors' and objects' layouts.
    None where there is no torch, or one without CUDA, whose tensors no native call takes."""
    try:
        import torch
    except ImportError:
        return None
    if torch.version.cuda is None:
        return None
    return f"torch {torch.__version__} abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)} {sys.implementation.cache_tag}"


def native_built_for():
    """The same of the _native.so that is there; None where nothing says so."""
    try:
        with open(NATIVE_FOR) as f:
            return f.read()
    except FileNotFoundError:
        return None


def _newer(built, deps):
    if not os.path.exists(built):
        return False
    t = os.path.getmtime(built)
    return all(os.path.getmtime(d) <= t for d in deps + [os.path.abspath(__file__)])


def _binding_command(out):
    import torch
    base = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    include = [os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"),
               os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    libs = ["c10", "c10_cuda", "torch", "torch_cpu", "torch_cuda", "torch_python"]
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-DTORCH_EXTENSION_NAME=_native",
            *[f"-I{d}" for d in include], BINDING, "-o", out, f"-L{os.path.join(base, 'lib')}", *[f"-l{n}" for n in libs],
            f"-L{PKG}", "-l:libnckv.so", "-Wl,-rpath,$ORIGIN"]


def _compile(cmd, verbose):
    res = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or res.returncode != 0:
        sys.stderr.write(" ".join(cmd) + "\n" + res.stdout + res.stderr)
    return res.returncode


def build(verbose=False, force=False):
    """Compile the sources of what is not current side by side, link them, and move each library into place in one
    step; several processes may call this at the same time."""
    if not force and up_to_date():
        return OUT
    with open(os.path.join(PKG, ".build.lock"), "w") as lock:
        fcntl.flock(lock, fcntl.LOCK_EX)
        if not force and up_to_date():  # another process has built it meanwhile
            return OUT
        with tempfile.TemporaryDirectory(dir=PKG, prefix=".build-") as tmp:
            if force or not _library_current():
                _build_library(tmp, verbose)
            if native_wanted() is not None and (force or not _native_current()):
                native = os.path.join(tmp, os.path.basename(NATIVE))
                if _compile(_binding_command(native), verbose):
                    raise RuntimeError("the host compiler failed building _native.so")
                with open(native + ".for", "w") as f:
                    f.write(native_wanted())
                os.replace(native, NATIVE)
                os.replace(native + ".for", NATIVE_FOR)
    return OUT


def _build_library(tmp, verbose):
    nvcc = _nvcc()
    flags = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
             "-Xcompiler", "-fvisibility=hidden"] + (["-Xptxas", "-v"] if verbose else [])
    objs = [os.path.join(tmp, os.path.splitext(s)[0] + ".o") for s in SOURCES]
    jobs = [[nvcc] + flags + ["-c", "-o", o, os.path.join(HERE, s)] for s, o in zip(SOURCES, objs)]
    linked = os.path.join(tmp, os.path.basename(OUT))
    with ThreadPoolExecutor(max(1, min(len(jobs), os.cpu_count() or 1))) as pool:
        failed = any(list(pool.map(lambda cmd: _compile(cmd, verbose), jobs)))
    if failed or _compile([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "--shared", "-o", linked] + objs, verbose):
        raise RuntimeError("nvcc failed building libnckv.so")
    os.replace(linked, OUT)


if __name__ == "__main__":
    build(verbose="--verbose" in sys.argv, force="--force" in sys.argv)
    print(OUT)
