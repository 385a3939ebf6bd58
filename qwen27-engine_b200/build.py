"""Builds libq27b_attn.so (CUDA kernels + C ABI) for sm_100a and q27b_binding.so (the CPython binding
of the per-layer entry points), in-tree.

nvcc cross-compiles without a GPU. No fast-math flag is used anywhere: the quantisers are
specified in IEEE operations, and the attention kernels ask for the approximate instructions
(ex2.approx) explicitly where they want them.
"""
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libq27b_attn.so")
SOURCES = ["host.cu", "kv_append.cu", "kv_wire.cu", "combine.cu", "decode.cu", "decode_tc.cu", "decode_ws.cu", "decode_wt.cu", "decode_ref.cu", "prefill.cu", "prefill_f16.cu", "sum_norm.cu", "peak_mma.cu", "pager.cu"]
BINDING = os.path.join(HERE, "q27b_binding.so")
BINDING_SOURCES = [os.path.join(CSRC, "binding.cpp"), os.path.join(HERE, "..", "include", "q27b_attn.h")]
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
         "--expt-relaxed-constexpr"]


def _deps():
    hdrs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    hdrs.append(os.path.join(HERE, "..", "include", "q27b_attn.h"))
    return hdrs


def _stale(target, sources):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(s) > t for s in sources)


def _compile(src, verbose):
    obj = os.path.join(OBJ, src.replace(".cu", ".o"))
    path = os.path.join(CSRC, src)
    if not _stale(obj, [path] + _deps()):
        return obj, ""
    cmd = [NVCC] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", path, "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed for %s:\n%s\n%s" % (src, r.stdout, r.stderr))
    return obj, r.stderr


def binding_key():
    """What a binary of the binding belongs to: it uses the C++ interface of torch and the C interface of this Python."""
    import torch
    return "torch %s, CXX11 ABI %d, %s" % (torch.__version__, torch._C._GLIBCXX_USE_CXX11_ABI, sysconfig.get_config_var("SOABI"))


def _binding_stale():
    try:
        with open(os.path.join(OBJ, "binding.key")) as f:
            key = f.read()
    except OSError:
        return True
    return key != binding_key() or _stale(BINDING, BINDING_SOURCES)


def _torch_root():
    import torch
    return os.path.dirname(torch.__file__)


def binding_compile(header_dir=os.path.dirname(BINDING_SOURCES[1])):
    """The compiler and its language options and include folders."""
    import torch
    cmd = [os.environ.get("CXX", "g++"), "-std=c++17", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
           "-I", header_dir]
    inc = os.path.join(_torch_root(), "include")
    for d in (inc, os.path.join(inc, "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"], "/usr/local/cuda/include"):
        cmd += ["-isystem", d]
    return cmd


def _build_binding():
    if not _binding_stale():
        return
    lib = os.path.join(_torch_root(), "lib")
    r = subprocess.run(binding_compile() + ["-O2", "-shared", "-fPIC", BINDING_SOURCES[0], "-o", BINDING, "-L" + lib,
                                            "-Wl,-rpath," + lib, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"],
                       capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("binding.cpp failed:\n%s\n%s" % (r.stdout, r.stderr))
    with open(os.path.join(OBJ, "binding.key"), "w") as f:
        f.write(binding_key())


def build(verbose=False, force=False):
    os.makedirs(OBJ, exist_ok=True)
    if force:
        for f in os.listdir(OBJ):
            os.remove(os.path.join(OBJ, f))
    srcs = [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]
    with ThreadPoolExecutor(max_workers=len(srcs) + 1) as ex:
        binding = ex.submit(_build_binding)
        res = list(ex.map(lambda s: _compile(s, verbose), srcs))
        binding.result()
    objs = [o for o, _ in res]
    if verbose:
        for _, log in res:
            if log:
                print(log)
    if _stale(LIB, objs):
        subprocess.check_call([NVCC, "-shared", "-o", LIB] + objs + ["-cudart", "static"])
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="--force" in sys.argv))
