"""Build libdfa3d_b200.so (CUDA kernels + C ABI), libdfa3d_rates.so (memory-primitive rate probes,
measurement code) and _native.so (host path of the autograd Functions) in-tree, for sm_100a.

The library is plain CUDA C++ behind an ``extern "C"`` interface (include/dfa3d_b200.h) without torch
headers; only _native.so, which contains no kernels, is compiled against torch, and carries the version of
the torch it was compiled against: with another one installed it is built anew.  The results are written
next to the Python package (``dfa3d_b200/``) so that they are found without any install step.
"""
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "dfa3d_b200", "libdfa3d_b200.so")
SOURCES = ["dfa3d_forward.cu", "dfa3d_forward_packed.cu", "dfa3d_backward.cu", "dfa3d_backward_packed.cu", "dfa3d_rebatch.cu", "dfa3d_dist_producer.cu",
           "dfa3d_fp64.cu", "dfa3d_layer_ops.cu", "dfa3d_capi.cu"]
RATES_SRC = os.path.join(CSRC, "rates", "dfa3d_rates.cu")
RATES_OUT = os.path.join(HERE, "dfa3d_b200", "libdfa3d_rates.so")
NATIVE_SRC = [os.path.join(CSRC, "binding", f) for f in ("dfa3d_torch.cpp", "dfa3d_torch_layers.cpp")]
NATIVE_OUT = os.path.join(HERE, "dfa3d_b200", "_native.so")
INCLUDE = os.path.join(HERE, "..", "include")
NVCC_FLAGS = ["-O3", "-I", INCLUDE, "-std=c++17", "-lineinfo", "-gencode", "arch=compute_100a,code=sm_100a",
              "-Xcompiler", "-fPIC", "-Xptxas", "-v"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _cuda_include():
    """The headers of the toolkit that `_nvcc` belongs to."""
    nvcc = shutil.which(_nvcc()) or "/usr/local/cuda/bin/nvcc"
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


def _built_for():
    """What _native.so is compiled against; it holds this text."""
    import sysconfig
    import torch
    return f"torch {torch.__version__} python {sysconfig.get_config_var('SOABI')}"


def _native_command():
    """g++ command of the torch binding: header and library folders come from the installed torch."""
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    inc = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
           sysconfig.get_paths()["include"], _cuda_include()]
    lib = os.path.join(root, "lib")
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DDFA3D_BUILT_FOR="{_built_for()}"',
            "-I", INCLUDE,
            *[a for i in inc for a in ("-isystem", i)], *NATIVE_SRC, "-o", NATIVE_OUT, "-L", lib,
            "-Wl,-rpath," + lib, "-ltorch_python", "-ltorch", "-ltorch_cuda", "-ltorch_cpu", "-lc10_cuda", "-lc10"]


def needs_build():
    outs = (OUT, RATES_OUT, NATIVE_OUT)
    if not all(os.path.exists(o) for o in outs):
        return True
    with open(NATIVE_OUT, "rb") as f:
        if _built_for().encode() not in f.read():
            return True
    t = min(os.path.getmtime(o) for o in outs)
    deps = [os.path.join(d, f) for d, _, fs in os.walk(CSRC) for f in fs]
    deps.append(os.path.join(HERE, "..", "include", "dfa3d_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    """Compile every .cu of csrc/ in parallel and link the shared library.  Returns its path."""
    if not force and not needs_build():
        return OUT
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    procs = []
    for src in SOURCES:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        cmd = [_nvcc(), *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, obj, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                                                 text=True)))
    rates = subprocess.Popen([_nvcc(), *NVCC_FLAGS, "-shared", "-cudart", "shared", RATES_SRC, "-o", RATES_OUT],
                             stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    native = subprocess.Popen(_native_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    objs = []
    for src, obj, pr in procs:
        log, _ = pr.communicate()
        with open(os.path.join(objdir, src + ".log"), "w") as f:
            f.write(log)
        if pr.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{log[-4000:]}")
        if verbose:
            print(log)
        objs.append(obj)
    cmd = [_nvcc(), "-shared", "-o", OUT, *objs, "-gencode", "arch=compute_100a,code=sm_100a",
           "-cudart", "shared"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}")
    log, _ = rates.communicate()
    with open(os.path.join(objdir, "dfa3d_rates.cu.log"), "w") as f:
        f.write(log)
    if rates.returncode != 0:
        raise RuntimeError(f"nvcc failed on dfa3d_rates.cu:\n{log[-4000:]}")
    log, _ = native.communicate()
    if native.returncode != 0:
        raise RuntimeError(f"g++ failed on csrc/binding:\n{log[-4000:]}")
    return OUT


if __name__ == "__main__":
    print(build(force="-f" in sys.argv, verbose="-v" in sys.argv))
