"""Build libanalog_b200.so (sm_100a, nvcc) and the Python extension that calls it (g++) in-tree.

    python aihwkit-lightning_b200/build.py [--force]

Both land in ``aihwkit_lightning_b200/lib/`` next to the Python package that loads them.  nvcc cross-compiles without a GPU.
Without torch or Python's headers only the C library is built: the extension is for the Python package, which needs both.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT_DIR = os.path.join(HERE, "aihwkit_lightning_b200", "lib")
OUT = os.path.join(OUT_DIR, "libanalog_b200.so")
HOST_OUT = os.path.join(OUT_DIR, "_host_calls.so")
SOURCES = [
    "api.cu",
    "reduce_kernels.cu",
    "prepass_kernels.cu",
    "ragged_kernels.cu",
    "split_kernels.cu",
    "gemm_simt.cu",
    "gemm_tcgen05_fwd.cu",
    "gemm_tcgen05_bwd.cu",
    "gemm_smallm.cu",
    "backward_kernels.cu",
    "conv_kernels.cu",
    "peer_kernels.cu",
    "decoder_glue_kernels.cu",
]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-lineinfo", "-std=c++17", "--expt-relaxed-constexpr", "--extended-lambda",
    "-Xcompiler", "-fPIC,-ffp-contract=off",
    "-Xptxas", "-v",
]


def _torch_version():
    """Version of the installed torch, or None where the extension cannot be built."""
    import sysconfig

    try:
        import torch
    except ImportError:
        return None
    return torch.__version__ if os.path.exists(os.path.join(sysconfig.get_paths()["include"], "Python.h")) else None


def _host_command():
    """g++ command of the extension: torch's headers, linked against the library next to it."""
    import sysconfig

    from torch._C import _GLIBCXX_USE_CXX11_ABI
    from torch.utils.cpp_extension import include_paths, library_paths

    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    includes = [*include_paths(), sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    return ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f'-DAL_TORCH_VERSION="{_torch_version()}"',
            f"-D_GLIBCXX_USE_CXX11_ABI={int(_GLIBCXX_USE_CXX11_ABI)}",
            *[f"-isystem{p}" for p in includes], os.path.join(CSRC, "host_calls.cpp"), "-o", HOST_OUT,
            *[f"-L{p}" for p in library_paths()], "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python",
            f"-L{OUT_DIR}", "-l:libanalog_b200.so", "-Wl,-rpath,$ORIGIN"]


def _stale() -> bool:
    version = _torch_version()
    outputs = [OUT] if version is None else [OUT, HOST_OUT]
    if not all(os.path.exists(p) for p in outputs):
        return True
    if version is not None and f"built for torch {version};".encode() not in open(HOST_OUT, "rb").read():
        return True
    built = min(os.path.getmtime(p) for p in outputs)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    deps.append(os.path.join(HERE, "..", "include", "analog_b200.h"))
    return any(os.path.getmtime(p) > built for p in deps)


def build_host() -> None:
    """The extension, or a line that says why there is none."""
    version = _torch_version()
    if version is None:
        print("torch or Python.h not found: the C library was built, the extension of the Python package was not")
        return
    res = subprocess.run(_host_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout)
        raise RuntimeError("g++ failed on host_calls.cpp")


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not _stale():
        return OUT
    os.makedirs(OUT_DIR, exist_ok=True)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    objs = []
    procs = []
    for src in SOURCES:
        obj = os.path.join(OUT_DIR, src.replace(".cu", ".o"))
        objs.append(obj)
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    log = []
    for src, proc in procs:
        out, _ = proc.communicate()
        log.append(f"==== {src}\n{out}")
        if proc.returncode != 0:
            sys.stderr.write("\n".join(log))
            raise RuntimeError(f"nvcc failed on {src}")
    with open(os.path.join(OUT_DIR, "ptxas.log"), "w") as fh:
        fh.write("\n".join(log))
    link = [nvcc, "-shared", "-o", OUT, *objs, "-lcudart", "-ldl"]
    res = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout)
        raise RuntimeError("link failed")
    build_host()
    if verbose:
        print("\n".join(log))
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
