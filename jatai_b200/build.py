"""Builds the native pieces in-tree: jatai_b200/libjatai_b200.so (the CUDA library, sm_100a only) and jatai_b200/_nativo.so (the host half
of the operator launcher, a CPython extension against PyTorch's headers)."""
import os
import subprocess
import sys

AQUI = os.path.dirname(os.path.abspath(__file__))
FONTE = os.path.join(AQUI, "csrc", "jatai_b200.cu")
SAIDA = os.path.join(AQUI, "libjatai_b200.so")
FONTE_NATIVO, SAIDA_NATIVO, MARCA_NATIVO = os.path.join(AQUI, "csrc", "nativo.cpp"), os.path.join(AQUI, "_nativo.so"), os.path.join(AQUI, "_nativo.versao")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-shared", "-Xcompiler", "-fPIC"]


def fontes():
    d = os.path.join(AQUI, "csrc")
    return [os.path.join(d, f) for f in sorted(os.listdir(d)) if f.endswith((".cu", ".cuh"))]


def desatualizada():
    if not os.path.exists(SAIDA):
        return True
    t = os.path.getmtime(SAIDA)
    return any(os.path.getmtime(f) > t for f in fontes())


def _marca():
    """What the module is built against: it uses the C++ interface of this PyTorch and the C interface of this Python."""
    import torch
    return f"{torch.__version__} python {sys.version_info[0]}.{sys.version_info[1]}"


def nativo_em_dia():
    """Whether the module is newer than its source and was built against the PyTorch and the Python that run."""
    if not (os.path.exists(SAIDA_NATIVO) and os.path.exists(MARCA_NATIVO)) or os.path.getmtime(SAIDA_NATIVO) < os.path.getmtime(FONTE_NATIVO):
        return False
    with open(MARCA_NATIVO) as fh:
        return fh.read().strip() == _marca()


def build_nativo(force=False):
    if not force and nativo_em_dia():
        return SAIDA_NATIVO
    import sysconfig
    import torch
    from torch.utils import cpp_extension as ce
    raiz = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DJT_MARCA="{_marca()}"']
    cmd += [f"-I{d}" for d in ce.include_paths("cuda")] + ["-I" + sysconfig.get_paths()["include"], FONTE_NATIVO, "-o", SAIDA_NATIVO]
    cmd += [f"-L{d}" for d in ce.library_paths("cuda")] + [f"-Wl,-rpath,{raiz}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    with open(MARCA_NATIVO, "w") as fh:
        fh.write(_marca() + "\n")
    return SAIDA_NATIVO


def build(force=False, verbose=False):
    """Compile what is older than its sources.  Raises if a compiler fails."""
    build_nativo(force)
    if not force and not desatualizada():
        return SAIDA
    cmd = [NVCC] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + [FONTE, "-o", SAIDA]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    if verbose:
        print(r.stderr)
    return SAIDA


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
