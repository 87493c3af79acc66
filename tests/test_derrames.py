"""Registers of the 8-bit product's raw forms: what the drain loop spills is paid for at every K-block."""
import os
import re
import shutil
import subprocess

import pytest

RAIZ = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(RAIZ, "jatai_b200", "csrc")
FORMAS = ["32, 1, 1, 128, false", "32, 1, 1, 64, true", "128, 1, 2, 128, false"]


def test_produto_cru_de_8_bits_sem_derrames(tmp_path):
    from jatai_b200 import build
    if not (os.path.exists(build.NVCC) or shutil.which(build.NVCC)):
        pytest.skip("needs nvcc")
    fonte = tmp_path / "formas.cu"
    args = "const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const int8_t*, const int8_t*, const int8_t*, const int8_t*, jt::SaidaGemm, int, int, int, int, int"
    fonte.write_text("#include <cstdio>\n#include <cstring>\n#include <cuda.h>\n#include <cuda_runtime.h>\n" +
                     "".join(f'#include "{f}.cuh"\n' for f in ("comum", "blocos", "gemm_comum", "gemm_simt", "gemm_tc")) +
                     "".join(f"template __global__ void jt::tc::k_gemm_tc<{f}>({args});\n" for f in FORMAS))
    r = subprocess.run([build.NVCC, "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-Xptxas", "-v", "-I", CSRC, "-c", str(fonte), "-o", str(tmp_path / "o.o")],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    derrames = re.findall(r"Function properties for (\S*k_gemm_tc\S*)\n.*?(\d+) bytes spill stores, (\d+) bytes spill loads", r.stderr)
    assert len(derrames) == len(FORMAS)
    assert not [d for d in derrames if d[1] != "0" or d[2] != "0"]
