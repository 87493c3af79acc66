"""The order of the half-precision product's barriers (jatai_b200/csrc/gemm_h_ordem.cuh), without a GPU: the loops of its loading and multiplying
warps, compiled for the host over simulated barriers, in drawn schedules in which loads complete in any order and warps stall anywhere."""
import os
import subprocess

import pytest

RAIZ = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def programa(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("ordem") / "ordem_gemm_h")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(RAIZ, "jatai_b200", "csrc"), os.path.join(RAIZ, "tests", "ordem_gemm_h.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("tiles", ["plain", "plain64", "plain128", "round", "sum"])
@pytest.mark.parametrize("pedacos", [1, 2, 3, 8, 16])
def test_cada_pedaco_uma_vez(programa, tiles, pedacos):
    """28 tiles of one kind: every chunk is multiplied when it has been loaded and put out once, in its order, and every wait ends."""
    if tiles == "plain128":
        pedacos *= 2                                   # (a K-block of 128 is two chunks)
    r = subprocess.run([programa, tiles, str(pedacos), "400"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_um_pedaco_por_tile(programa):
    """Tiles of one chunk (K <= 64), rounded and summed ones in any order: a multiplying warp that falls behind still finds its plans."""
    r = subprocess.run([programa, "mixed", "1", "2000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("pedacos", [2, 3, 4, 5, 8, 12, 16])
def test_arredondados_e_somados(programa, pedacos):
    """Rounded and summed tiles in any order, sums of 2 to 16 chunks: no multiplying warp takes a chunk for loaded, or a stage for drained, by the parity
    of a phase that it has not followed."""
    r = subprocess.run([programa, "mixed", str(pedacos), "2000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
