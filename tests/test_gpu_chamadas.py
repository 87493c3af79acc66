"""Calls in the forms that the other tests do not use: tensors that start anywhere in a larger buffer, pairs given as lists, several streams,
little memory, a first call inside a recording, very many heads.  Everything against the oracle, or against the same operator called
the plain way."""
import tempfile

import pytest
import torch

import casos
from oracle import spec
from test_gpu_ops import compara, para_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture
def amb():
    from jatai_b200 import ops, registro
    ops.define_blk(32)
    reg = registro.Registro(tempfile.mkdtemp(), "chamadas", vigiar=True, eco=False, salvar=False)
    oc = ops.OpsCuda(reg)
    reg.novo_passo(0)
    yield ops, oc, reg
    ops.define_blk(32)
    ops.ATENCAO_LIMITE = False
    oc.lib.jt_gemm_via(0)


def deslocado(t, n):
    """A contiguous tensor equal to `t` that starts n elements into a buffer of its own (torch aligns the buffer to 512 bytes)."""
    b = torch.zeros(t.numel() + n, dtype=t.dtype, device="cuda")
    v = b[n:].view(t.shape)
    v.copy_(t)
    return v


@pytest.mark.parametrize("blk,M,N,K", [(32, 256, 256, 2048), (128, 256, 256, 2048), (32, 64, 128, 1024)])
def test_produto_com_expoentes_em_qualquer_endereco(amb, blk, M, N, K):
    """Exponent tensors at every byte offset of a word, on sizes whose rows have a multiple of four exponents: the half-precision
    path (chosen by itself, and forced) reads whole words of them only where they are aligned."""
    ops, oc, reg = amb
    ops.define_blk(blk)
    G = casos.Gen(5 + M + blk, blk)
    A, B = para_gpu(G.bloco(M, K, espalha=6, zera=0.1)), para_gpu(G.bloco(N, K, espalha=6, zera=0.1))
    s = spec.Spec(blk)
    ref = [s.gemm(A, B), s.gemm(A, B, cru=True)]
    for via in (0, 4):
        oc.lib.jt_gemm_via(via)
        for n in (1, 2, 3):
            A1, B1 = (A[0], deslocado(A[1], n)), (B[0], deslocado(B[1], 4 - n))
            assert A1[1].data_ptr() % 4 and B1[1].data_ptr() % 4
            for cru in (False, True):
                compara(f"gemm, exponents at offset {n}, via {via}, cru {cru}", oc.gemm(A1, B1, cru=cru), ref[cru])


@pytest.mark.parametrize("blk,Bt,T,H,hd", [(32, 2, 64, 8, 4), (32, 1, 160, 8, 4), (128, 1, 288, 32, 4), (32, 2, 96, 4, 16), (32, 1, 160, 2, 64)])
def test_atencao_em_qualquer_endereco(amb, blk, Bt, T, H, hd):
    """P at addresses that are no multiple of 16 (or of 4), and for heads of 4 mantissas at a multiple of 4 that is none of 8: what the
    kernels with wider accesses cannot take goes to the general ones."""
    ops, oc, reg = amb
    ops.define_blk(blk)
    D, M = H * hd, Bt * T
    G = casos.Gen(17 + T + H, blk)
    qkv, go = para_gpu(G.bloco(M, 3 * D, espalha=4, zera=0.02)), para_gpu(G.bloco(M, D, e0=-20, espalha=4))
    o, P = oc.atencao(qkv, Bt, T, H)
    ref = oc.atencao_back(go, qkv, P, Bt, T, H)
    s = spec.Spec(blk)
    compara("atencao", [*o, P], [*casos.plano(s.atencao(qkv, Bt, T, H))])
    compara("atencao_back", ref, s.atencao_back(go, qkv, P, Bt, T, H))
    for n in (1, 4, 8):
        compara(f"atencao_back, P at offset {n}", oc.atencao_back(go, qkv, deslocado(P, n), Bt, T, H), ref)
    for n in (4, 8, 12) if hd == 4 else ():
        q2, g2 = (deslocado(qkv[0], n), deslocado(qkv[1], 1)), (deslocado(go[0], n), deslocado(go[1], 3))
        o2, P2 = oc.atencao(q2, Bt, T, H)
        compara(f"atencao, mantissas at offset {n}", [*o2, P2], [*o, P])
        compara(f"atencao_back, mantissas at offset {n}", oc.atencao_back(g2, q2, P, Bt, T, H), ref)
        compara(f"atencao_back, everything at offset {n}", oc.atencao_back(g2, q2, deslocado(P, n), Bt, T, H), ref)
