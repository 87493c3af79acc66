"""Parity of the CUDA kernels with the oracle, through the C ABI (jatai_b200.ops.OpsCuda -> libjatai_b200.so).

Every case of tests/casos.py (the reference's own edge-case list at reduced sizes) runs at block 32 and 128 and
must equal, bit for bit, (a) the oracle on the same seeded inputs and (b) the committed golden outputs that the
reference's OpsRef produced.  GEMMs additionally run on each of the three kernel paths.
"""
import os
import tempfile

import pytest
import torch

import casos
import golden_util as gu
from oracle import spec

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def amb():
    from jatai_b200 import ops, registro
    reg = registro.Registro(tempfile.mkdtemp(), "teste", vigiar=True, eco=False, salvar=False)
    oc = ops.OpsCuda(reg)
    reg.novo_passo(0)
    yield ops, oc, reg
    ops.define_blk(32)
    oc.lib.jt_gemm_via(0)


def para_gpu(a):
    if torch.is_tensor(a):
        return a.to(DEV).contiguous()
    if isinstance(a, tuple):
        return tuple(para_gpu(x) for x in a)
    return a


class Adapt:
    """OpsCuda with the `limite` attribute casos.roda toggles (a module global in the operator module)."""

    def __init__(self, ops, oc):
        self._ops, self._oc = ops, oc

    def __getattr__(self, n):
        return getattr(self._oc, n)

    @property
    def limite(self):
        return self._ops.ATENCAO_LIMITE

    @limite.setter
    def limite(self, v):
        self._ops.ATENCAO_LIMITE = bool(v)


def _ids(blk):
    return [n for n, _, _ in casos.tabela(blk)]


def compara(nome, outs, refs):
    assert len(outs) == len(refs)
    for i, (a, b) in enumerate(zip(outs, refs)):
        a, b = a.cpu(), b.cpu()
        assert a.dtype == b.dtype and a.shape == b.shape, f"{nome} out {i}: {a.dtype}{tuple(a.shape)} vs {b.dtype}{tuple(b.shape)}"
        dif = a != b
        if dif.any():
            p = tuple(dif.nonzero()[0].tolist())
            raise AssertionError(f"{nome} out {i}: {int(dif.sum())} of {a.numel()} differ; first at {p}: cuda {a[p].item()} oracle {b[p].item()}")


@pytest.mark.parametrize("nome,blk,f", casos.tabela(32) + casos.tabela(128), ids=_ids(32) + _ids(128))
def test_tabela(amb, nome, blk, f):
    ops, oc, reg = amb
    ops.define_blk(blk)
    oc.lib.jt_gemm_via(0)
    reg.novo_passo(0)
    G = casos.Gen(casos.semente(nome), blk)
    op, args, kw = f(G)
    outs = casos.roda(Adapt(ops, oc), op, tuple(para_gpu(a) for a in args), kw)
    torch.cuda.synchronize()
    refs = casos.roda(spec.Spec(blk), op, args, kw)
    compara(nome, outs, refs)
    meta, arrs = gu.carrega(blk)
    gu.confere_saidas(nome, meta[nome], arrs, outs)


GEMMS = [(n, b, f) for n, b, f in casos.tabela(32) + casos.tabela(128) if "/gemm" in n]


@pytest.mark.parametrize("via", [1, 2, 3])
@pytest.mark.parametrize("nome,blk,f", GEMMS, ids=[n for n, _, _ in GEMMS])
def test_gemm_vias(amb, nome, blk, f, via):
    """via 1 = tensor core forced (block 32: FMA rounding with its range check, which the saturated-mantissa case sends to the
    conversion; block 128: conversion), 2 = CUDA cores, 3 = tensor core with the conversion everywhere."""
    ops, oc, reg = amb
    ops.define_blk(blk)
    assert oc.lib.jt_gemm_via(via) == 0
    try:
        reg.novo_passo(0)
        G = casos.Gen(casos.semente(nome), blk)
        op, args, kw = f(G)
        outs = casos.roda(oc, op, tuple(para_gpu(a) for a in args), kw)
        torch.cuda.synchronize()
        compara(f"{nome} via {via}", outs, casos.roda(spec.Spec(blk), op, args, kw))
    finally:
        oc.lib.jt_gemm_via(0)


def test_config1(amb):
    """Benchmark configuration 1: linear layer forward + both backward GEMMs at block 32, against the reference digests."""
    import json
    ops, oc, reg = amb
    ops.define_blk(32)
    reg.novo_passo(0)
    with open(os.path.join(gu.AQUI, "config1_b32.json")) as fh:
        rec = json.load(fh)
    X, W, dY = (para_gpu(t) for t in casos.config1(32))
    Y = oc.gemm(X, W)
    dX = oc.gemm(dY, oc.transpoe(W))
    dW = oc.gemm(oc.transpoe(dY), oc.transpoe(X), cru=True)
    torch.cuda.synchronize()
    assert [gu.digest(t) for t in Y] == rec["Y"]
    assert [gu.digest(t) for t in dX] == rec["dX"]
    assert [gu.digest(t) for t in dW] == rec["dW"]


@pytest.mark.parametrize("blk", [32, 128])
@pytest.mark.parametrize("M,N,K,cru", [(256, 256, 1024, False), (512, 384, 512, True), (128, 128, 4096, True), (1024, 1536, 512, False),
                                       (64, 128, 256, False), (192, 256, 384, True)])
def test_gemm_formas(amb, blk, M, N, K, cru):
    """Shape sweep against the oracle evaluated on the GPU in int64 (includes split-K raw outputs and the
    shapes only the CUDA-core path takes: M or K not a multiple of 128)."""
    ops, oc, reg = amb
    ops.define_blk(blk)
    reg.novo_passo(0)
    G = casos.Gen(1000 + M + N + K, blk)
    A, B = para_gpu(G.bloco(M, K, faixa=(-12, -4))), para_gpu(G.bloco(N, K, espalha=6, zera=0.05))
    out = oc.gemm(A, B, cru=cru)
    torch.cuda.synchronize()
    compara(f"gemm {M}x{N}x{K}", casos.plano(out), casos.plano(spec.Spec(blk).gemm(A, B, cru=cru)))


def _somas(blk, tn, K):
    """The values of jt_gemm_somas that mean different kernels for a half-precision product: one, or without sums and with them."""
    return (1, 2) if blk == 32 and tn == 128 and K <= 1024 else (0,)


@pytest.mark.parametrize("tn", [64, 128])
@pytest.mark.parametrize("blk,M,N,K", [(32, 64, 128, 32), (32, 128, 128, 96), (32, 192, 256, 2080), (32, 320, 384, 512), (32, 2432, 1408, 160), (32, 128, 128, 8192),
                                       (32, 320, 128, 544), (32, 192, 256, 1056),
                                       (128, 64, 128, 128), (128, 192, 384, 640), (128, 2432, 1408, 256)])
def test_gemm_meia_precisao(amb, blk, M, N, K, tn):
    """The half-precision tensor path, forced, in every mode against the oracle: rows that fill no tile, a K of half a chunk, more tiles
    than SMs, K ranges added with atomics or over clusters of 2, 4 and 8 blocks (one of them without chunks), exponents spread beyond what f16 holds, zero blocks; and saturated rows, whose norms
    exclude the fast rounding."""
    ops, oc, reg = amb
    ops.define_blk(blk)
    assert oc.lib.jt_gemm_via(4) == 0 and oc.lib.jt_gemm_tn(tn) == 0
    try:
        reg.novo_passo(0)
        G = casos.Gen(31 + M + N + K + blk, blk)
        A, B, X = para_gpu(G.bloco(M, K, espalha=15, zera=0.1)), para_gpu(G.bloco(N, K, espalha=5)), para_gpu(G.bloco(M, N, espalha=4))
        A[0][5::64, :2048] = 127                      # (more saturated K-blocks than this would overflow the accumulator)
        A[1][5::64] = -8
        B[0][7::32, :2048] = -127
        B[1][7::32] = -8
        s = spec.Spec(blk)
        for op, args, kw in (("gemm", (A, B), {}), ("gemm", (A, B), dict(cru=True)), ("gemm_soma", (A, B, X), {}), ("gemm_relu2", (A, B), {}), ("gemm_relu2_back", (A, B, X), {})):
            quer = casos.roda(s, op, args, kw)
            for somas in _somas(blk, tn, K):
                assert oc.lib.jt_gemm_somas(somas) == 0
                outs = casos.roda(oc, op, args, kw)
                torch.cuda.synchronize()
                compara(f"{op} {kw} {M}x{N}x{K} blk {blk} tn {tn} somas {somas}", outs, quer)
    finally:
        oc.lib.jt_gemm_via(0)
        oc.lib.jt_gemm_tn(0)
        oc.lib.jt_gemm_somas(0)
        ops.define_blk(32)


@pytest.mark.parametrize("M,N,K", [(2432, 1024, 1056), (2368, 1024, 96), (1088, 1024, 4160), (960, 128, 2048), (1024, 128, 2080)])
def test_gemm_meia_precisao_64_ondas_e_grupos(amb, M, N, K):
    """The same with 64-wide tiles: two or three per block, with whole chunks and half ones; more than 32 K-blocks; 15 and 16 tiles, on either side of what
    goes to clusters of 8."""
    test_gemm_meia_precisao(amb, 32, M, N, K, 64)


def test_gemm_maximos_externos(amb):
    """Row maxima supplied by the caller (the data-parallel path): two K halves with the global maxima add up to
    the full GEMM, bit for bit."""
    ops, oc, reg = amb
    ops.define_blk(32)
    reg.novo_passo(0)
    G = casos.Gen(77, 32)
    A, B = para_gpu(G.bloco(256, 1024, espalha=8)), para_gpu(G.bloco(128, 1024, espalha=8))
    RA, RB = oc.max_linha(A), oc.max_linha(B)
    assert torch.equal(RA.cpu(), A[1].cpu().amax(1)) and torch.equal(RB.cpu(), B[1].cpu().amax(1))
    inteiro = oc.gemm(A, B, cru=True)
    soma = None
    for h in range(2):
        a = (A[0][:, h * 512:(h + 1) * 512].contiguous(), A[1][:, h * 16:(h + 1) * 16].contiguous())
        b = (B[0][:, h * 512:(h + 1) * 512].contiguous(), B[1][:, h * 16:(h + 1) * 16].contiguous())
        acc, e = oc.gemm(a, b, cru=True, RA=RA, RB=RB)
        assert torch.equal(e, inteiro[1])
        soma = acc if soma is None else soma + acc
    assert torch.equal(soma, inteiro[0])


def test_sentinela_token_invalido(amb):
    """An out-of-range token is recorded (code 6) and reported with operation and position; nothing traps."""
    from jatai_b200.registro import ErroJatai
    ops, oc, reg = amb
    ops.define_blk(32)
    reg.novo_passo(0)
    G = casos.Gen(5, 32)
    W = para_gpu(G.bloco(256, 128))
    tok = G.tok(64, 256)
    tok[17] = 300
    reg.vigiar = False
    try:
        X = oc.embed(W, tok.to(DEV))
        with pytest.raises(ErroJatai) as ei:
            reg.confere_device()
        assert "embed" in str(ei.value) and "linha 17" in str(ei.value) and "300" in str(ei.value)
        assert int(X[0][17].abs().sum()) == 0 and int(X[1][17, 0]) == -127
    finally:
        reg.vigiar = True
        reg.novo_passo(0)


def test_referencia_compat(amb):
    """Compatibility format (block 128): the reference's own CUDA library, compiled for sm_100a from its source,
    is driven through the same operator class and must agree with this library bit for bit."""
    caminho = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle", "_ref", "libjatai_ref.so")
    if not os.path.exists(caminho):
        pytest.skip("oracle/_ref/libjatai_ref.so not built (needs the reference checkout at build time)")
    from jatai_b200 import registro
    ops, oc, reg = amb
    ops.define_blk(128)
    reg.novo_passo(0)
    reg2 = registro.Registro(tempfile.mkdtemp(), "ref", vigiar=True, eco=False, salvar=False)
    ocr = ops.OpsCuda(reg2, biblioteca=caminho)
    ops.OpsCuda.lib_global = oc.lib
    reg2.novo_passo(0)
    G = casos.Gen(9, 128)
    M, D, FF = 256, 256, 1024
    x, w1, w2, r = para_gpu(G.bloco(M, D)), para_gpu(G.bloco(FF, D)), para_gpu(G.bloco(D, FF)), para_gpu(G.bloco(M, D, espalha=8))
    for nome, f in [("gemm", lambda o: o.gemm(x, w1)), ("gemm_cru", lambda o: o.gemm(x, w1, cru=True)),
                    ("gemm_relu2", lambda o: o.gemm_relu2(x, w1)), ("gemm_soma", lambda o: o.gemm_soma(o.gemm_relu2(x, w1)[1], w2, r)),
                    ("transpoe", lambda o: o.transpoe(w1)), ("rms", lambda o: o.rms(x)), ("soma", lambda o: o.soma(x, r))]:
        a, b = casos.plano(f(oc)), casos.plano(f(ocr))
        torch.cuda.synchronize()
        compara(f"ref/{nome}", a, b)


ATENCOES = [  # blk, Bt, T, H, D  (head dim D/H in {4, 16, 64}; T also off the 128 grid; block 128 with wide heads)
    (32, 2, 64, 4, 64), (32, 2, 128, 2, 128), (32, 1, 256, 8, 512), (32, 1, 160, 2, 128), (32, 2, 96, 16, 64),
    (128, 2, 64, 2, 128), (128, 1, 192, 8, 128), (32, 1, 512, 2, 128), (32, 1, 192, 2, 128), (128, 1, 320, 2, 128), (32, 3, 128, 1, 64),
]


@pytest.mark.parametrize("limite", [False, True])
@pytest.mark.parametrize("blk,Bt,T,H,D", ATENCOES)
def test_atencao_generalizada(amb, blk, Bt, T, H, D, limite):
    """Attention forward + backward at head dimensions and sequence lengths the reference kernels do not reach,
    against the generalised oracle (which reduces to the reference at head dimension 4)."""
    ops, oc, reg = amb
    ops.define_blk(blk)
    reg.novo_passo(0)
    G = casos.Gen(31 * T + H + D + blk, blk)
    M = Bt * T
    qkv, go = G.bloco(M, 3 * D, espalha=5, zera=0.05), G.bloco(M, D, e0=-20, espalha=6, zera=0.05)
    s = spec.Spec(blk, limite=limite)
    (o_r, P_r) = s.atencao(qkv, Bt, T, H)
    g_r = s.atencao_back(go, qkv, P_r, Bt, T, H)
    ops.ATENCAO_LIMITE = limite
    try:
        o_c, P_c = oc.atencao(para_gpu(qkv), Bt, T, H)
        g_c = oc.atencao_back(para_gpu(go), para_gpu(qkv), P_c, Bt, T, H)
        torch.cuda.synchronize()
    finally:
        ops.ATENCAO_LIMITE = False
    compara(f"atencao {blk}/{Bt}/{T}/{H}/{D}", [*o_c, P_c], [*o_r, P_r])
    compara(f"atencao_back {blk}/{Bt}/{T}/{H}/{D} limite={limite}", list(g_c), list(g_r))


@pytest.mark.parametrize("R,C,esp,zera", [(256, 512, 4, 0.0), (128, 1024, 12, 0.1), (384, 256, 60, 0.3), (128, 256, 0, 0.0), (256, 768, 25, 0.5)])
def test_transpoe_largo(amb, R, C, esp, zera):
    """The wide-tile block-32 transposition (fp32 exact quantiser) against the oracle, including exponent spreads
    beyond what fp32 can align (integer path) and mostly-zero tensors."""
    ops, oc, reg = amb
    ops.define_blk(32)
    reg.novo_passo(0)
    G = casos.Gen(4000 + R + C + esp, 32)
    X = G.bloco(R, C, espalha=esp, zera=zera, e0=-5)
    out = oc.transpoe(para_gpu(X))
    torch.cuda.synchronize()
    compara(f"transpoe {R}x{C} esp {esp}", list(out), list(spec.Spec(32).transpoe(X)))


GEMMS32 = [(n, b, f) for n, b, f in casos.tabela(32) if "/gemm" in n]


@pytest.mark.parametrize("tn", [64, 128])
@pytest.mark.parametrize("nome,blk,f", GEMMS32, ids=[n for n, _, _ in GEMMS32])
def test_gemm_largura_do_tile(amb, nome, blk, f, tn):
    """Both tile widths of the tensor-core GEMM (64 and 128 columns), forced, on every GEMM case of the table."""
    ops, oc, reg = amb
    ops.define_blk(32)
    oc.lib.jt_gemm_via(0)
    assert oc.lib.jt_gemm_tn(tn) == 0
    try:
        reg.novo_passo(0)
        G = casos.Gen(casos.semente(nome), blk)
        op, args, kw = f(G)
        outs = casos.roda(oc, op, tuple(para_gpu(a) for a in args), kw)
        torch.cuda.synchronize()
        compara(f"{nome} tn {tn}", outs, casos.roda(spec.Spec(blk), op, args, kw))
    finally:
        oc.lib.jt_gemm_tn(0)


@pytest.mark.parametrize("tn", [64, 128])
@pytest.mark.parametrize("caso", ["expoentes afastados", "linhas nulas", "acumuladores grandes"])
@pytest.mark.parametrize("op", ["gemm", "gemm_soma", "gemm_relu2", "gemm_relu2_back"])
@pytest.mark.parametrize("blk,via", [(32, 0), (32, 4), (128, 0), (128, 4)])
def test_gemm_estagio_de_saida(amb, op, caso, tn, blk, via):
    """The output stage of the tensor-core GEMM quantises in fp32 when that is exact and in integers otherwise.  These
    inputs force the integer side: column exponents of one block more than 64 apart, all-zero rows of B (row maximum
    -127 next to ordinary rows), accumulators at or above 2^24 - each against the specification, on the 8-bit kernel (which
    these sizes take by themselves) and on the half-precision one, which has its own tables for that decision."""
    ops, oc, reg = amb
    if blk == 128 and tn == 64:
        pytest.skip("64-column tiles exist for block 32 only")
    ops.define_blk(blk)
    assert oc.lib.jt_gemm_via(via) == 0 and oc.lib.jt_gemm_tn(tn) == 0
    try:
        reg.novo_passo(0)
        G = casos.Gen(4242, blk)
        M, K, N = 256, 512, 256
        A, B = G.bloco(M, K, espalha=2), G.bloco(N, K, espalha=2)
        if caso == "expoentes afastados":
            B[1][0::2] -= 50                      # even rows of B 70 exponents below the odd ones, inside every block of columns
            B[1][1::2] += 20                      # (output exponents stay far from the int8 limits, squared too)
        elif caso == "linhas nulas":
            B[0][::3] = 0
            B[1][::3] = -127
        else:
            A = (torch.full_like(A[0], 127), torch.full_like(A[1], -8))
            B = (torch.full_like(B[0], 127), torch.full_like(B[1], -8))
        X = G.bloco(M, N, espalha=3)
        args = {"gemm": (A, B), "gemm_soma": (A, B, X), "gemm_relu2": (A, B), "gemm_relu2_back": (A, B, X)}[op]
        quer = casos.roda(spec.Spec(blk), op, args, {})
        for somas in _somas(blk, tn, K) if via == 4 else (0,):
            assert oc.lib.jt_gemm_somas(somas) == 0
            outs = casos.roda(oc, op, tuple(para_gpu(a) for a in args), {})
            torch.cuda.synchronize()
            compara(f"{op} {caso} tn {tn} blk {blk} via {via} somas {somas}", outs, quer)
    finally:
        oc.lib.jt_gemm_tn(0)
        oc.lib.jt_gemm_via(0)
        oc.lib.jt_gemm_somas(0)
        ops.define_blk(32)


@pytest.mark.parametrize("blk", [32, 128])
@pytest.mark.parametrize("ef", [0, 1])
def test_momento_peso_junto(amb, blk, ef):
    """The fused optimiser launch gives the bits of momento followed by peso (and of the specification), including
    zero blocks of momentum and residual and gradients of very different magnitudes."""
    ops, oc, reg = amb
    ops.define_blk(blk)
    try:
        reg.novo_passo(0)
        G = casos.Gen(77 + blk + ef, blk)
        R_, C_ = 256, 512
        grad = G.cru(R_, C_, bits=26, e0=-35)
        grad[0][::7] = 0
        mom, w, res = G.bloco(R_, C_, espalha=6, zera=0.1, e0=-14), G.bloco(R_, C_, espalha=3, e0=-9), G.bloco(R_, C_, espalha=5, zera=0.2, e0=-17)
        copia = lambda t: tuple(x.clone().cuda() for x in t)
        g_d = para_gpu(grad)
        m1, w1, r1 = copia(mom), copia(w), copia(res)
        m1 = oc.momento(g_d, m1)
        w1, r1 = oc.peso(w1, m1, r1, 4, ef)
        m2, w2, r2 = oc.momento_peso(g_d, copia(mom), copia(w), copia(res), 4, ef)
        torch.cuda.synchronize()
        ref = spec.Spec(blk).momento_peso(grad, mom, w, res, 4, ef)
        compara(f"momento_peso blk {blk} ef {ef} (vs separate launches)", casos.plano((m2, w2, r2)), casos.plano((m1, w1, r1)))
        compara(f"momento_peso blk {blk} ef {ef} (vs specification)", casos.plano((m2, w2, r2)), casos.plano(ref))
    finally:
        ops.define_blk(32)


@pytest.mark.parametrize("blk,R,C1,C2", [(32, 256, 256, 512), (32, 2048, 512, 1536), (32, 2048, 256, 512), (32, 4096, 2048, 512),
                                         (32, 8192, 2048, 2048), (32, 256, 192, 512), (128, 256, 256, 512)])
def test_transpoe_par(amb, blk, R, C1, C2):
    """The paired transposition launch gives the bits of two single launches and of the specification, for every tile
    height it picks, unequal widths, a width that falls back to the generic kernel, and block 128."""
    ops, oc, reg = amb
    ops.define_blk(blk)
    try:
        reg.novo_passo(0)
        G = casos.Gen(500 + R + C1 + C2, blk)
        X1, X2 = G.bloco(R, C1, espalha=8, zera=0.1), G.bloco(R, C2, espalha=3, zera=0.05)
        d1, d2 = para_gpu(X1), para_gpu(X2)
        juntos = oc.transpoe2(d1, d2)
        separados = (oc.transpoe(d1), oc.transpoe(d2))
        torch.cuda.synchronize()
        compara(f"transpoe2 {R}x({C1},{C2}) blk {blk} (vs single launches)", casos.plano(juntos), casos.plano(separados))
        compara(f"transpoe2 {R}x({C1},{C2}) blk {blk} (vs specification)", casos.plano(juntos), casos.plano(spec.Spec(blk).transpoe2(X1, X2)))
    finally:
        ops.define_blk(32)


@pytest.mark.parametrize("blk,M,D", [(32, 256, 512), (32, 128, 1024), (32, 64, 2048), (32, 40, 256), (128, 256, 512)])
def test_rms_back_soma_junto(amb, blk, M, D):
    """The fused RMSNorm-backward + residual-add launch gives the bits of the two launches and of the specification
    (rows that do not fill the last CTA, every row width the kernel is instantiated for, zero blocks in the residual)."""
    ops, oc, reg = amb
    ops.define_blk(blk)
    try:
        reg.novo_passo(0)
        G = casos.Gen(900 + M + D, blk)
        x = G.bloco(M, D, espalha=5, zera=0.1, e0=-12)
        y, cache = spec.Spec(blk).rms(x)
        g, res = G.bloco(M, D, espalha=4, e0=-20), G.bloco(M, D, espalha=6, zera=0.15, e0=-19)
        dg, dy, dc, dr = para_gpu(g), para_gpu(y), tuple(t.cuda() for t in cache), para_gpu(res)
        junto = oc.rms_back_soma(dr, dg, dy, dc)
        separado = oc.soma(dr, oc.rms_back(dg, dy, dc))
        torch.cuda.synchronize()
        compara(f"rms_back_soma {M}x{D} blk {blk} (vs two launches)", casos.plano(junto), casos.plano(separado))
        compara(f"rms_back_soma {M}x{D} blk {blk} (vs specification)", casos.plano(junto), casos.plano(spec.Spec(blk).rms_back_soma(res, g, y, cache)))
    finally:
        ops.define_blk(32)


@pytest.mark.parametrize("tn", [64, 128])
@pytest.mark.parametrize("caso", ["tudo +127", "sinais alternados", "uma linha saturada", "um bloco saturado por linha"])
@pytest.mark.parametrize("via", [0, 4])
def test_gemm_produtos_parciais_grandes(amb, caso, tn, via):
    """Partial products at and above 2^18 with no alignment shift (s = 0): the inputs on which rounding by an FMA against
    1.5*2^23 would leave its exact range.  The kernels must find them (the 8-bit one, which these sizes take by themselves, by a range check
    on the biased patterns, the half-precision one by the norms of the K-blocks) and round those by conversion - in whole
    tiles, in single rows and in single K-blocks, for positive and negative products.  (Without shifts nothing is rounded, so the half-precision
    kernel runs without sums in tensor memory, where it converts, and with them, where it adds up 2 to 16 chunks.)"""
    ops, oc, reg = amb
    ops.define_blk(32)
    assert oc.lib.jt_gemm_via(via) == 0 and oc.lib.jt_gemm_tn(tn) == 0
    try:
        reg.novo_passo(0)
        G = casos.Gen(8181, 32)
        M, K, N = 256, 512, 256
        A, B = G.bloco(M, K, espalha=0), G.bloco(N, K, espalha=0)
        if caso == "tudo +127":
            A, B = (torch.full_like(A[0], 127), A[1]), (torch.full_like(B[0], 127), B[1])
        elif caso == "sinais alternados":            # every K-block of a row entirely +127 or -127: products of both signs at 32 * 127^2
            sa = (torch.arange(K // 32) % 2 * 2 - 1).repeat_interleave(32).to(torch.int8)
            A = ((127 * sa).expand(M, K).contiguous(), A[1])
            B = (torch.where(torch.arange(N)[:, None] % 3 == 0, -127, 127).to(torch.int8).expand(N, K).contiguous(), B[1])
        elif caso == "uma linha saturada":
            A[0][37] = 127
            B[0][101] = -127
        else:                                         # one saturated K-block per row, at a different place in every row
            for i in range(M):
                b = i % (K // 32)
                A[0][i, 32 * b:32 * b + 32] = 127 if i % 2 else -127
            B = (torch.full_like(B[0], 127), B[1])
        for cru in (False, True):
            quer = casos.plano(spec.Spec(32).gemm(A, B, cru=cru))
            for somas in _somas(32, tn, K) if via == 4 and not cru else (0,):
                assert oc.lib.jt_gemm_somas(somas) == 0
                outs = casos.plano(oc.gemm(para_gpu(A), para_gpu(B), cru=cru))
                torch.cuda.synchronize()
                compara(f"gemm {caso} tn {tn} via {via} cru {cru} somas {somas}", outs, quer)
    finally:
        oc.lib.jt_gemm_tn(0)
        oc.lib.jt_gemm_via(0)
        oc.lib.jt_gemm_somas(0)


@pytest.mark.parametrize("caso", ["um expoente", "dois", "saturado", "saturado a 4", "sem blocos", "um bloco fora"])
@pytest.mark.parametrize("op", ["gemm", "gemm_soma", "gemm_relu2", "gemm_relu2_back"])
@pytest.mark.parametrize("M,N,K", [(64, 128, 32), (192, 256, 160), (128, 128, 992), (128, 128, 1024)])
def test_gemm_somas_em_memoria_de_tensor(amb, caso, M, N, K, op):
    """Tiles whose K-blocks need no rounding (exponents within 4 of their rows' maxima, both sides together) add up in tensor memory: one
    sum, several where the bound on the sums (2^24 last places) splits them, and none where one K-block of one row lies further down.  In
    every output stage that has sums, with rows that fill no tile."""
    ops, oc, reg = amb
    ops.define_blk(32)
    assert oc.lib.jt_gemm_via(4) == 0 and oc.lib.jt_gemm_tn(128) == 0 and oc.lib.jt_gemm_somas(2) == 0
    try:
        reg.novo_passo(0)
        G = casos.Gen(77, 32)
        A, B = G.bloco(M, K, espalha=0), G.bloco(N, K, espalha=0)
        nb = K // 32
        if caso == "dois":                            # shifts 0 to 2 on either side
            A, B = (A[0], -8 - torch.randint(0, 3, (M, nb), generator=G.g).to(torch.int8)), (B[0], -8 - torch.randint(0, 3, (N, nb), generator=G.g).to(torch.int8))
        elif caso.startswith("saturado"):             # the largest sums there are; "a 4": in units of 1, all but the first K-block
            A, B = (torch.full_like(A[0], 127), A[1].clone()), (torch.full_like(B[0], -127), B[1].clone())
            if caso == "saturado a 4":
                A[1][:, 1:] -= 4
        elif caso == "sem blocos":                    # all-zero K-blocks, exponents far down: they round nothing
            A[0][:, 32:64] = 0
            A[1][:, 1:2] = -127
        elif caso == "um bloco fora":
            A[1][M // 2, nb - 1] -= 5
            A[0][M // 2] |= 1
        args = (A, B, G.bloco(M, N, espalha=3)) if op in ("gemm_soma", "gemm_relu2_back") else (A, B)
        outs = casos.roda(oc, op, tuple(para_gpu(a) for a in args), {})
        torch.cuda.synchronize()
        compara(f"{op} {caso} {M}x{N}x{K}", outs, casos.roda(spec.Spec(32), op, args, {}))
    finally:
        oc.lib.jt_gemm_tn(0)
        oc.lib.jt_gemm_via(0)
        oc.lib.jt_gemm_somas(0)


@pytest.mark.parametrize("K", [64, 96, 512, 1024])
def test_gemm_somas_e_arredondamentos_alternados(amb, K):
    """160 tiles, a few more than SMs: most blocks have one, twelve have two, each of which adds up or rounds.  Raw outputs, which have no sums, beside
    the block outputs."""
    ops, oc, reg = amb
    ops.define_blk(32)
    g = torch.Generator(device=DEV).manual_seed(K)
    M, N = 2560, 1024                                 # 160 tiles
    def bloco(R, quem):
        m = torch.randint(-127, 128, (R, K), generator=g, device=DEV, dtype=torch.int32).to(torch.int8)
        e = torch.randint(-8, -6, (R, K // 32), generator=g, device=DEV, dtype=torch.int32)
        e -= 6 * (torch.randint(0, 2, (R // 128,), generator=g, device=DEV).repeat_interleave(128)[:, None] * torch.randint(0, 2, e.shape, generator=g, device=DEV)) * quem
        return m, e.to(torch.int8)
    A, B = bloco(M, 1), bloco(N, 0)
    reg.novo_passo(0)
    try:
        for cru in (False, True):
            assert oc.lib.jt_gemm_via(2) == 0
            quer = oc.gemm(A, B, cru=cru)
            assert oc.lib.jt_gemm_via(4) == 0 and oc.lib.jt_gemm_tn(128) == 0 and oc.lib.jt_gemm_somas(2) == 0
            tem = oc.gemm(A, B, cru=cru)
            assert all(torch.equal(x, y) for x, y in zip(quer, tem))
    finally:
        oc.lib.jt_gemm_tn(0)
        oc.lib.jt_gemm_via(0)
        oc.lib.jt_gemm_somas(0)


@pytest.mark.parametrize("op", ["gemm", "gemm_soma", "gemm_relu2", "gemm_relu2_back"])
@pytest.mark.parametrize("K,arredonda", [(64, 0.5), (96, 0.3), (320, 0.5), (512, 0.8), (1024, 0.1), (1024, 0.5)])
def test_gemm_somas_e_arredondamentos_treze_tiles_por_bloco(amb, K, arredonda, op):
    """2032 tiles, 13 or 14 to a block, in random order: tiles that round (a share of the bands of 128 rows), that add up in one sum, and in sums of 8, 4
    and 2 chunks (blocks at the ends of the mantissas' range, up to 1, 2 or 3 places below their rows' maxima).  Every output stage that
    the summing kernel has, the last band of rows half full, against the CUDA-core kernel."""
    ops, oc, reg = amb
    ops.define_blk(32)
    g = torch.Generator(device=DEV).manual_seed(1000 * K + int(10 * arredonda))
    M, N = 127 * 128 - 64, 2048
    ints = lambda a, b, forma: torch.randint(a, b + 1, forma, generator=g, device=DEV, dtype=torch.int32)
    faixa = torch.arange(M, device=DEV) // 128
    arr = (torch.rand(127, generator=g, device=DEV) < arredonda)[faixa]
    desce = ints(0, 3, (127,))[faixa]                              # 0: one sum; 1 to 3: several
    m = torch.where((desce > 0)[:, None], 254 * ints(0, 1, (M, K)) - 127, ints(-127, 127, (M, K)))
    e = -8 - torch.remainder(ints(0, 1 << 20, (M, K // 32)), (desce + 1)[:, None])
    e -= 9 * (arr[:, None] & (ints(0, 2, e.shape) == 0)).to(torch.int32)
    A = (m.to(torch.int8), e.to(torch.int8))
    B = ((254 * ints(0, 1, (N, K)) - 127).to(torch.int8), torch.full((N, K // 32), -8, device=DEV, dtype=torch.int8))
    X = (ints(-127, 127, (M, N)).to(torch.int8), ints(-12, -4, (M, N // 32)).to(torch.int8))
    args = {"gemm": (A, B), "gemm_soma": (A, B, X), "gemm_relu2": (A, B), "gemm_relu2_back": (A, B, X)}[op]
    reg.novo_passo(0)
    try:
        assert oc.lib.jt_gemm_via(2) == 0
        quer = casos.roda(oc, op, args, {})
        assert oc.lib.jt_gemm_via(4) == 0 and oc.lib.jt_gemm_tn(128) == 0 and oc.lib.jt_gemm_somas(2) == 0
        for _ in range(3):
            tem = casos.roda(oc, op, args, {})
            assert len(quer) == len(tem) and all(torch.equal(x, y) for x, y in zip(quer, tem))
    finally:
        oc.lib.jt_gemm_tn(0)
        oc.lib.jt_gemm_via(0)
        oc.lib.jt_gemm_somas(0)


@pytest.mark.parametrize("op", ["gemm", "gemm_relu2"])
@pytest.mark.parametrize("afasta", [1, 9])
@pytest.mark.parametrize("M,K", [(37 * 128, 1024), (36 * 128, 1024), (37 * 128, 1056), (37 * 128 - 64, 32), (37 * 128, 64)])
def test_gemm_somas_regra(amb, M, K, afasta, op):
    """Both sides of the lines of the automatic choice (592 tiles against 576, K = 1024 against 1056, the smallest K), with exponents that round
    nothing and with exponents that round everywhere, against the CUDA-core kernel."""
    ops, oc, reg = amb
    ops.define_blk(32)
    g = torch.Generator(device=DEV).manual_seed(M + K + afasta)
    ints = lambda a, b, forma: torch.randint(a, b + 1, forma, generator=g, device=DEV, dtype=torch.int32).to(torch.int8)
    A, B = ((ints(-127, 127, (R, K)), ints(-8, -9 + afasta, (R, K // 32))) for R in (M, 2048))
    reg.novo_passo(0)
    try:
        assert oc.lib.jt_gemm_via(2) == 0
        quer = casos.roda(oc, op, (A, B), {})
        for via in (0, 4):
            assert oc.lib.jt_gemm_via(via) == 0
            tem = casos.roda(oc, op, (A, B), {})
            assert len(quer) == len(tem) and all(torch.equal(x, y) for x, y in zip(quer, tem))
    finally:
        oc.lib.jt_gemm_via(0)


@pytest.mark.parametrize("limite", [False, True])
@pytest.mark.parametrize("blk,Bt,T,H,D", [(32, 2, 128, 2, 128), (32, 1, 192, 2, 128), (32, 1, 160, 2, 128), (32, 2, 256, 8, 512), (128, 2, 128, 2, 128),
                                         (32, 1, 704, 1, 64), (32, 1, 320, 3, 192)])
def test_atencao_nucleos_tensor_e_cuda(amb, blk, Bt, T, H, D, limite):
    """Head dimension 64 has two implementations - tensor cores (the default) and the CUDA-core kernels (jt_atencao_via(1),
    also what the no-allocation entry point runs, and what sequence lengths that are no multiple of 64 get): forward and backward
    must agree bit for bit, on sequence lengths that fill whole key chunks and on ones that do not."""
    ops, oc, reg = amb
    ops.define_blk(blk)
    reg.novo_passo(0)
    G = casos.Gen(7 * T + H + D + blk, blk)
    M = Bt * T
    qkv, go = para_gpu(G.bloco(M, 3 * D, espalha=6, zera=0.05)), para_gpu(G.bloco(M, D, e0=-20, espalha=6, zera=0.05))
    ops.ATENCAO_LIMITE = limite
    saidas = []
    try:
        for via in (0, 1):
            assert oc.lib.jt_atencao_via(via) == 0
            o, P = oc.atencao(qkv, Bt, T, H)
            g = oc.atencao_back(go, qkv, P, Bt, T, H)
            torch.cuda.synchronize()
            saidas.append([*o, P, *g])
    finally:
        ops.ATENCAO_LIMITE = False
        oc.lib.jt_atencao_via(0)
        ops.define_blk(32)
    compara(f"atencao tensor x cuda {blk}/{Bt}/{T}/{H}/{D} limite={limite}", saidas[0], saidas[1])


@pytest.mark.parametrize("limite", [False, True])
@pytest.mark.parametrize("Bt,T,H,D", [(2, 128, 2, 128), (1, 256, 8, 512), (1, 192, 2, 128), (1, 1024, 1, 64)])
def test_atencao_com_quant_fundido(amb, Bt, T, H, D, limite):
    """The attention kernels that write their outputs already quantised (block length 32, head dimension 64) against
    quant(atencao(...)) / quant(atencao_back(...)) of the specification, including rows whose block of 32 columns is entirely
    zero and key tiles that end beyond T."""
    ops, oc, reg = amb
    ops.define_blk(32)
    reg.novo_passo(0)
    G = casos.Gen(11 * T + H + D, 32)
    M = Bt * T
    qkv, go = G.bloco(M, 3 * D, espalha=5, zera=0.1), G.bloco(M, D, e0=-20, espalha=6, zera=0.1)
    s = spec.Spec(32, limite=limite)
    o_r, P_r = s.atencao_quant(qkv, Bt, T, H)
    g_r = s.atencao_back_quant(go, qkv, P_r, Bt, T, H)
    ops.ATENCAO_LIMITE = limite
    try:
        o_c, P_c = oc.atencao_quant(para_gpu(qkv), Bt, T, H)
        g_c = oc.atencao_back_quant(para_gpu(go), para_gpu(qkv), P_c, Bt, T, H)
        torch.cuda.synchronize()
    finally:
        ops.ATENCAO_LIMITE = False
    assert reg.lancamentos[-1]["op"] == "atencao_back_quant"          # the fused entry point ran, not the composition
    compara(f"atencao_quant {Bt}/{T}/{H}/{D}", [*o_c, P_c], [*o_r, P_r])
    compara(f"atencao_back_quant {Bt}/{T}/{H}/{D} limite={limite}", list(g_c), list(g_r))


@pytest.mark.gpu
def test_espera_limitada_desiste_e_o_contexto_segue(amb):
    """The bounded wait of the tensor-core kernels on its own: one warp waits on a barrier that nothing completes, gives up
    after the (shortened) limit, records code 7 at place 99 and returns; the next GEMM is bit-exact as ever.  No copy,
    MMA or second CTA is involved, and the wait is the library's own `espera`."""
    import ctypes
    import json
    import time
    ops, oc, reg = amb
    lib = oc.lib
    ops.define_blk(32)
    torch.cuda.synchronize()
    assert lib.jt_erro_limpa() == 0
    saiu = torch.zeros(1, dtype=torch.int32, device=DEV)
    assert lib.jt_espera_limite(ctypes.c_longlong(2_000_000)) == 0          # about a millisecond
    try:
        t0 = time.time()
        assert lib.jt_teste_espera(ctypes.c_void_p(saiu.data_ptr()), ctypes.c_int(5)) == 0
        torch.cuda.synchronize()
        dt = time.time() - t0
        out = (ctypes.c_longlong * 6)()
        n = lib.jt_erro_le(out)
        assert saiu.item() == 2, "the wait must give up"
        assert n >= 1 and out[1] == 7 and out[2] == 5 and out[3] == 99, list(out)
        assert dt < 2.0, f"gave up after {dt:.2f} s with a limit of about 1 ms"
    finally:
        assert lib.jt_espera_limite(ctypes.c_longlong(0)) == 0
        assert lib.jt_erro_limpa() == 0
    reg.novo_passo(0)
    with open(os.path.join(gu.AQUI, "config1_b32.json")) as fh:
        rec = json.load(fh)
    X, W, _ = (para_gpu(t) for t in casos.config1(32))
    Y = oc.gemm(X, W)
    torch.cuda.synchronize()
    assert [gu.digest(t) for t in Y] == rec["Y"]


@pytest.mark.gpu
@pytest.mark.parametrize("R,C1,C2,esp", [(256, 256, 512, 8), (2048, 512, 1536, 3), (128, 256, 256, 40), (4096, 2048, 512, 60), (8192, 2048, 2048, 5)])
def test_transpoe_par_com_maximos(amb, R, C1, C2, esp):
    """jt_transpoe2_max = jt_transpoe2 followed by jt_max_linha of both results, bit for bit, with the maxima written (as a
    maximum into a buffer pre-set to -128) by the transposition kernel itself: every tile height, exponents far apart (the
    integer path of the kernel), all-zero blocks."""
    ops, oc, reg = amb
    ops.define_blk(32)
    reg.novo_passo(0)
    G = casos.Gen(900 + R + C1 + C2, 32)
    d1, d2 = para_gpu(G.bloco(R, C1, espalha=esp, zera=0.1)), para_gpu(G.bloco(R, C2, espalha=3, zera=0.3))
    separados = oc.transpoe2(d1, d2)
    r1, r2 = oc.max_linha(separados[0]), oc.max_linha(separados[1])
    buf = torch.full((C1 + C2 + 256,), -128, dtype=torch.int8, device=DEV)
    juntos = oc.transpoe2_max(d1, d2, buf[256:256 + C1], buf[256 + C1:])
    torch.cuda.synchronize()
    assert juntos is not None
    compara(f"transpoe2_max {R}x({C1},{C2})", casos.plano(juntos), casos.plano(separados))
    assert torch.equal(buf[256:256 + C1], r1) and torch.equal(buf[256 + C1:], r2)
    assert bool((buf[:256] == -128).all())
    assert oc.transpoe2_max(para_gpu(G.bloco(128, 192, espalha=2, zera=0.0)), para_gpu(G.bloco(128, 256, espalha=2, zera=0.0)), buf[:192], buf[256:512]) is None


@pytest.mark.gpu
def test_gemm_abandona_uma_espera_e_o_seguinte_e_exato(amb):
    """The abort path of the tensor-core GEMM itself: with its operand loads switched off (nothing asynchronous in flight) and
    the wait limit shortened, the MMA warp's first wait runs out, the CTAs record code 7 with the launch id of that GEMM,
    every warp leaves through the normal exit and the launch returns; the next GEMM is bit-exact."""
    import ctypes
    import json
    import time
    ops, oc, reg = amb
    lib = oc.lib
    ops.define_blk(32)
    X, W, _ = (para_gpu(t) for t in casos.config1(32))
    torch.cuda.synchronize()
    assert lib.jt_erro_limpa() == 0
    vigiar, reg.vigiar = reg.vigiar, False                       # the registry would raise on the record this test provokes
    assert lib.jt_espera_limite(ctypes.c_longlong(2_000_000)) == 0 and lib.jt_gemm_sem_cargas(1) == 0
    try:
        reg.novo_passo(0)
        t0 = time.time()
        oc.gemm(X, W)
        kid = len(reg.lancamentos) - 1
        torch.cuda.synchronize()
        dt = time.time() - t0
        out = (ctypes.c_longlong * 6)()
        n = lib.jt_erro_le(out)
        assert n >= 1 and out[1] == 7 and out[2] == kid, list(out)
        assert dt < 5.0, f"the aborted GEMM took {dt:.2f} s with a limit of about 1 ms"
    finally:
        assert lib.jt_gemm_sem_cargas(0) == 0 and lib.jt_espera_limite(ctypes.c_longlong(0)) == 0
        assert lib.jt_erro_limpa() == 0
        reg.vigiar = vigiar
    reg.novo_passo(0)
    with open(os.path.join(gu.AQUI, "config1_b32.json")) as fh:
        rec = json.load(fh)
    Y = oc.gemm(X, W)
    torch.cuda.synchronize()
    assert [gu.digest(t) for t in Y] == rec["Y"]


@pytest.mark.gpu
@pytest.mark.parametrize("mmax,esp,T", [(127, 5, 1024), (9, 2, 1024), (2, 0, 768), (40, 12, 512)])
def test_atencao_pedacos_de_chaves_sem_efeito(amb, mmax, esp, T):
    """The forward leaves out key chunks its norm bound proves to have P = 0 exactly: large and tiny q, k magnitudes (the bound
    decides how many chunks stay), several sequence lengths, against the oracle bit for bit (P included), and the backward on
    that P."""
    ops, oc, reg = amb
    ops.define_blk(32)
    reg.novo_passo(0)
    Bt, H, D = 1, 2, 128
    G = casos.Gen(77 + mmax + T, 32)
    qkv, go = G.bloco(Bt * T, 3 * D, espalha=esp, zera=0.02, mmax=mmax), G.bloco(Bt * T, D, e0=-20, espalha=4)
    s = spec.Spec(32)
    o_r, P_r = s.atencao(qkv, Bt, T, H)
    g_r = s.atencao_back(go, qkv, P_r, Bt, T, H)
    o_c, P_c = oc.atencao(para_gpu(qkv), Bt, T, H)
    g_c = oc.atencao_back(para_gpu(go), para_gpu(qkv), P_c, Bt, T, H)
    torch.cuda.synchronize()
    compara(f"atencao mmax {mmax} T {T}", [*o_c, P_c], [*o_r, P_r])
    compara(f"atencao_back mmax {mmax} T {T}", list(g_c), list(g_r))


@pytest.mark.gpu
@pytest.mark.parametrize("blk,Bt,T,H,D,e0,longe", [(32, 2, 32, 2, 128, -8, 0), (32, 1, 96, 4, 64, -8, 1), (128, 1, 160, 8, 128, -8, 2), (32, 1, 288, 26, 416, -5, 3),
                                                   (32, 1, 416, 2, 128, -8, 4), (32, 1, 1024, 34, 544, -4, 0), (32, 1, 1024, 2, 128, -8, 5),
                                                   (32, 1, 160, 8, 32, -8, 2), (128, 1, 288, 32, 128, -5, 3), (32, 1, 1024, 72, 288, -6, 0), (32, 2, 416, 8, 32, -8, 4)])
def test_atencao_janelas(amb, blk, Bt, T, H, D, e0, longe):
    """The tensor-core attention walks the keys in windows of 128 that end with a tile of 64 queries: sequence lengths from one
    half tile to 16 tiles, odd numbers of half tiles, the head dimensions, scores and slopes (heads 16 and on) that need several
    windows, and a backward on a P with non-zeros put far from the diagonal, against the oracle."""
    ops, oc, reg = amb
    ops.define_blk(blk)
    reg.novo_passo(0)
    G = casos.Gen(911 + T + H + D, blk)
    qkv, go = G.bloco(Bt * T, 3 * D, e0=e0, espalha=4, zera=0.02), G.bloco(Bt * T, D, e0=-20, espalha=4)
    s = spec.Spec(blk)
    o_r, P_r = s.atencao(qkv, Bt, T, H)
    try:
        o_c, P_c = oc.atencao(para_gpu(qkv), Bt, T, H)
        P = P_r.clone()
        for n in range(longe):                       # [Bt*H, T (keys), T (queries)]
            j = (37 * n) % (T // 4)
            P[n % (Bt * H), j, T - 1 - 29 * n] = 200
            P[(n + 1) % (Bt * H), j + 3, (T // 2 + 64 * n) % T:] = 3 if j + 3 < (T // 2 + 64 * n) % T else 0
        g_r = s.atencao_back(go, qkv, P, Bt, T, H)
        g_c = oc.atencao_back(para_gpu(go), para_gpu(qkv), para_gpu(P), Bt, T, H)
        torch.cuda.synchronize()
    finally:
        ops.define_blk(32)
    compara(f"atencao T {T} H {H} D {D}", [*o_c, P_c], [*o_r, P_r])
    compara(f"atencao_back T {T} H {H} D {D}", list(g_c), list(g_r))


@pytest.mark.gpu
@pytest.mark.parametrize("limite", [False, True])
@pytest.mark.parametrize("blk,Bt,T,H,e0,esp", [(32, 1, 32, 8, -8, 4), (128, 1, 64, 32, -4, 3), (32, 1, 128, 64, -8, 4), (32, 1, 96, 8, -1, 0), (32, 2, 128, 8, 0, 0),
                                               (32, 1, 64, 8, 1, 0)])
def test_atencao_cabecas_de_4(amb, blk, Bt, T, H, e0, esp, limite):
    """Heads of 4 at T <= 128: every slope (64 heads), score shifts on both sides of the float rounding's range (shift 3; 1 and a
    left shift take the general way), and a backward on a P with entries put far from the diagonal, against the oracle."""
    ops, oc, reg = amb
    ops.define_blk(blk)
    reg.novo_passo(0)
    D = 4 * H
    G = casos.Gen(3 * T + H + e0, blk)
    qkv, go = G.bloco(Bt * T, 3 * D, e0=e0, espalha=esp, zera=0.02 if esp else 0.0), G.bloco(Bt * T, D, e0=-20, espalha=4)
    s = spec.Spec(blk, limite=limite)
    o_r, P = s.atencao(qkv, Bt, T, H)
    ops.ATENCAO_LIMITE = limite
    try:
        o_c, P_c = oc.atencao(para_gpu(qkv), Bt, T, H)
        P2 = P.clone()                               # [Bt*H, T (keys), T (queries)]
        P2[0, 1, T - 1] = 255
        P2[1, 5:9, T - 20:] = 7
        g_r = s.atencao_back(go, qkv, P2, Bt, T, H)
        g_c = oc.atencao_back(para_gpu(go), para_gpu(qkv), para_gpu(P2), Bt, T, H)
        torch.cuda.synchronize()
    finally:
        ops.ATENCAO_LIMITE = False
        ops.define_blk(32)
    compara(f"atencao T {T} H {H} e0 {e0}", [*o_c, P_c], [*o_r, P])
    compara(f"atencao_back T {T} H {H} e0 {e0} limite {limite}", list(g_c), list(g_r))


@pytest.mark.gpu
def test_atencao_back_com_P_alterado(amb):
    """The backward works from the P it is given: with whole tiles of P zeroed by hand (tiles its zero map then leaves out, tiles
    next to the diagonal, a whole key range) it still equals the oracle's backward on that same P."""
    ops, oc, reg = amb
    ops.define_blk(32)
    reg.novo_passo(0)
    Bt, T, H, D = 1, 1024, 2, 128
    G = casos.Gen(4242, 32)
    qkv, go = G.bloco(Bt * T, 3 * D, espalha=3, zera=0.02, mmax=30), G.bloco(Bt * T, D, e0=-20, espalha=4)
    s = spec.Spec(32)
    _, P = s.atencao(qkv, Bt, T, H)
    P = P.clone()                                    # [Bt*H, T (keys), T (queries)]
    P[0, 0:128, 256:] = 0                            # a far key range for all later queries
    P[0, 512:576, 576:640] = 0                       # the tile right of a diagonal tile
    P[1, 640:704, 640:704] = 0                       # a diagonal tile itself
    P[1, :, 896:960] = 0                             # every key of one query tile
    g_r = s.atencao_back(go, qkv, P, Bt, T, H)
    g_c = oc.atencao_back(para_gpu(go), para_gpu(qkv), para_gpu(P), Bt, T, H)
    torch.cuda.synchronize()
    compara("atencao_back with hand-zeroed tiles of P", list(g_c), list(g_r))


@pytest.mark.gpu
@pytest.mark.parametrize("R,C", [(128, 192), (256, 64), (8192, 1088)])
@pytest.mark.parametrize("afasta,fundo", [(0, 0), (14, 0), (15, 8), (24, 9), (24, 10), (25, 0), (100, 0), (101, 0)])
def test_transpoe_metades_e_fp32(amb, R, C, afasta, fundo):
    """The transposition in halves up to its limits and beyond: rows whose exponents lie `afasta` below their neighbours' (24 is the last that halves hold, 100 the last
    for fp32), zero blocks, columns that only the lower rows have and, with `fundo`, columns whose largest element lies so far down
    that the factor is 2^15 or 2^16."""
    ops, oc, reg = amb
    ops.define_blk(32)
    reg.novo_passo(0)
    G = casos.Gen(R + C + afasta, 32)
    m, E = G.bloco(R, C, e0=-10, espalha=0, zera=0.05)
    zero = E == -127
    E[1::3] -= afasta
    E[zero] = -127
    m[::3, 5::64] = 0
    m[2::3, 5::64] = 0
    if fundo:                                            # 1 at 2^-fundo, or nothing: Eo = -fundo - 6
        m[:, 9::64] = 0
        m[1::3, 9::64] = 1
        E[1::3] = torch.where(zero[1::3], E[1::3], torch.full_like(E[1::3], -10 - fundo))
    X = para_gpu((m, E))
    out = oc.transpoe(X)
    torch.cuda.synchronize()
    compara(f"transpoe {R}x{C} afasta {afasta} fundo {fundo}", list(out), list(spec.Spec(32).transpoe(X)))
