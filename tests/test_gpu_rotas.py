"""Which kernel a call takes and with how many blocks (read from a recording of the call), and the kernels' forms that only particular sizes or data reach,
each against the specification or the CUDA-core kernel."""
import ctypes
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
    reg = registro.Registro(tempfile.mkdtemp(), "rotas", vigiar=True, eco=False, salvar=False)
    oc = ops.OpsCuda(reg)
    reg.novo_passo(0)
    yield ops, oc, reg
    ops.define_blk(32)
    oc.lib.jt_gemm_via(0)
    oc.lib.jt_gemm_tn(0)


class _Lancamento(ctypes.Structure):                     # CUDA_KERNEL_NODE_PARAMS
    _fields_ = [("func", ctypes.c_void_p), ("grade", ctypes.c_uint * 3), ("bloco", ctypes.c_uint * 3), ("smem", ctypes.c_uint),
                ("args", ctypes.c_void_p), ("extra", ctypes.c_void_p), ("kern", ctypes.c_void_p), ("ctx", ctypes.c_void_p)]


def lancamentos(oc, f, ao_lado=False):
    """The kernels that f launches: (name, blocks)."""
    cu = ctypes.CDLL("libcuda.so.1")
    f()                                                  # (kernel attributes are set at a first launch)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    vigiar, oc.reg.vigiar = oc.reg.vigiar, False         # (the check after each operator waits for the GPU)
    try:
        with torch.cuda.graph(g):
            (oc.lib.jt_stream_ao_lado if ao_lado else oc.lib.jt_stream)(torch.cuda.current_stream().cuda_stream)
            f()
    finally:
        oc.lib.jt_stream(None)
        oc.reg.vigiar = vigiar
    grafo, n = ctypes.c_void_p(g.raw_cuda_graph()), ctypes.c_size_t(0)
    assert cu.cuGraphGetNodes(grafo, None, ctypes.byref(n)) == 0
    nos = (ctypes.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(grafo, nos, ctypes.byref(n)) == 0
    r = []
    for no in nos:
        tipo = ctypes.c_int(-1)
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(no), ctypes.byref(tipo)) == 0
        if tipo.value != 0:
            continue
        p, nome = _Lancamento(), ctypes.c_char_p()
        assert cu.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(no), ctypes.byref(p)) == 0
        assert (cu.cuKernelGetName(ctypes.byref(nome), ctypes.c_void_p(p.kern)) if p.kern else cu.cuFuncGetName(ctypes.byref(nome), ctypes.c_void_p(p.func))) == 0
        r.append((nome.value.decode(), p.grade[0] * p.grade[1] * p.grade[2]))
    return r


def inteiros(semente):
    g = torch.Generator(device="cuda").manual_seed(semente)
    return lambda a, b, forma: torch.randint(a, b + 1, forma, generator=g, device="cuda", dtype=torch.int32).to(torch.int8)


# ------------------------------------------------------------------------------------------------ transposition
def em_metades(X, colunas):
    """How many (32 rows x 128 columns, columns a lane) pieces meet both conditions of the transposition in halves, of how many: exponents at most 24 apart,
    all-zero blocks aside, and no column whose largest element lies so far down that its factor exceeds 2^15 (with one column a lane, in a block whose largest
    exponent is below -80)."""
    m, E = (t.to(torch.int64) for t in X)
    R, C = m.shape
    falta = -C % 128
    m = torch.nn.functional.pad(m, (0, falta)).reshape(R // 32, 32, -1, 4, 32)
    E = torch.nn.functional.pad(E, (0, falta // 32), value=casos.E_ZERO).reshape(R // 32, 32, -1, 4)
    ref = E.amax(1, keepdim=True)
    perto = ((ref - E <= 24) | (E == casos.E_ZERO)).all(3).all(1)
    # log2 of a column's largest element: a mantissa below 2^b at exponent e counts b + e
    bits = torch.frexp(m.abs().to(torch.float64))[1].to(torch.int64)
    topo = torch.where(m != 0, bits + E[..., None], torch.full_like(m, -1000)).amax(1)
    serve = (topo == -1000) | (ref[:, 0, :, :, None] - (topo - 7) <= 15)
    if colunas == 1:
        serve = serve | (ref[:, 0, :, :, None] >= -80)
    serve = serve.reshape(*serve.shape[:3], 8, 4)        # 8 lanes of 4 columns in a block
    serve = serve.all(4).all(3).all(2) if colunas == 4 else serve.all(3).all(2)
    return int((perto[..., None] & serve.reshape(*perto.shape, -1)).sum()), serve.numel()


@pytest.mark.parametrize("R,C,colunas", [(128, 192, 1), (8192, 1088, 4)])
@pytest.mark.parametrize("afasta", [14, 15, 20, 24])
def test_transpoe_metades_todos_os_fatores(amb, R, C, colunas, afasta):
    """Every factor 2^0 to 2^-afasta of the transposition in halves, subnormal ones among them, beside rows at the block's largest exponent, so that every piece
    is put out in halves."""
    ops, oc, reg = amb
    G = casos.Gen(R + C + afasta, 32)
    m, E = G.bloco(R, C, e0=-10, espalha=0, zera=0.05)
    zero = E == casos.E_ZERO
    E[1::3] -= torch.randint(0, afasta + 1, E[1::3].shape, generator=G.g).to(torch.int8)
    E[1::12] = -10 - afasta
    E[zero] = casos.E_ZERO
    tem, de = em_metades((m, E), colunas)
    assert tem == de
    X = para_gpu((m, E))
    compara(f"transpoe {R}x{C} afasta {afasta}", list(oc.transpoe(X)), list(spec.Spec(32).transpoe(X)))


@pytest.mark.parametrize("R,C,colunas", [(128, 192, 1), (8192, 1088, 4)])
@pytest.mark.parametrize("e0", [-10, -80, -81])
@pytest.mark.parametrize("fundo", [8, 9, 10, 24])
def test_transpoe_metades_fatores_grandes(amb, R, C, colunas, e0, fundo):
    """In one block of four, a column that holds nothing but ones `fundo` below the largest exponent: its factor is 2^14, 2^15 (the largest half), 2^16 or 2^30 (the most
    there is), which take two multiplications, or fp32 with four columns a lane or below the exponent -80."""
    ops, oc, reg = amb
    G = casos.Gen(R + C + fundo, 32)
    m, E = G.bloco(R, C, e0=e0, espalha=0)
    E[1::3, 1::4] = e0 - fundo
    m[:, 41::128] = 0
    m[1::3, 41::128] = 1
    tem, de = em_metades((m, E), colunas)
    assert tem == de if fundo <= 9 or (colunas == 1 and e0 >= -80) else tem < de
    X = para_gpu((m, E))
    compara(f"transpoe {R}x{C} e0 {e0} fundo {fundo}", list(oc.transpoe(X)), list(spec.Spec(32).transpoe(X)))


@pytest.mark.parametrize("R,C,colunas", [(128, 192, 1), (8192, 1088, 4)])
def test_transpoe_metades_esparsa(amb, R, C, colunas):
    """Few elements of any size at exponents 24 apart: columns with every factor in one warp, empty ones among them."""
    ops, oc, reg = amb
    G = casos.Gen(R + C, 32)
    m, E = G.bloco(R, C, e0=-20, espalha=12)
    m[torch.rand(R, C, generator=G.g) > 0.04] = 0
    tem, de = em_metades((m, E), colunas)
    assert tem == de if colunas == 1 else tem < de
    X = para_gpu((m, E))
    compara(f"transpoe {R}x{C}", list(oc.transpoe(X)), list(spec.Spec(32).transpoe(X)))


@pytest.mark.parametrize("R,C", [(128, 192), (8192, 1088)])
@pytest.mark.parametrize("e0", [-126, -120, -103, -102, -95, -81, -80, -10, 0])
def test_transpoe_menor_expoente_com_mantissas(amb, R, C, e0):
    """Blocks of exponent -127 whose mantissas are not cleared: their elements count as what they are (all but nothing), also where they are a column's only ones, or beside
    ones 24 below the largest exponent."""
    ops, oc, reg = amb
    G = casos.Gen(R + C + 1000 - e0, 32)
    m, E = G.bloco(R, C, e0=e0, espalha=0)
    E[1::5] = max(e0 - 24, -126)
    E[2::5] = casos.E_ZERO
    linha = torch.arange(R) % 5
    m[linha != 2, 7::32] = 0
    m[(linha != 2) & (linha != 1), 9::32] = 0
    m[linha == 1, 9::32] = 1
    X = para_gpu((m, E))
    compara(f"transpoe {R}x{C} e0 {e0}", list(oc.transpoe(X)), list(spec.Spec(32).transpoe(X)))


# ------------------------------------------------------------------------------------------------ products
@pytest.mark.parametrize("M,N,largura,so", [(9472, 128, 64, 1), (9600, 128, 128, 0), (2048, 768, 128, 0), (18944, 128, 128, 0), (2048, 1280, 64, 0), (4096, 1024, 128, 0)])
@pytest.mark.parametrize("cru", [False, True])
def test_gemm_8_bits_largura(amb, M, N, largura, so, cru):
    """The 8-bit kernel's tiles by their number: 74 (64 wide, an SM each), 75, 96 and 148 (128 wide), 160 (64 wide, two to an SM), 256 (128 wide, two rounds)."""
    ops, oc, reg = amb
    ints = inteiros(M + N)
    A, B = ((ints(-127, 127, (R, 256)), ints(-12, -4, (R, 8))) for R in (M, N))
    f = lambda: list(oc.gemm(A, B, cru=cru))
    assert oc.lib.jt_gemm_via(2) == 0
    quer = f()
    assert oc.lib.jt_gemm_via(1) == 0
    assert [n for n, b in lancamentos(oc, f) if "k_gemm_tc" in n and f"ELi{largura}ELb{so}E" in n and b == M // 128 * (N // largura)]
    compara(f"{M}x{N}x256 cru {cru}", f(), quer)


@pytest.mark.parametrize("M,N,K,op,nucleo", [(2048, 640, 128, "gemm", "tc"), (2048, 640, 256, "gemm cru", "tc"), (1920, 1024, 256, "gemm", "tc"), (2048, 1536, 128, "gemm", "tc"),
                                             (2048, 1536, 128, "gemm cru", "tc"), (8192, 512, 128, "gemm cru", "tc"), (2048, 1280, 256, "gemm_relu2_back", "tc"),
                                             (2048, 1536, 512, "gemm", "h"), (2048, 2048, 256, "gemm", "h"), (4096, 2048, 128, "gemm", "h"), (2048, 1024, 1024, "gemm cru", "h")])
def test_gemm_escolha_com_K_curto(amb, M, N, K, op, nucleo):
    """Products of one to four rounds of tiles and short K take the kernel that is measured to be faster: the 8-bit one up to K = 128 or 256, by the output."""
    ops, oc, reg = amb
    ints = inteiros(M + K)
    A, B, X = (ints(-127, 127, (M, K)), ints(-9, -8, (M, K // 32))), (ints(-127, 127, (N, K)), ints(-9, -8, (N, K // 32))), (ints(-127, 127, (M, N)), ints(-12, -4, (M, N // 32)))
    f = lambda: casos.roda(oc, op.split()[0], (A, B, X) if "back" in op else (A, B), dict(cru=True) if "cru" in op else {})
    assert oc.lib.jt_gemm_via(2) == 0
    quer = f()
    assert oc.lib.jt_gemm_via(0) == 0
    assert [n for n, _ in lancamentos(oc, f) if f"k_gemm_{nucleo}" in n]
    compara(f"{op} {M}x{N}x{K}", f(), quer)


@pytest.mark.parametrize("M,N,K,via,nucleo,blocos", [(1024, 512, 4096, 0, "h", 32), (256, 256, 2048, 1, "tc", 4), (256, 256, 4096, 0, "tc", 64), (512, 512, 8192, 0, "tc", 128),
                                                     (256, 256, 4224, 1, "tc", 4), (512, 256, 4608, 1, "tc", 32), (320, 512, 8320, 0, "h", 96), (128, 128, 16384, 4, "h", 32),
                                                     (1024, 1024, 4096, 4, "h", 64), (12288, 640, 4096, 0, "tc", 480)])
def test_gemm_bloco_128_partes(amb, M, N, K, via, nucleo, blocos):
    """Raw products of block 128 and few tiles: K ranges where they are worth what clearing and adding cost, by the kernel that is faster with them."""
    ops, oc, reg = amb
    ops.define_blk(128)
    ints = inteiros(M + N + K)
    A, B = ((ints(-127, 127, (R, K)), ints(-12, -4, (R, K // 128))) for R in (M, N))
    f = lambda: list(oc.gemm(A, B, cru=True))
    assert oc.lib.jt_gemm_via(2) == 0
    quer = f()
    assert oc.lib.jt_gemm_via(via) == 0
    assert [b for n, b in lancamentos(oc, f) if f"k_gemm_{nucleo}" in n] == [blocos]
    compara(f"{M}x{N}x{K} via {via}", f(), quer)


@pytest.mark.parametrize("caso", ["comum", "saturados", "expoentes afastados", "linhas nulas", "acumuladores grandes"])
@pytest.mark.parametrize("op", ["gemm", "gemm cru", "gemm_soma", "gemm_relu2", "gemm_relu2_back"])
def test_gemm_64_dois_por_sm(amb, op, caso):
    """The 8-bit kernel's 64-wide tiles with two blocks on an SM (more than 148 of them) in every output mode: the rounding's range check and the output stage's
    integer side as well as the ordinary ones."""
    ops, oc, reg = amb
    M, N, K = 2432, 1024, 512
    G = casos.Gen(4243, 32)
    A, B, X = G.bloco(M, K, espalha=2 if caso != "comum" else 8, zera=0.05 if caso == "comum" else 0.0), G.bloco(N, K, espalha=2), G.bloco(M, N, espalha=3)
    if caso == "saturados":
        A[0][5::64], B[0][7::32] = 127, -127
        A[1][5::64], B[1][7::32] = -8, -8
    elif caso == "expoentes afastados":
        B[1][0::2] -= 50
        B[1][1::2] += 20
    elif caso == "linhas nulas":
        B[0][::3], B[1][::3] = 0, casos.E_ZERO
    elif caso == "acumuladores grandes":
        A, B = (torch.full_like(A[0], 127), torch.full_like(A[1], -8)), (torch.full_like(B[0], 127), torch.full_like(B[1], -8))
    A, B, X = para_gpu(A), para_gpu(B), para_gpu(X)
    args, kw = ((A, B, X) if op in ("gemm_soma", "gemm_relu2_back") else (A, B)), (dict(cru=True) if op == "gemm cru" else {})
    assert oc.lib.jt_gemm_via(1) == 0 and oc.lib.jt_gemm_tn(64) == 0
    f = lambda: casos.roda(oc, op.split()[0], args, kw)
    assert [(n, b) for n, b in lancamentos(oc, f) if "k_gemm_tc" in n and "ELi1ELi64ELb0E" in n and b == 304]
    tem = f()
    torch.cuda.synchronize()
    compara(f"{op} {caso}", tem, casos.roda(spec.Spec(32), op.split()[0], args, kw))


@pytest.mark.parametrize("M,N,soma", [(4736, 512, False), (19072, 128, True)])
@pytest.mark.parametrize("op", ["gemm", "gemm_relu2"])
@pytest.mark.parametrize("afasta", [0, 12])
def test_gemm_somas_linha(amb, M, N, soma, op, afasta):
    """148 tiles, a tile per SM, and 149: from there on half-precision products look for tiles that add up in tensor memory.  With exponents that round nothing
    and with ones that round everywhere."""
    ops, oc, reg = amb
    K = 512
    ints = inteiros(M + afasta)
    A, B = ((ints(-127, 127, (R, K)), ints(-9 - afasta, -8, (R, K // 32))) for R in (M, N))
    assert oc.lib.jt_gemm_via(2) == 0
    quer = casos.roda(oc, op, (A, B), {})
    assert oc.lib.jt_gemm_via(4) == 0
    f = lambda: casos.roda(oc, op, (A, B), {})
    assert [n for n, _ in lancamentos(oc, f) if "k_gemm_h" in n and f"ELi128ELb0ELb{int(soma)}E" in n]
    compara(f"{op} {M}x{N}x{K} afasta {afasta}", f(), quer)


# ------------------------------------------------------------------------------------------------ beside another chain
LADO = 48                                                # most blocks of a product there that has more of them than 128 x 128 tiles


@pytest.mark.parametrize("via", [0, 1])
@pytest.mark.parametrize("M,N,K,cru", [(1536, 512, 1024, True), (2048, 512, 1024, True), (512, 2048, 1024, True), (1024, 512, 512, True), (2048, 512, 512, False),
                                       (512, 512, 256, True), (256, 256, 4096, True), (384, 1024, 4096, True), (512, 384, 128, False), (10240, 128, 128, False)])
def test_ao_lado_blocos(amb, M, N, K, cru, via):
    """Under jt_stream_ao_lado a product of any kernel has at most 48 blocks, or one for each of its 128 x 128 tiles, and gives the same bits."""
    ops, oc, reg = amb
    ints = inteiros(M + N + K)
    A, B = ((ints(-127, 127, (R, K)), ints(-12, -4, (R, K // 32))) for R in (M, N))
    assert oc.lib.jt_gemm_via(via) == 0
    f = lambda: oc.gemm(A, B, cru=cru)
    quer = f()
    blocos = [b for n, b in lancamentos(oc, f, ao_lado=True) if "k_gemm" in n]
    assert len(blocos) == 1 and blocos[0] <= max(LADO, (M // 128) * (N // 128))
    try:
        oc.lib.jt_stream_ao_lado(None)
        tem = f()
    finally:
        oc.lib.jt_stream(None)
    torch.cuda.synchronize()
    compara(f"{M}x{N}x{K} cru {cru} via {via}", list(tem), list(quer))


@pytest.mark.parametrize("M,N,K", [(1536, 512, 1024), (2048, 512, 1024), (512, 2048, 1024)])
def test_ao_lado_o_mesmo_nucleo(amb, M, N, K):
    """What takes the half-precision kernel alone takes it beside another chain too: that 64-wide tiles are ruled out there does not send it to the 8-bit kernel."""
    ops, oc, reg = amb
    ints = inteiros(M + N + K)
    A, B = ((ints(-127, 127, (R, K)), ints(-12, -4, (R, K // 32))) for R in (M, N))
    f = lambda: oc.gemm(A, B, cru=True)
    for ao_lado in (False, True):
        assert [n for n, _ in lancamentos(oc, f, ao_lado) if "k_gemm_h" in n]
