"""Calls in the forms that the other tests do not use: tensors that start anywhere in a larger buffer, pairs given as lists, several streams,
little memory, a first call inside a recording, very many heads.  Everything against the oracle, or against the same operator called
the plain way."""
import gc
import tempfile
import threading
import time

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


def _limita_torch(folga):
    """PyTorch's allocator gets `folga` bytes beyond what it holds (and nothing that earlier tests still hold comes free meanwhile)."""
    gc.collect()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + folga) / torch.cuda.mem_get_info()[1])


@pytest.fixture
def memoria(amb):
    gc.collect()
    torch.cuda.empty_cache()                           # (else the test's tensors may share a segment with a large free rest of an earlier test's)
    yield _limita_torch
    torch.cuda.set_per_process_memory_fraction(1.0)
    amb[1].lib.jt_espaco_limite(0)


def _problema(blk, Bt, T, H, hd, semente=23):
    G = casos.Gen(semente + T + H, blk)
    D, M = H * hd, Bt * T
    return para_gpu(G.bloco(M, 3 * D, espalha=4, zera=0.02)), para_gpu(G.bloco(M, D, e0=-20, espalha=4)), (Bt, T, H)


def _tudo(oc, qkv, go, forma):
    """Raw and quantised attention, both ways."""
    o, P = oc.atencao(qkv, *forma)
    g = oc.atencao_back(go, qkv, P, *forma)
    oq, Pq = oc.atencao_quant(qkv, *forma)
    return [*o, P, *g, *oq, Pq, *oc.atencao_back_quant(go, qkv, P, *forma)]


ESPACOS = [(32, 2, 96, 2, 64), (32, 2, 128, 2, 64), (32, 3, 64, 16, 16), (32, 1, 288, 8, 4), (128, 1, 160, 8, 16)]


@pytest.mark.parametrize("blk,Bt,T,H,hd", ESPACOS)
def test_atencao_sem_memoria_para_o_espaco(amb, memoria, blk, Bt, T, H, hd):
    """Same bits with the workspace of the caller's allocator, of the library's own pool (the launches are on another stream than the
    allocator's) and with none: too little memory for either."""
    ops, oc, reg = amb
    ops.define_blk(blk)
    qkv, go, forma = _problema(blk, Bt, T, H, hd)
    ref = _tudo(oc, qkv, go, forma)
    s = spec.Spec(blk)
    compara("atencao", ref[:3], casos.plano(s.atencao(qkv, *forma)))
    compara("atencao_back", ref[3:5], s.atencao_back(go, qkv, ref[2], *forma))
    outro = torch.cuda.Stream()
    torch.cuda.synchronize()
    for limite in (0, 4096 + 4 * Bt * H * (8 + T), 1024):
        oc.lib.jt_espaco_limite(limite)
        with torch.cuda.stream(outro):                 # the library goes on launching on the default stream, which waits for nobody here
            if limite != 1024:
                out = _tudo(oc, qkv, go, forma)
                torch.cuda.synchronize()
                compara(f"own workspace, at most {limite} bytes", out, ref)
            else:
                with pytest.raises(Exception, match="refused the launch of 'atencao_back'"):      # not even the sums of the rows
                    oc.atencao_back(go, qkv, ref[2], *forma)
    oc.lib.jt_espaco_limite(0)
    assert oc.lib.jt_espaco_libera() == 0


def test_atencao_com_o_alocador_cheio(amb, memoria):
    """PyTorch's allocator has room for the outputs and none for the workspace: the library's pool serves, then the general kernels."""
    ops, oc, reg = amb
    qkv, go, forma = _problema(32, 8, 128, 64, 16)
    o, P = oc.atencao(qkv, *forma)
    ref = [*o, P, *oc.atencao_back(go, qkv, P, *forma)]
    del o, P
    for limite in (0, 1 << 20):
        oc.lib.jt_espaco_limite(limite)
        memoria(50 << 20)                              # outputs 15 and 19 MB (in segments of 20 and 34), workspaces 33 and 50
        o, P = oc.atencao(qkv, *forma)
        compara("forward", [*o, P], ref[:3])
        del o, P
        memoria(45 << 20)
        g = oc.atencao_back(go, qkv, ref[2], *forma)
        compara("backward", g, ref[3:])
        del g


def test_atencao_em_duas_correntes(amb):
    """Two problems at the same time on two streams: neither sees the other's workspace, with the allocator's and with the library's."""
    ops, oc, reg = amb
    reg.vigiar = False
    ps = [_problema(32, 64, 128, 32, 16, semente=n) for n in (1, 2)]
    refs = [_tudo(oc, *p) for p in ps]
    torch.cuda.synchronize()
    st = [torch.cuda.Stream() for _ in ps]
    try:
        for volta in range(12):
            outs = [[], []]
            for n in (0, 1):
                with torch.cuda.stream(st[n]):
                    torch.cuda._sleep(2_000_000)       # the second one's launches are queued before the first one starts
            for rep in range(2):
                for n in (0, 1):
                    with torch.cuda.stream(st[n]):
                        oc.lib.jt_stream(st[n].cuda_stream)
                        outs[n].append(_tudo(oc, *ps[n]))
            torch.cuda.synchronize()
            for n in (0, 1):
                for out in outs[n]:
                    compara(f"stream {n}, time {volta}", out, refs[n])
    finally:
        oc.lib.jt_stream(None)


@pytest.mark.parametrize("proprio", [False, True])
def test_atencao_primeira_chamada_numa_gravacao(amb, proprio):
    """The first call at a size, both ways, inside a CUDA graph: with the allocator's workspace and with the library's (the graph's own); two
    graphs recorded on one stream are replayed at the same time on two."""
    ops, oc, reg = amb
    reg.vigiar = False
    ps = [_problema(32, 64, 96, 32, 16, semente=n) for n in (1, 2)]
    refs = [_tudo(oc, *p) for p in ps]
    torch.cuda.synchronize()
    if proprio:
        oc._ws_at = (0, 0)                             # the launcher brings none
    grafos, saidas = [], []
    try:
        for p in ps:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                oc.lib.jt_stream(torch.cuda.current_stream().cuda_stream)
                saidas.append(_tudo(oc, *p))
            grafos.append(g)
    finally:
        oc.lib.jt_stream(None)
    st = [torch.cuda.Stream() for _ in ps]
    for volta in range(4):
        for g, s in zip(grafos, st):
            with torch.cuda.stream(s):
                g.replay()
                g.replay()
        torch.cuda.synchronize()
        for n in (0, 1):
            compara(f"replay {volta} of graph {n}", saidas[n], refs[n])
    del grafos


@pytest.mark.parametrize("blk", [32, 128])
def test_produto_com_espaco_de_128_em_128_bytes(amb, blk):
    """The workspace of a product may start at any multiple of 128 bytes (small blocks of PyTorch's allocator start at multiples of 512): on
    64 rows, which only the half-precision path of the forced ones takes, the call must serve."""
    import ctypes
    ops, oc, reg = amb
    ops.define_blk(blk)
    M, N, K = 64, 128, 256
    G = casos.Gen(12, blk)
    A, B = para_gpu(G.bloco(M, K, espalha=4)), para_gpu(G.bloco(N, K, espalha=4))
    ref = spec.Spec(blk).gemm(A, B)
    oc.lib.jt_gemm_via(4)
    n = oc.lib.jt_gemm_ws_bytes(M, N, K, 0)
    assert n > 0
    buf = torch.empty(n + 2048, dtype=torch.uint8, device="cuda")
    for desl in (128, 512, 896):
        ws = buf[(-buf.data_ptr()) % 1024 + desl:]
        C = torch.zeros(M, N, dtype=torch.int8, device="cuda"), torch.zeros(M, N // blk, dtype=torch.int8, device="cuda")
        p = [ctypes.c_void_p(t.data_ptr()) if t is not None else None for t in (*A, *B, *C, *[None] * 8, ws)]
        assert oc.lib.jt_gemm_ws(*p, *(ctypes.c_int(v) for v in (M, N, K, 0, 0))) == 0
        torch.cuda.synchronize()
        compara(f"workspace at {desl}", C, ref)


@pytest.mark.parametrize("via,hd,H", [(0, 16, 16), (1, 16, 16), (0, 64, 16)])
def test_atencao_com_mais_de_65535_cabecas(amb, via, hd, H):
    """(Sequences x heads) beyond the limit of a grid's y: 17 sequences repeated 241 times give 241 times what they give alone."""
    ops, oc, reg = amb
    reg.vigiar = False
    n, T = 241, 32
    qkv, go, _ = _problema(32, 17, T, H, hd)
    o, P = oc.atencao(qkv, 17, T, H)
    ref = [*o, P, *oc.atencao_back(go, qkv, P, 17, T, H)]
    assert 17 * n * H > 65535
    oc.lib.jt_atencao_via(via)
    try:
        big, gobig = tuple(t.repeat(n, 1) for t in qkv), tuple(t.repeat(n, 1) for t in go)
        o, P = oc.atencao(big, 17 * n, T, H)
        out = [*o, P, *oc.atencao_back(gobig, big, P, 17 * n, T, H)]
    finally:
        oc.lib.jt_atencao_via(0)
    for i, (a, b) in enumerate(zip(out, ref)):
        assert bool((a.view(n, *b.shape) == b).all()), f"output {i}"


def test_memoria_esgotada_tem_o_tipo_do_alocador(amb, memoria):
    """Where an output does not fit, every kind of operator raises what PyTorch's allocator raises, and works again once there is room."""
    ops, oc, reg = amb
    G = casos.Gen(41, 32)
    A, B, (qkv, go, forma) = para_gpu(G.bloco(16384, 2048)), para_gpu(G.bloco(2048, 2048)), _problema(32, 64, 128, 32, 64)
    c = oc.gemm(A, B, cru=True)
    # (every call wants 32 MB somewhere: more than what is free in a segment that is in use)
    for nome, f in (("relu2", lambda: oc.relu2(A)), ("gemm", lambda: oc.gemm(A, B)), ("gemm_cru", lambda: oc.gemm(A, B, cru=True)),
                    ("gemm_relu2", lambda: oc.gemm_relu2(A, B)), ("quant", lambda: oc.quant(c)), ("atencao", lambda: oc.atencao(qkv, *forma)),
                    ("atencao_quant", lambda: oc.atencao_quant(qkv, *forma)), ("rms", lambda: oc.rms(A))):
        memoria(1 << 20)
        try:
            f()
            raise AssertionError(f"{nome} found memory; {torch.cuda.memory_reserved() - torch.cuda.memory_allocated()} bytes were free")
        except torch.OutOfMemoryError:
            pass
    torch.cuda.set_per_process_memory_fraction(1.0)
    compara("relu2", oc.relu2(B), spec.Spec(32).relu2(B))


@pytest.mark.parametrize("externos", [False, True])
def test_produto_sem_memoria_para_o_espaco(amb, memoria, externos):
    """A product whose workspace does not fit beside its output runs on the kernels that need none, with the same bits."""
    ops, oc, reg = amb
    G = casos.Gen(43, 32)
    A, B = para_gpu(G.bloco(4096, 8192, espalha=4)), para_gpu(G.bloco(2048, 8192, espalha=4))
    kw = dict(RA=oc.max_linha(A), RB=oc.max_linha(B)) if externos else {}
    ref = oc.gemm(A, B, **kw)
    assert oc.lib.jt_gemm_ws_bytes(4096, 2048, 8192, 0) > 64 << 20
    memoria(64 << 20)
    out = oc.gemm(A, B, **kw)
    compara("gemm", out, ref)


def test_outros_fios_andam_enquanto_um_lancamento_espera(amb):
    """Launches beyond what the GPU's queue holds wait behind a kernel of about a second; another Python thread runs meanwhile."""
    ops, oc, reg = amb
    reg.vigiar = False
    A = para_gpu(casos.Gen(3, 32).bloco(128, 128))
    oc.relu2(A)
    torch.cuda.synchronize()
    marcas, fim = [], threading.Event()

    def bate():
        while not fim.is_set():
            marcas.append(time.perf_counter())
            time.sleep(0.001)

    fio = threading.Thread(target=bate)
    fio.start()
    t0 = time.perf_counter()
    torch.cuda._sleep(2_000_000_000)
    for _ in range(4000):
        oc.relu2(A)
    dt = time.perf_counter() - t0
    torch.cuda.synchronize()
    fim.set()
    fio.join()
    assert dt > 0.5, "the launches did not have to wait"
    assert max(b - a for a, b in zip(marcas, marcas[1:])) < 0.4 * dt


def test_pares_em_listas(amb):
    """A (mantissas, exponents) pair may be a list: every operator gives what it gives for the tuple, and the messages of the checks stay."""
    from jatai_b200.registro import ErroJatai
    ops, oc, reg = amb
    G = casos.Gen(51, 32)
    A, B, X, W = (para_gpu(G.bloco(256, 256, espalha=4)) for _ in range(4))
    qkv, go, forma = _problema(32, 2, 64, 2, 64)
    c, alvo = oc.gemm(A, B, cru=True), torch.randint(0, 256, (256,), device="cuda", dtype=torch.int32)
    y, cache = oc.rms(A)
    P = oc.atencao(qkv, *forma)[1]
    novo = lambda t: tuple(x.clone() for x in t)
    for f in (lambda k: oc.gemm(k(A), k(B)), lambda k: oc.gemm_soma(k(A), k(B), k(X)), lambda k: oc.gemm_relu2_back(k(A), B, k(X)), lambda k: oc.transpoe(k(A)),
              lambda k: oc.transpoe2(k(A), k(B)), lambda k: oc.quant(k(c)), lambda k: oc.soma(k(A), B), lambda k: oc.relu2(k(A)), lambda k: oc.rms(k(A)),
              lambda k: oc.rms_back(k(X), k(y), cache), lambda k: oc.softmax_ce(k(c), alvo), lambda k: oc.momento(k(c), k(novo(X))), lambda k: oc.max_linha(k(A)),
              lambda k: oc.momento_peso(k(c), k(novo(X)), k(novo(W)), k(novo(B)), 4, True), lambda k: oc.peso(k(novo(W)), k(X), k(novo(B)), 4, True),
              lambda k: oc.atencao(k(qkv), *forma), lambda k: oc.atencao_back(k(go), k(qkv), P, *forma), lambda k: oc.atencao_quant(k(qkv), *forma)):
        compara("list", casos.plano(f(list)), casos.plano(f(tuple)))
    with pytest.raises(ErroJatai, match="argument 'A' is not a valid block tensor"):
        oc.gemm([A[0], A[1][:1]], B)


def _alguns(oc, A, B, c, qkv, forma):
    """One launch of each way a launch is made: a product, one with external maxima, an attention, an operator of the general launcher."""
    return [oc.gemm(A, B), oc.gemm(A, B, cru=True, RA=oc.max_linha(A), RB=oc.max_linha(B)), *oc.atencao_quant(qkv, *forma), oc.quant(c)]


@pytest.mark.parametrize("perfil", [False, True])
def test_registro_de_fora(amb, perfil):
    """The launcher keeps to the registry's protocol: registra before and depois after every launch of a registry that is not the plain one -
    one derived from it, and one that has only the reference's methods - with the launch id that registra gave."""
    from jatai_b200 import registro
    ops, oc0, reg0 = amb
    G = casos.Gen(61, 32)
    A, B = para_gpu(G.bloco(256, 256)), para_gpu(G.bloco(256, 256))
    c = oc0.gemm(A, B, cru=True)
    qkv, go, forma = _problema(32, 2, 64, 2, 64)
    ref = _alguns(oc0, A, B, c, qkv, forma)

    class Derivado(registro.Registro):
        def registra(self, op, ent, forma):
            self.visto = getattr(self, "visto", []) + [(op, sorted(ent), tuple(forma))]
            return super().registra(op, ent, forma)

        def depois(self, kid, rc):
            self.fim = getattr(self, "fim", []) + [(kid, rc)]
            super().depois(kid, rc)

    class Minimo:
        """What jatai_cuda/registro.py:66-116 has of it."""
        vigiar, lib = False, None

        def __init__(self):
            self.perfil, self.lancamentos, self.visto, self.fim = perfil, [], [], []

        def onde(self):
            return "-"

        def registra(self, op, ent, forma):
            self.visto.append((op, sorted(ent), tuple(forma)))
            return 100 + len(self.visto) - 1

        def depois(self, kid, rc):
            self.fim.append((kid, rc))

        def novo_passo(self, p):
            pass

        def confere_bloco(self, nome, t):
            pass

        def exige(self, c, msg):
            assert c, msg

    esperado = [("gemm", ["A", "B", "EA", "EB"], (256, 256)), ("max_linha", ["E"], (256, 1)), ("max_linha", ["E"], (256, 1)),
                ("gemm_cru", ["A", "B", "EA", "EB"], (256, 256)), ("atencao_quant", ["qkv", "qkvE"], (128, 128)), ("quant", ["acc", "e"], (256, 256))]
    for reg in (Derivado(tempfile.mkdtemp(), "d", perfil=perfil, eco=False, salvar=False), Minimo()):
        oc = ops.OpsCuda(reg)
        reg.novo_passo(0)
        compara(type(reg).__name__, casos.plano(_alguns(oc, A, B, c, qkv, forma)), casos.plano(ref))
        assert reg.visto == esperado
        k0 = 0 if isinstance(reg, registro.Registro) else 100
        assert reg.fim == [(k0 + i, 0) for i in range(6)]
    if perfil:
        plano = registro.Registro(tempfile.mkdtemp(), "p", perfil=True, eco=False, salvar=False)
        oc = ops.OpsCuda(plano)
        plano.novo_passo(0)
        _alguns(oc, A, B, c, qkv, forma)
        plano.fim_passo()
        assert sorted(plano.tempos) == sorted({e[0] for e in esperado}) and all(v > 0 for v in plano.tempos.values())


def _tok_fora(oc):
    W = para_gpu(casos.Gen(3, 32).bloco(256, 128))
    return W, torch.full((64,), 300, dtype=torch.int32, device="cuda")


def test_registro_de_erros_limpo_antes_de_lido(amb):
    """The record is cleared in the order of a stream and read after that: a sentinel of the step before does not come back."""
    ops, oc, reg = amb
    reg.vigiar = False
    W, tok = _tok_fora(oc)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    try:
        with torch.cuda.stream(s):
            oc.lib.jt_stream(s.cuda_stream)
            oc.embed(W, tok)
            torch.cuda.synchronize()
            torch.cuda._sleep(200_000_000)
            reg.novo_passo(1)
            reg.confere_device()
    finally:
        oc.lib.jt_stream(None)


@pytest.mark.parametrize("n", [1, 20])
def test_registro_de_erros_limpo_antes_de_outra_corrente(amb, n):
    """A clearing that is still queued on one stream does not wipe out what a launch on another one finds afterwards, whichever of n it is."""
    from jatai_b200.registro import ErroJatai
    ops, oc, reg = amb
    reg.vigiar = False
    W, tok = _tok_fora(oc)
    bom = torch.zeros_like(tok)
    a, outras = torch.cuda.Stream(), [torch.cuda.Stream() for _ in range(n)]
    torch.cuda.synchronize()
    try:
        with torch.cuda.stream(a):
            oc.lib.jt_stream(a.cuda_stream)
            torch.cuda._sleep(200_000_000)
            reg.novo_passo(1)
        for i, b in enumerate(outras):
            with torch.cuda.stream(b):
                oc.lib.jt_stream(b.cuda_stream)
                oc.embed(W, tok if i == n - 1 else bom)
        oc.lib.jt_stream(a.cuda_stream)
        with torch.cuda.stream(a):
            oc.embed(W, bom)
        torch.cuda.synchronize()
        with pytest.raises(ErroJatai, match="outside the vocabulary"):
            reg.confere_device()
    finally:
        oc.lib.jt_stream(None)


def test_registro_de_erros_limpo_antes_de_uma_repeticao(amb):
    """The same for a recorded step that is replayed on a stream which is not the library's."""
    from jatai_b200 import modelo
    from jatai_b200.registro import ErroJatai
    ops, oc, reg = amb
    reg.vigiar = False
    m = modelo.Modelo(256, 128, 2, 256, 1, 0, "cuda", oc, reg)
    x = torch.randint(0, 256, (2, 64), device="cuda")
    m.passo(x, x, k_lr=4)
    g = modelo.PassoGravado(m, 2, 64, 4)
    ruim = x.clone()
    ruim[1, 17] = 300
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    try:
        with torch.cuda.stream(a):
            oc.lib.jt_stream(a.cuda_stream)
            torch.cuda._sleep(200_000_000)
            reg.novo_passo(1)
        with torch.cuda.stream(b):
            g(ruim, x)
        torch.cuda.synchronize()
        with pytest.raises(ErroJatai, match="forward / embedding"):
            reg.confere_device()
    finally:
        oc.lib.jt_stream(None)


@pytest.mark.parametrize("M,N,K,cru", [(512, 512, 2048, True), (2048, 512, 2048, True), (128, 128, 4096, True), (1024, 1024, 8192, True), (2048, 512, 1536, False)])
def test_ao_lado_mesmos_bits(amb, M, N, K, cru):
    """jt_stream_ao_lado changes how a product is cut (clusters, 64-wide tiles, K ranges), not what it gives; jt_stream takes it back."""
    ops, oc, reg = amb
    ops.define_blk(32)
    g = torch.Generator(device="cuda").manual_seed(M + K)
    ints = lambda a, b, forma: torch.randint(a, b + 1, forma, generator=g, device="cuda", dtype=torch.int32).to(torch.int8)
    A, B = ((ints(-127, 127, (R, K)), ints(-12, -4, (R, K // 32))) for R in (M, N))
    reg.novo_passo(0)
    try:
        quer = oc.gemm(A, B, cru=cru)
        oc.lib.jt_stream_ao_lado(None)
        tem = oc.gemm(A, B, cru=cru)
        oc.lib.jt_stream(None)
        outra = oc.gemm(A, B, cru=cru)
    finally:
        oc.lib.jt_stream(None)
    for x, y, z in zip(quer, tem, outra):
        assert torch.equal(x, y) and torch.equal(x, z)
