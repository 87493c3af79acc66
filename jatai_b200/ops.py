"""Operator API of the integer training step on B200: the host-side mirror of jatai_cuda/ops.py.

`OpsCuda(reg)` has the method names, argument meaning, return values and error behaviour of the reference's
`OpsCuda` (jatai_cuda/ops.py:294-515): every method checks its inputs through the registry, allocates its
outputs as torch tensors, registers the launch (-> kid) and calls one `jt_*` entry point of
libjatai_b200.so with raw device pointers.  A model written against the reference operator API
(`modelo.py`) therefore runs unchanged on these kernels.

Formats: Bloco = (m int8 [R,C], E int8 [R,C/BLK]), value m * 2^E, zero block E = -127;
         Cru = (acc int32 [R,C], e int16 [R,C]).

Module-level names kept from the reference: BLK, E_ZERO, GA, ATENCAO_LIMITE, g_rms, OpsCuda (class attribute
lib_global).  New: define_blk (the reference's block length is a compile-time 128; here 32 is native and 128
is the compatibility format), and optional arguments for the data-parallel step (RA / RB of `gemm`, log2M of
`softmax_ce`).  There is no CPU path: constructing OpsCuda without the compiled library, or calling it with
CPU tensors, raises.
"""
import ctypes
import functools
import math
import os

import torch

from .registro import Registro

BLK = 32
E_ZERO = -127
GA = 4                     # guard bits of q/k/v/dO aligned inside a head (reference ops.py:20)
ATENCAO_LIMITE = False     # attention backward: shifts from upper bounds instead of exact maxima (ops.py:21-23)
AQUI = os.path.dirname(os.path.abspath(__file__))
BIBLIOTECA = os.path.join(AQUI, "libjatai_b200.so")

_INT_FUNCS = ("jt_gemm", "jt_gemm_f", "jt_gemm_ext", "jt_max_linha", "jt_quant", "jt_soma", "jt_relu2", "jt_relu2_back",
              "jt_momento", "jt_peso", "jt_momento_peso", "jt_transpoe", "jt_transpoe2", "jt_embed", "jt_um_quente", "jt_rms", "jt_rms_back", "jt_rms_back_soma", "jt_atencao",
              "jt_atencao_back", "jt_softmax_ce", "jt_erro_le", "jt_erro_limpa", "jt_sincroniza", "jt_para16", "jt_para8",
              "jt_soma16", "jt_res_estocastico", "jt_blk", "jt_blk_atual", "jt_gemm_via", "jt_gemm_tn", "jt_gemm_somas", "jt_atencao_back_fixo", "jt_atencao_via", "jt_atencao_quant", "jt_atencao_back_quant",
              "jt_espera_limite", "jt_teste_espera", "jt_transpoe2_max", "jt_pdl", "jt_gemm_sem_cargas", "jt_gemm_ws", "jt_perda", "jt_atencao_ws", "jt_atencao_back_ws", "jt_espaco_limite", "jt_espaco_libera")


def g_rms(D):
    """(guard bits of RMSNorm forward, of its backward) for D columns; reference ops.py:28-30."""
    return _g_rms(D, BLK)


@functools.lru_cache(maxsize=64)
def _g_rms(D, blk):
    nb = D // blk
    return 2 * ((8 - int(math.log2(nb))) // 2), 14 - int(math.log2(D))


def carrega_biblioteca(caminho=None):
    """dlopen the C-ABI library and declare the return types.  Raises if it has not been built."""
    caminho = caminho or BIBLIOTECA
    if not os.path.exists(caminho):
        raise RuntimeError(f"{caminho} not found: build it with `python -m jatai_b200.build` (needs nvcc, sm_100a)")
    lib = ctypes.CDLL(caminho)
    lib.jt_stream.argtypes = [ctypes.c_void_p]
    lib.jt_stream.restype = None
    lib.jt_erro_le.argtypes = [ctypes.c_void_p]
    for f in _INT_FUNCS:
        if hasattr(lib, f):
            getattr(lib, f).restype = ctypes.c_int
    if hasattr(lib, "jt_stream_ao_lado"):
        lib.jt_stream_ao_lado.argtypes = [ctypes.c_void_p]
        lib.jt_stream_ao_lado.restype = None
    if hasattr(lib, "jt_gemm_ws_bytes"):
        lib.jt_gemm_ws_bytes.restype = ctypes.c_longlong
        lib.jt_atencao_ws_bytes.restype = ctypes.c_longlong
        lib.jt_espaco_limite.argtypes = [ctypes.c_longlong]
        lib.jt_stream_atual.restype = ctypes.c_void_p
    return lib


def carrega_nativo():
    """The native half of the launcher.  Raises if it has not been built, or was built against another PyTorch or Python."""
    from . import build
    como = "build it with `python -m jatai_b200.build`"
    try:
        from . import _nativo
    except ImportError as e:
        raise RuntimeError(f"{build.SAIDA_NATIVO} does not load ({e}): {como}") from e
    if _nativo.MARCA != build._marca():
        raise RuntimeError(f"{build.SAIDA_NATIVO} was built against {_nativo.MARCA}, this is {build._marca()}: {como}")
    return _nativo


def define_blk(blk, lib=None):
    """Select the exponent block length (32 or 128) for this module and for the library."""
    global BLK
    if blk not in (32, 128):
        raise ValueError("block length must be 32 or 128")
    BLK = blk
    lib = lib or getattr(OpsCuda, "lib_global", None)
    if lib is not None and hasattr(lib, "jt_blk"):
        if lib.jt_blk(blk) != 0:
            raise RuntimeError(f"library refused block length {blk}")
    elif lib is not None and blk != 128:
        raise RuntimeError("this library has a fixed block length of 128")


class OpsCuda:
    """Launcher of the CUDA kernels; interface of the reference's OpsCuda (ops.py:294-515)."""
    nome = "cuda"
    lib_global = None

    def __init__(self, reg, biblioteca=None):
        if not torch.cuda.is_available():
            raise RuntimeError("OpsCuda needs a CUDA device; there is no CPU implementation in this package")
        self.reg = reg
        self.lib = carrega_biblioteca(biblioteca)
        reg.lib = self.lib
        self.lib.jt_erro_limpa()
        OpsCuda.lib_global = self.lib
        if hasattr(self.lib, "jt_blk"):
            if self.lib.jt_blk(BLK) != 0:
                raise RuntimeError(f"library refused block length {BLK}")
        elif BLK != 128:
            raise RuntimeError("this library has a fixed block length of 128; call ops.define_blk(128) first")
        if hasattr(self.lib, "jt_pdl"):                           # programmatic dependent launches: JT_PDL=0 switches them off
            self.lib.jt_pdl(0 if os.environ.get("JT_PDL", "1") == "0" else 1)
        self._nat = carrega_nativo()
        self._fn = {}                                             # address of every entry point used so far
        self._ws = self._endereco("jt_gemm_ws_bytes"), self._endereco("jt_stream_atual")
        self._ws_gemm = self._endereco("jt_gemm_ws"), self._endereco("jt_gemm_ext")
        self._ws_at = self._endereco("jt_atencao_ws_bytes"), self._endereco("jt_stream_atual")
        self._at_frente = self._endereco("jt_atencao_ws"), self._endereco("jt_atencao")
        self._at_tras = self._endereco("jt_atencao_back_ws"), self._endereco("jt_atencao_back")
        # a library with only the reference's entry points: the fused extras read as absent, callers fall back to the separate operations
        for metodo, fn in (("transpoe2", "jt_transpoe2"), ("momento_peso", "jt_momento_peso"), ("rms_back_soma", "jt_rms_back_soma"),
                           ("max_linha", "jt_max_linha"), ("atencao_quant", "jt_atencao_quant"), ("atencao_back_quant", "jt_atencao_back_quant"),
                           ("perda", "jt_perda")):
            if not hasattr(self.lib, fn):
                setattr(self, metodo, None)

    # ------------------------------------------------------------------ plumbing
    # Checks, output allocation and the call itself run in the native module (csrc/nativo.cpp); what is wrong with an argument it leaves to
    # the Python checks of the registry, which name it.
    def _endereco(self, fn):
        e = self._fn.get(fn)
        if e is None:
            e = self._fn[fn] = ctypes.cast(getattr(self.lib, fn), ctypes.c_void_p).value if hasattr(self.lib, fn) else 0
        return e

    def _lanca(self, op, fn, tensores, inteiros, nomes, forma):
        """Registers the launch and calls the entry point: pointers of `tensores` (None = null), then `inteiros`, then the launch id.
        `nomes` name the first tensors in the launch record (None leaves one out)."""
        reg, f = self.reg, self._fn.get(fn) or self._endereco(fn)
        # The native calls append to the launch list of a plain Registro that times nothing; of any other registry they call registra and depois.
        if reg.perfil or reg.__class__ is not Registro:
            self._nat.lanca(f, reg, op, reg.onde(), nomes, tensores, inteiros, forma)
            return
        r = self._nat.lanca(f, reg.lancamentos, op, reg.onde(), nomes, tensores, inteiros, forma)
        if r is not None:
            reg.depois(*r)
        elif reg.vigiar:
            reg.depois(len(reg.lancamentos) - 1, 0)

    def _blocos(self, nomes, *tensores):
        """(R1, C1, R2, C2, ...) of valid block tensors; raises, naming the argument, otherwise."""
        d = self._nat.blocos(BLK, *tensores)
        if d is None:
            for n, t in zip(nomes, tensores):
                self.reg.confere_bloco(n, t)
            d = self._nat.blocos(BLK, *(tuple(t) for t in tensores))      # a pair may come in another container than a tuple
            if d is None:
                self.reg.falha(f"{nomes}: not block tensors (mantissa and exponent tensors on the GPU)")
        return d

    def _cru(self, nome, t):
        d = self._nat.cru(t)
        if d is None:
            self.reg.confere_cru(nome, t)
            d = self._nat.cru(tuple(t))
            if d is None:
                self.reg.falha(f"argument '{nome}' is not a raw tensor of two dimensions")
        return d

    # ------------------------------------------------------------------ GEMM family
    def _gemm(self, op, modo, A, B, X=None, duas=False, RA=None, RB=None):
        reg, nat = self.reg, self._nat
        if RA is None and RB is None:
            alheio = reg.perfil or reg.__class__ is not Registro
            r = nat.gemm(*self._ws, *self._ws_gemm, BLK, reg if alheio else reg.lancamentos, op, reg.onde(), modo, A, B, X, duas)
            if r.__class__ is tuple:
                if reg.vigiar and not alheio:
                    reg.depois(len(reg.lancamentos) - 1, 0)
                return r
            if r is not None:
                reg.depois(len(reg.lancamentos) - 1, r)
        # with external row maxima, for a library with only the reference's entry points - and what is wrong with an argument
        if X is None:
            M, K, N, Kb = self._blocos(("A", "B"), A, B)
        else:
            M, K, N, Kb, Mx, Nx = self._blocos(("A", "B", "X"), A, B, X)
        (a, ea), (b, eb) = A, B
        if Kb != K:
            reg.falha(f"{op}: K differs, A {tuple(a.shape)} x B {tuple(b.shape)}")
        if M % 64 or N % 128 or K % BLK:
            reg.falha(f"{op}: M must be a multiple of 64, N of 128, K of {BLK} (M={M}, N={N}, K={K})")
        if X is None:
            x, nomes = (None, None), ("A", "EA", "B", "EB")
        else:
            if Mx != M or Nx != N:
                reg.falha(f"{op}: X has shape {(Mx, Nx)}, expected {(M, N)}")
            x, nomes = X, ("A", "EA", "B", "EB", None, None, None, None, "X", "XE")
        for nome, r, n in (("RA", RA, M), ("RB", RB, N)):
            if r is not None:
                reg.exige(r.dtype == torch.int8 and r.is_cuda and r.is_contiguous() and r.numel() == n,
                          f"{op}: {nome} must be a contiguous int8 CUDA tensor with {n} elements")
        nada = (None, None)
        Cb, Cr = (nada, nat.novo_cru(a, M, N)) if modo == 1 else (nat.novo_bloco(a, M, N, BLK), nada)
        C2 = nat.novo_bloco(a, M, N, BLK) if duas else nada
        t = (a, ea, b, eb, *Cb, *Cr, *x, *C2)
        ws = nat.espaco_gemm(*self._ws, a, M, N, K, modo)
        if ws is not None:
            self._lanca(op, "jt_gemm_ws", (*t, RA, RB, ws), (M, N, K, modo), nomes, (M, N))
        elif self._endereco("jt_gemm_ext"):
            self._lanca(op, "jt_gemm_ext", (*t, RA, RB), (M, N, K, modo), nomes, (M, N))
        else:       # a library with only the reference's entry points (no external row maxima)
            reg.exige(RA is None and RB is None, f"{op}: this library has no jt_gemm_ext (RA / RB unsupported)")
            self._lanca(op, "jt_gemm_f", t, (M, N, K, modo), nomes, (M, N))
        if modo == 1:
            return Cr
        return (Cb, C2) if duas else Cb

    def gemm(self, A, B, cru=False, RA=None, RB=None):
        """C = A . B^T, operands blocked along K.  cru=True: raw int32 accumulators + int16 exponents.
        RA / RB (optional int8 vectors): row-maximum exponents to align to instead of the operands' own
        (a data-parallel rank passes the maxima over all ranks)."""
        return self._gemm("gemm_cru" if cru else "gemm", 1 if cru else 0, A, B, RA=RA, RB=RB)

    def gemm_soma(self, A, B, X):
        return self._gemm("gemm_soma", 2, A, B, X=X)

    def gemm_relu2(self, A, B):
        return self._gemm("gemm_relu2", 3, A, B, duas=True)

    def gemm_relu2_back(self, A, B, Hh):
        return self._gemm("gemm_relu2_back", 4, A, B, X=Hh)

    def max_linha(self, X):
        """Row-maximum exponents (int8 [R]) of a block tensor: the RA / RB a GEMM derives from its operand."""
        self._blocos(("X",), X)
        E = X[1]
        R = torch.empty(E.shape[0], dtype=torch.int8, device=E.device)
        self._lanca("max_linha", "jt_max_linha", (E, R), (E.shape[0], E.shape[1]), ("E",), (E.shape[0], 1))
        return R

    def transpoe(self, X):
        R, C = self._blocos(("X",), X)
        m, E = X
        if R % 128 or C % 64:
            self.reg.falha(f"transpoe: rows {R} must be a multiple of 128 and columns {C} of 64")
        Y = self._nat.novo_bloco(m, C, R, BLK)
        self._lanca("transpoe", "jt_transpoe", (m, E, *Y), (R, C), ("X", "EX"), (C, R))
        return Y

    def transpoe2(self, X1, X2):
        """(transpoe(X1), transpoe(X2)) for two block tensors with the same number of rows, in one launch (an addition of
        this library; the two operands of a weight-gradient GEMM)."""
        R, C1, R2, C2 = self._blocos(("X1", "X2"), X1, X2)
        if R2 != R:
            self.reg.falha(f"transpoe2: row counts differ ({R} and {R2})")
        if R % 128 or C1 % 64 or C2 % 64:
            self.reg.falha(f"transpoe2: rows {R} must be a multiple of 128 and columns {C1}, {C2} of 64")
        m = X1[0]
        Y1, Y2 = self._nat.novo_bloco(m, C1, R, BLK), self._nat.novo_bloco(m, C2, R, BLK)
        self._lanca("transpoe2", "jt_transpoe2", (*X1, *Y1, *X2, *Y2), (C1, C2, R), ("X1", "EX1", None, None, "X2", "EX2"), (C1 + C2, R))
        return Y1, Y2

    def transpoe2_max(self, X1, X2, R1, R2):
        """transpoe2, and the row maxima of both results (max_linha) written into R1 [C1] / R2 [C2] - int8 views the caller has
        pre-set to -128 (data parallel: slices of the buffer of its MAX collective).  None where this library or these
        shapes do not offer it (the caller then uses transpoe2 and max_linha)."""
        R, C1 = X1[0].shape
        C2 = X2[0].shape[1]
        if BLK != 32 or C1 % 256 or C2 % 256 or R % 128 or X2[0].shape[0] != R or not hasattr(self.lib, "jt_transpoe2_max"):
            return None
        self._blocos(("X1", "X2"), X1, X2)
        self.reg.exige(R1.numel() == C1 and R2.numel() == C2 and R1.dtype == torch.int8 and R2.dtype == torch.int8 and
                       R1.data_ptr() % 4 == 0 and R2.data_ptr() % 4 == 0, "transpoe2_max: row-maximum views of the wrong size, type or alignment")
        m = X1[0]
        Y1, Y2 = self._nat.novo_bloco(m, C1, R, BLK), self._nat.novo_bloco(m, C2, R, BLK)
        self._lanca("transpoe2", "jt_transpoe2_max", (*X1, *Y1, *X2, *Y2, R1, R2), (C1, C2, R), ("X1", "EX1", None, None, "X2", "EX2"), (C1 + C2, R))
        return Y1, Y2

    # ------------------------------------------------------------------ block elementwise
    def quant(self, Cc):
        R, C = self._cru("C", Cc)
        if C % BLK:
            self.reg.falha(f"quant: {C} columns is not a multiple of {BLK}")
        Y = self._nat.novo_bloco(Cc[0], R, C, BLK)
        self._lanca("quant", "jt_quant", (*Cc, *Y), (R * C // BLK,), ("acc", "e"), (R, C))
        return Y

    def _elemento(self, op, fn, X, nomes):
        R, C = self._blocos(nomes[:1], X)
        Z = self._nat.novo_bloco(X[0], R, C, BLK)
        self._lanca(op, fn, (*X, *Z), (R * C // BLK,), nomes, (R, C))
        return Z

    def _elemento2(self, op, fn, X, Y, nomes):
        R, C, R2, C2 = self._blocos(nomes[::2], X, Y)
        if R2 != R or C2 != C:
            self.reg.falha(f"{op}: '{nomes[2]}' has shape {(R2, C2)}, expected {(R, C)}")
        Z = self._nat.novo_bloco(X[0], R, C, BLK)
        self._lanca(op, fn, (*X, *Y, *Z), (R * C // BLK,), nomes, (R, C))
        return Z

    def soma(self, X, Y):
        return self._elemento2("soma", "jt_soma", X, Y, ("x", "xE", "y", "yE"))

    def relu2(self, Hh):
        return self._elemento("relu2", "jt_relu2", Hh, ("h", "hE"))

    def relu2_back(self, Gg, Hh):
        return self._elemento2("relu2_back", "jt_relu2_back", Gg, Hh, ("g", "gE", "h", "hE"))

    def embed(self, W, tok):
        V, D = self._blocos(("W",), W)
        M = tok.numel()
        X = self._nat.novo_bloco(W[0], M, D, BLK)
        self._lanca("embed", "jt_embed", (*W, tok, *X), (M, D, V), ("W", None, "tok"), (M, D))
        return X

    def um_quente(self, tok, V):
        M = tok.numel()
        U = self._nat.novo_bloco(tok, M, V, BLK)
        self._lanca("um_quente", "jt_um_quente", (tok, *U), (M, V), ("tok",), (M, V))
        return U

    # ------------------------------------------------------------------ RMSNorm
    def rms(self, X):
        M, D = self._blocos(("x",), X)
        if D > 2048 or D & (D - 1):
            self.reg.falha(f"rms: D={D} must be a power of two <= 2048")
        nat, m = self._nat, X[0]
        Y, r, emax = nat.novo_bloco(m, M, D, BLK), nat.novo(m, "i4", M), nat.novo(m, "i4", M)
        self._lanca("rms", "jt_rms", (*X, *Y, r, emax), (M, D, D.bit_length() - 1, g_rms(D)[0]), ("x", "xE"), (M, D))
        return Y, (r, emax)

    def rms_back(self, Gg, Y, cache):
        M, D, _, _ = self._blocos(("g", "y"), Gg, Y)
        O = self._nat.novo_bloco(Gg[0], M, D, BLK)
        self._lanca("rms_back", "jt_rms_back", (*Gg, *Y, *cache, *O), (M, D, D.bit_length() - 1, *g_rms(D)), ("g", "gE", "y", "yE", "r", "emax"), (M, D))
        return O

    def rms_back_soma(self, X, Gg, Y, cache):
        """soma(X, rms_back(Gg, Y, cache)) in one launch (an addition of this library; same results)."""
        Mx, Dx, M, D, _, _ = self._blocos(("x", "g", "y"), X, Gg, Y)
        if Mx != M or Dx != D:
            self.reg.falha(f"rms_back_soma: x has shape {(Mx, Dx)}, expected {(M, D)}")
        O = self._nat.novo_bloco(Gg[0], M, D, BLK)
        self._lanca("rms_back_soma", "jt_rms_back_soma", (*Gg, *Y, *cache, *X, *O), (M, D, D.bit_length() - 1, *g_rms(D)),
                    ("g", "gE", "y", "yE", "r", "emax", "x", "xE"), (M, D))
        return O

    # ------------------------------------------------------------------ attention
    def _atencao_nativa(self, op, entradas, blocos, QKV, GO, P, Bt, T, H):
        """The call in one piece, workspace included (`entradas`: the entry points with one and, raw outputs only, without), or None: block
        outputs without a workspace, a library with only the reference's entry points - and what is wrong with an argument."""
        reg = self.reg
        alheio = reg.perfil or reg.__class__ is not Registro
        r = self._nat.atencao(*self._ws_at, *entradas, BLK, reg if alheio else reg.lancamentos, op, reg.onde(), QKV, GO, P, Bt, T, H, GA,
                              int(ATENCAO_LIMITE), blocos)
        if r.__class__ is int:
            reg.depois(len(reg.lancamentos) - 1, r)
        elif r is not None and reg.vigiar and not alheio:
            reg.depois(len(reg.lancamentos) - 1, 0)
        return r

    def atencao(self, QKV, Bt, T, H):
        r = self._atencao_nativa("atencao", self._at_frente, False, QKV, None, None, Bt, T, H)
        if r is not None:
            return r
        M, D3 = self._blocos(("qkv",), QKV)
        D = D3 // 3
        hd = D // H
        if M != Bt * T or H * hd != D or hd not in (4, 16, 64) or T % 32 or T > 1024:
            self.reg.falha(f"atencao: rows {M} (= Bt*T = {Bt * T}), head dim {hd} (4, 16 or 64), T={T} (multiple of 32, <= 1024)")
        o, P = self._nat.novo_cru(QKV[0], M, D), self._nat.novo(QKV[0], "u1", Bt * H, T, T)
        self._lanca("atencao", "jt_atencao", (*QKV, *o, P), (Bt, T, H, D, GA), ("qkv", "qkvE"), (M, D))
        return o, P

    def atencao_back(self, GO, QKV, P, Bt, T, H):
        r = self._atencao_nativa("atencao_back", self._at_tras, False, QKV, GO, P, Bt, T, H)
        if r is not None:
            return r
        M, D, _, _ = self._blocos(("go", "qkv"), GO, QKV)
        g = self._nat.novo_cru(QKV[0], Bt * T, 3 * D)
        self._lanca("atencao_back", "jt_atencao_back", (*GO, *QKV, P, *g), (Bt, T, H, D, GA, int(ATENCAO_LIMITE)), ("go", "goE", "qkv", "qkvE", "P"),
                    (Bt * T, 3 * D))
        return g

    def _atencao_fundida(self, T, H, D):
        """Whether the library quantises the attention outputs in its own output stage for this shape (else: two launches)."""
        return BLK == 32 and D == 64 * H and T % 32 == 0 and T <= 1024 and GA <= 4

    def atencao_quant(self, QKV, Bt, T, H):
        """(quant(O), P) of atencao(QKV, Bt, T, H): one launch where the library offers it and its workspace is to be had (an addition of
        this library; same results)."""
        D = QKV[0].shape[1] // 3
        if self._atencao_fundida(T, H, D):
            r = self._atencao_nativa("atencao_quant", self._at_frente, True, QKV, None, None, Bt, T, H)
            if r is not None:
                return r
        oc, P = self.atencao(QKV, Bt, T, H)
        return self.quant(oc), P

    def atencao_back_quant(self, GO, QKV, P, Bt, T, H):
        """quant(atencao_back(GO, QKV, P, Bt, T, H)): one launch sequence without the raw intermediate where the library offers it and its
        workspace is to be had."""
        if self._atencao_fundida(T, H, GO[0].shape[1]):
            r = self._atencao_nativa("atencao_back_quant", self._at_tras, True, QKV, GO, P, Bt, T, H)
            if r is not None:
                return r
        return self.quant(self.atencao_back(GO, QKV, P, Bt, T, H))

    # ------------------------------------------------------------------ loss and optimiser
    def softmax_ce(self, L, alvo, log2M=None):
        """log2M: log2 of the token count the gradient is averaged over (default: rows of L; a data-parallel
        rank passes the global count)."""
        M, V = self._cru("logits", L)
        if log2M is None:
            if M & (M - 1):
                self.reg.falha(f"softmax_ce: {M} rows is not a power of two")
            log2M = M.bit_length() - 1
        if V > 2048 or V % BLK:
            self.reg.falha(f"softmax_ce: V={V}")
        nat, acc = self._nat, L[0]
        g, d, s = nat.novo_bloco(acc, M, V, BLK), nat.novo(acc, "i4", M), nat.novo(acc, "i4", M)
        self._lanca("softmax_ce", "jt_softmax_ce", (*L, alvo, *g, d, s), (M, V, log2M), ("acc", "e", "alvo"), (M, V))
        return g, d, s

    def perda(self, d_alvo, soma):
        """The loss report of softmax_ce's outputs, mean over the tokens of d_alvo / 256 + log(soma / 4096) in double precision (an addition of
        this library: the terms in one launch, then the mean)."""
        p = torch.empty(d_alvo.numel(), dtype=torch.float64, device=d_alvo.device)
        self._lanca("perda", "jt_perda", (d_alvo, soma, p), (d_alvo.numel(),), ("d_alvo", "soma"), (d_alvo.numel(), 1))
        return p.mean()

    def momento(self, Gc, Mom):
        d = self._cru("grad", Gc)
        R, C = self._blocos(("momento",), Mom)
        if d != (R, C):
            self.reg.falha("momento: gradient and momentum shapes differ")
        self._lanca("momento", "jt_momento", (*Gc, *Mom), (R * C // BLK,), ("g", "ge"), (R, C))
        return Mom

    def momento_peso(self, Gc, Mom, W, R, k, ef):
        """momento(Gc, Mom) followed by peso(W, Mom, R, k, ef) in one launch (an addition of this library; same results).
        Returns (Mom, W, R), all updated in place."""
        d = self._cru("grad", Gc)
        Rw, Cw, Rm, Cm, _, _ = self._blocos(("W", "momento", "residuo"), W, Mom, R)
        if not d == (Rw, Cw) == (Rm, Cm):
            self.reg.falha("momento_peso: gradient, momentum and weight shapes differ")
        self._lanca("momento_peso", "jt_momento_peso", (*Gc, *Mom, *W, *R), (k, int(ef), Rw * Cw // BLK), ("g", "ge"), (Rw, Cw))
        return Mom, W, R

    def peso(self, W, Mom, R, k, ef):
        Rw, Cw, _, _, _, _ = self._blocos(("W", "momento", "residuo"), W, Mom, R)
        self._lanca("peso", "jt_peso", (*W, *Mom, *R), (k, int(ef), Rw * Cw // BLK), (), (Rw, Cw))
        return W, R
