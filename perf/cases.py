"""What the framework is timed on: whole training steps, the evaluation pass, and the operators that a model is written with.

Every case goes through the public entry points: `modelo.Modelo` / `modelo.PassoGravado` for steps, `ops.OpsCuda` for operators.

kind     what a pass is
passo    one training step: "gravado" = replayed from its recording (how training runs), "eager" = launched operator by operator
         (a run's first step, its statistics and profile steps, `--eager`), "avalia" = the forward pass alone (validation)
linear   one linear layer: Y = X W^T, dX = dY W, dW = dY^T X, the transpositions included
gemm     one forward product with its fused output stage, on any size that the operator takes
atencao  attention forward and backward with the quantisation of both results
blocos   the bandwidth operators of a layer, the loss and the optimiser on one tensor size

Ranges: head dimension 4, 16 or 64; block length 32 or 128; T a multiple of 32 up to 1024; rows from 64 to 16384; columns from 128 to
4096 (RMSNorm: powers of two up to 2048).
"""
import functools
import math
import tempfile

import torch

from jatai_b200 import modelo, ops, registro

V = 256                # byte vocabulary
K_LR = 4               # learning rate 2^-4
N_LOTES = 8            # batches that a step's program cycles through
MAX_SAIDAS = 64        # most tensors handed back by one pass
MAX_ESCORES = 1 << 28  # Bt * H * T * T of the largest attention


def listed():
    return [
        # a toy model: the smallest step, all launches (the size of the repository's own model tests)
        dict(name="passo_minimo", kind="passo", modo="gravado", blk=32, D=128, H=2, FF=256, L=2, T=64, Bt=2),
        # the ordinary training step: 12 layers, 2048 byte tokens (the benchmark's default)
        dict(name="passo_12_camadas", kind="passo", modo="gravado", blk=32, D=512, H=8, FF=2048, L=12, T=256, Bt=8),
        # the size and block length of existing checkpoints: 64 heads of 4, block 128
        dict(name="passo_bloco_128", kind="passo", modo="gravado", blk=128, D=256, H=64, FF=1024, L=12, T=128, Bt=16),
        # the widest and longest configuration, 16384 tokens; 4 of its 24 (identical) layers
        dict(name="passo_largo", kind="passo", modo="gravado", blk=32, D=1024, H=16, FF=4096, L=4, T=1024, Bt=16),
        # validation between the steps of a training run: 8 sequences, forward only, launched operator by operator
        dict(name="avalia_12_camadas", kind="passo", modo="avalia", blk=32, D=512, H=8, FF=2048, L=12, T=256, Bt=8),
        # a training step that is not recorded, on a small model
        dict(name="passo_eager", kind="passo", modo="eager", blk=32, D=256, H=4, FF=1024, L=6, T=128, Bt=4),
        # one linear layer, forward and backward: of the 12-layer model, and the largest of the benchmark's sweep
        dict(name="linear_512", kind="linear", blk=32, M=2048, N=512, K=512),
        dict(name="linear_4096", kind="linear", blk=32, M=16384, N=4096, K=4096),
        # rows that fill no 128-row tile and a reduced dimension that fills no 128-byte piece: an odd batch
        dict(name="gemm_irregular", kind="gemm", op="soma", blk=32, M=1984, N=1408, K=1056),
        # sequences cut at a length that is no multiple of 64
        dict(name="atencao_T416", kind="atencao", blk=32, Bt=4, T=416, H=8, hd=64),
        # many small heads, beyond the short sequences
        dict(name="atencao_hd16_T288", kind="atencao", blk=32, Bt=8, T=288, H=16, hd=16),
        # the bandwidth operators at 16384 tokens
        dict(name="blocos_16384x1024", kind="blocos", blk=32, R=16384, C=1024),
    ]


# ------------------------------------------------------------------------------------------------ drawn cases
def _log(rng, a, b):
    """A whole number from a to b, even over the logarithm."""
    return max(a, min(b, int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))))


def _mult(rng, passo, a, b):
    """A multiple of `passo` from a to b, even over the logarithm."""
    return passo * _log(rng, a // passo, b // passo)


def draw(rng):
    kind = rng.choices(["passo", "linear", "gemm", "atencao", "blocos"], [7, 3, 3, 3, 3])[0]
    blk = rng.choice([32, 32, 32, 128])
    if kind == "passo":
        # a step's token count is a power of two (the mean over the tokens is a shift), its layers have D = 2^n and FF = n * 128
        while True:
            D = rng.choice([128, 256, 512, 1024])
            hd = rng.choice([64, 64, 64, 16, 4])
            T = rng.choice([64, 128, 256, 512, 1024])
            M = 1 << rng.randint(7, 13)
            L = rng.randint(1, 6)
            FF = _mult(rng, 128, D, 4 * D)
            if M >= T and D % blk == 0 and D // hd >= 1 and (M // T) * (D // hd) * T * T <= MAX_ESCORES // 4:
                return dict(kind=kind, modo=rng.choice(["gravado", "gravado", "eager", "avalia"]), blk=blk, D=D, H=D // hd, FF=FF, L=L, T=T, Bt=M // T)
    if kind == "linear":
        return dict(kind=kind, blk=blk, M=_mult(rng, 128, 128, 16384), N=_mult(rng, 128, 128, 4096), K=_mult(rng, 128, 128, 4096))
    if kind == "gemm":
        return dict(kind=kind, op=rng.choice(["bloco", "cru", "soma", "relu2", "relu2_back"]), blk=blk, M=_mult(rng, 64, 64, 16384),
                    N=_mult(rng, 128, 128, 4096), K=_mult(rng, rng.choice([128, blk]), 128, 4096))
    if kind == "atencao":
        while True:
            hd, T, Bt = rng.choice([64, 64, 16, 4]), _mult(rng, 32, 32, 1024), _log(rng, 1, 16)
            D = rng.choice([128, 256, 512, 1024])
            if D % blk == 0 and Bt * (D // hd) * T * T <= MAX_ESCORES and Bt * T >= 64:
                return dict(kind=kind, blk=blk, Bt=Bt, T=T, H=D // hd, hd=hd)
    return dict(kind="blocos", blk=blk, R=_log(rng, 64, 16384), C=rng.choice([256, 512, 1024, 2048]))


# ------------------------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _pasta():
    return tempfile.mkdtemp()


def _lancador(blk):
    ops.define_blk(blk)
    reg = registro.Registro(_pasta(), "perf", eco=False, salvar=False)
    oc = ops.OpsCuda(reg)
    reg.novo_passo(0)
    return oc, reg


class _Sorteio:
    """Seeded inputs made on the GPU: uniform mantissas, one exponent per block; raw tensors with an exponent per element."""

    def __init__(self, seed, blk):
        self.g, self.blk = torch.Generator(device="cuda").manual_seed(seed), blk

    def _ints(self, a, b, forma, tipo):
        return torch.randint(a, b + 1, forma, generator=self.g, device="cuda", dtype=torch.int32).to(tipo)

    def bloco(self, R, C, e0=-8, esp=4):
        return self._ints(-127, 127, (R, C), torch.int8), self._ints(e0 - esp, e0 + esp, (R, C // self.blk), torch.int8)

    def cru(self, R, C, bits, e0):
        return self._ints(-(1 << bits), (1 << bits) - 1, (R, C), torch.int32), self._ints(e0 - 3, e0 + 3, (R, C), torch.int16)

    def tok(self, n):
        return self._ints(0, V - 1, (n,), torch.int32)


def _lotes(seed, Bt, T):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randint(0, V, (N_LOTES, Bt, T + 1), generator=g, device="cuda")
    return [(x[i, :, :-1].contiguous(), x[i, :, 1:].contiguous()) for i in range(N_LOTES)]


def prepare(case, seed):
    c = dict(case)
    oc, reg = _lancador(c["blk"])
    s = dict(caso=c, oc=oc, reg=reg, n=0)
    if c["kind"] == "passo":
        # what a training program holds: the model, its batches on the GPU and, after a first step, the step's recording
        s["m"] = modelo.Modelo(V, c["D"], c["H"], c["FF"], c["L"], seed, "cuda", oc, reg)
        s["lotes"] = _lotes(seed, c["Bt"], c["T"])
        if c["modo"] == "gravado":
            s["m"].passo(*s["lotes"][0], k_lr=K_LR)
            s["passo"] = modelo.PassoGravado(s["m"], c["Bt"], c["T"], K_LR)
        return s
    g = _Sorteio(seed, c["blk"])
    if c["kind"] == "linear":
        s["X"], s["W"], s["dY"] = g.bloco(c["M"], c["K"]), g.bloco(c["N"], c["K"]), g.bloco(c["M"], c["N"])
    elif c["kind"] == "gemm":
        s["A"], s["B"], s["X"] = g.bloco(c["M"], c["K"]), g.bloco(c["N"], c["K"]), g.bloco(c["M"], c["N"])
    elif c["kind"] == "atencao":
        M, D = c["Bt"] * c["T"], c["H"] * c["hd"]
        s["qkv"], s["go"] = g.bloco(M, 3 * D, e0=-10, esp=3), g.bloco(M, D, e0=-20)
    else:
        R, C = c["R"], c["C"]
        s["x"], s["h"], s["g"] = g.bloco(R, C, e0=-10), g.bloco(R, C, e0=-10), g.bloco(R, C, e0=-20)
        s["o"] = g.cru(R, C, 24, -30)
        s["logits"], s["alvo"] = g.cru(R, V, 22, -20), g.tok(R)
        s["grad"], s["mom"], s["w"], s["res"] = g.cru(R, C, 26, -45), g.bloco(R, C, e0=-40), g.bloco(R, C, e0=-9), g.bloco(R, C, e0=-20)
    return s


# ------------------------------------------------------------------------------------------------ one pass
def _estado(m):
    """The updated state, up to the number of tensors a pass may hand back: every weight's mantissas first, then exponents, then residual
    and momentum of each weight in turn."""
    nomes = sorted(m.p)
    t = [m.p[n][0] for n in nomes] + [x for n in reversed(nomes) for x in (*m.res[n], *m.mom[n], m.p[n][1])]
    return t[:MAX_SAIDAS - 1]


def run(state):
    s, c, oc, reg = state, state["caso"], state["oc"], state["reg"]
    s["n"] += 1
    if c["kind"] == "passo":
        lote = s["lotes"][s["n"] % N_LOTES]
        if c["modo"] == "gravado":
            return [s["passo"](*lote), *_estado(s["m"])]
        reg.novo_passo(s["n"])
        if c["modo"] == "avalia":
            return s["m"].passo(*lote)
        return [s["m"].passo(*lote, k_lr=K_LR), *_estado(s["m"])]
    reg.novo_passo(s["n"])
    if c["kind"] == "linear":
        X, W, dY = s["X"], s["W"], s["dY"]
        Y = oc.gemm(X, W)
        dX = oc.gemm(dY, oc.transpoe(W))
        a, b = oc.transpoe2(dY, X)
        return Y, dX, oc.gemm(a, b, cru=True)
    if c["kind"] == "gemm":
        op = c["op"]
        if op == "soma":
            return oc.gemm_soma(s["A"], s["B"], s["X"])
        if op == "relu2":
            return oc.gemm_relu2(s["A"], s["B"])
        if op == "relu2_back":
            return oc.gemm_relu2_back(s["A"], s["B"], s["X"])
        return oc.gemm(s["A"], s["B"], cru=op == "cru")
    if c["kind"] == "atencao":
        (o, P), forma = oc.atencao(s["qkv"], c["Bt"], c["T"], c["H"]), (c["Bt"], c["T"], c["H"])
        g = oc.atencao_back(s["go"], s["qkv"], P, *forma)
        return P, o, g, oc.quant(o), oc.quant(g)
    y, cache = oc.rms(s["x"])
    a = oc.relu2(s["h"])
    gh = oc.relu2_back(s["g"], s["h"])
    gx = oc.rms_back(gh, y, cache)
    z = oc.soma(gx, s["g"])
    q = oc.quant(s["o"])
    loss = oc.softmax_ce(s["logits"], s["alvo"], log2M=14)
    mom = oc.momento(s["grad"], s["mom"])
    w, r = oc.peso(s["w"], mom, s["res"], K_LR, True)
    return y, cache, a, gh, gx, z, q, loss, mom, w, r


# ------------------------------------------------------------------------------------------------ what a pass needs
def work(case):
    """Inputs read once, outputs written once; 2 operations per multiply-add of every contraction."""
    c = case
    b1 = 1 + 1.0 / c["blk"]                  # bytes per element of a block tensor; a raw tensor has 6
    if c["kind"] == "passo":
        D, FF, L, M, T = c["D"], c["FF"], c["L"], c["Bt"] * c["T"], c["T"]
        pesos = L * (4 * D * D + 2 * D * FF) + V * D                   # multiplied matrices: the layers and the output head
        escores = L * c["Bt"] * D * (T * T + T)                        # multiply-adds of one causal product of T x hd x T, all heads, times 2
        treina = c["modo"] != "avalia"
        n_par = pesos + V * D                                           # and the embedding table
        # a training step reads and writes weights, momentum and residual; gradients of the weights add two products per weight, the
        # embedding's gradient one; attention is 2 products forward and 4 more backward (dO v^T, dS k, dS^T q, P^T dO)
        return {"bytes": n_par * b1 * (6 if treina else 1) + 2 * M * 8,
                "flops": 2 * M * pesos * (3 if treina else 1) + (2 * M * V * D if treina else 0) + escores * (6 if treina else 2)}
    if c["kind"] == "linear":
        M, N, K = c["M"], c["N"], c["K"]
        return {"bytes": (M * K + N * K + M * N) * b1 + (M * N + M * K) * b1 + N * K * 6, "flops": 6 * M * N * K}
    if c["kind"] == "gemm":
        M, N, K = c["M"], c["N"], c["K"]
        saida = {"bloco": b1, "cru": 6, "soma": 2 * b1, "relu2": 2 * b1, "relu2_back": 2 * b1}[c["op"]]
        return {"bytes": (M * K + N * K) * b1 + M * N * saida, "flops": 2 * M * N * K}
    if c["kind"] == "atencao":
        Bt, T, H, hd = c["Bt"], c["T"], c["H"], c["hd"]
        MD = Bt * T * H * hd
        return {"bytes": 4 * MD * b1 + Bt * H * T * T + 4 * MD * (6 + b1), "flops": 6 * Bt * H * hd * (T * T + T)}
    R, C = c["R"], c["C"]
    return {"bytes": R * C * (15 * b1 + 12) + R * (V * (6 + b1) + 4 + 16), "flops": 0}      # 6 block and 2 raw tensors in, 9 block tensors out; the loss


def tolerance(case):
    # every operator is integer arithmetic with its rounding specified; the loss report of a step is a mean of doubles (1e-12: the
    # rounding of a sum of at most 16384 of them, in any order)
    return {"rel": 1e-12} if case["kind"] == "passo" else "exact"
