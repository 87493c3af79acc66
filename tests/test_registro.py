"""The launch registry on its own (no GPU): section labels."""
import tempfile

import pytest

from jatai_b200 import registro


class _Lib:
    """A library whose error record holds one sentinel of launch 0."""

    def jt_erro_le(self, rec):
        rec[0], rec[1], rec[2], rec[3], rec[4], rec[5] = 1, 6, 0, 5, 300, 256
        return 1

    def jt_erro_limpa(self):
        return 0


def _novo():
    r = registro.Registro(tempfile.mkdtemp(), "r", lib=_Lib(), eco=False, salvar=False)
    r.novo_passo(0)
    return r


def test_rotulos_depois_de_um_erro():
    """A sentinel found inside nested sections is blamed on the failing launch's section; once the blocks have been left there is no label,
    and the launches of the next step carry their own."""
    r = _novo()
    with r.trecho("forward"), r.trecho("embedding"):
        r.registra("embed", {}, (1, 4))
    with pytest.raises(registro.ErroJatai, match="forward / embedding"):
        with r.trecho("backward"), r.trecho("camada 1"), r.trecho("mlp"):
            r.confere_device()
    assert r.onde() == "-"
    with pytest.raises(registro.ErroJatai, match="forward / embedding"):
        with r.trecho("fim"):
            r.confere_device()
    assert r.onde() == "-"
    with pytest.raises(registro.ErroJatai, match="forward / embedding"):
        r.confere_device()
    assert r.onde() == "-"
    with r.trecho("a"):
        with pytest.raises(registro.ErroJatai, match="forward / embedding"):
            r.confere_device()
        assert r.onde() == "a"
    assert r.onde() == "-"


def test_rotulo_como_decorador():
    r = _novo()

    @r.trecho("f")
    def f(n):
        return f(n - 1) if n else r.onde()

    assert f(0) == "f" and f(2) == "f / f / f" and r.onde() == "-"
