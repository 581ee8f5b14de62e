"""The smoke entry point, with the oracle and without it."""
import pytest

import __graft_entry__
from oracle import oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("oracle", [True, False])
def test_smoke(monkeypatch, tmp_path, capsys, oracle):
    if oracle and not O.available():
        pytest.skip("the oracle is not built here")
    if not oracle:
        monkeypatch.setattr(O, "LIB_PATH", tmp_path / "none.so")
    __graft_entry__.smoke()
    assert "smoke ok" in capsys.readouterr().out
