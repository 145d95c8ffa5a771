"""The smoke run works where the oracle is not built."""
import pytest

pytestmark = pytest.mark.gpu


def test_smoke_without_the_oracle(monkeypatch, capsys):
    import __graft_entry__
    from oracle import ref
    monkeypatch.setattr(ref, "available", lambda: False)
    __graft_entry__.smoke()
    assert "smoke ok" in capsys.readouterr().out
