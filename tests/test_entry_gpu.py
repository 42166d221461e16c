"""smoke() of the entry file runs on a machine without the oracle's library, against the committed record."""
import importlib

import pytest


@pytest.mark.gpu
def test_smoke_without_the_oracle(cuda_device, monkeypatch, capsys):
    from oracle import ref
    monkeypatch.setattr(ref, "available", lambda: False)
    importlib.import_module("__graft_entry__").smoke()
    assert "committed record" in capsys.readouterr().out
