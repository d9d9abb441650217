"""smoke() goes without the oracle only where there is nothing to build it from."""
import importlib.util
import os

import pytest

ENTRY = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "__graft_entry__.py")


def test_missing_oracle_is_an_error_beside_the_sources(tmp_path, monkeypatch):
    spec = importlib.util.spec_from_file_location("entry", ENTRY)
    entry = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(entry)
    (tmp_path / "reference" / "src").mkdir(parents=True)
    monkeypatch.setattr(entry, "ROOT", str(tmp_path))
    monkeypatch.setattr(entry, "REFERENCE", str(tmp_path / "reference"))
    with pytest.raises(RuntimeError, match="oracle is not built"):
        entry.smoke()
