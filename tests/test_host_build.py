"""The host extension is tied to the torch that it was built against: another version's file is never loaded."""
import os

import pytest
import torch

from crownest_b200 import CrownestError, _lib


def test_an_extension_built_for_another_torch_is_missing_not_loaded(monkeypatch):
    built = _lib.host_path()
    assert os.path.exists(built) and torch.__version__.replace("+", "_") in os.path.basename(built)
    monkeypatch.setattr(torch, "__version__", "0.1")
    monkeypatch.setattr(_lib, "_host", None)
    assert _lib.host_path() != built
    with pytest.raises(CrownestError, match="is missing: run"):
        _lib.host()
