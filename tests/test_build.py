"""What counts as a fresh build of the host extension."""
import os

import torch

from simplicial_attention_b200 import build


def test_extension_is_tied_to_torch_and_python(monkeypatch):
    path = build.ext_path()
    assert os.path.exists(build.build_ext()) and not build.ext_is_stale()
    monkeypatch.setattr(torch, "__version__", "0.0.0+other")
    assert build.ext_path() != path and build.ext_is_stale()
