"""The PyTorch front-end is rebuilt when the installed torch changes, not only when its sources do."""
import torch

from d2conv3d_b200 import build


def test_front_end_is_tied_to_the_torch_it_was_built_against(tmp_path, monkeypatch):
    lib, stamp = tmp_path / "_C.so", tmp_path / "stamp"
    monkeypatch.setattr(build, "TORCH_LIB", str(lib))
    monkeypatch.setattr(build, "TORCH_STAMP", str(stamp))
    lib.write_bytes(b"")                          # newer than its sources
    assert build._torch_needs_build()             # nobody knows what it was built against
    stamp.write_text(build._torch_stamp())
    assert not build._torch_needs_build()
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    assert build._torch_needs_build()
