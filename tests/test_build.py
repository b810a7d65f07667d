"""When the incremental build rebuilds the host path: it is bound to the torch it was built against."""

import os

import pytest
import torch

import build_lib


@pytest.fixture
def built(tmp_path, monkeypatch):
    """A host path that was just built, in a scratch place."""
    monkeypatch.setattr(build_lib, "TORCH_EXT", str(tmp_path / "_fda_torch.so"))
    monkeypatch.setattr(build_lib, "TORCH_STAMP", str(tmp_path / "_fda_torch.txt"))
    command = build_lib._torch_command()
    for path, text in ((build_lib.TORCH_EXT, ""), (build_lib.TORCH_STAMP, build_lib._torch_stamp(command))):
        with open(path, "w") as f:
            f.write(text)
    return command


def test_unchanged_host_path_is_kept(built):
    assert not build_lib._torch_ext_stale(built)


def test_other_torch_rebuilds_the_host_path(built, monkeypatch):
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    assert build_lib._torch_ext_stale(built)


def test_other_flags_rebuild_the_host_path(built):
    assert build_lib._torch_ext_stale(built + ["-I/elsewhere"])


def test_host_path_of_unknown_origin_is_rebuilt(built):
    os.remove(build_lib.TORCH_STAMP)
    assert build_lib._torch_ext_stale(built)
