"""The extension that issues short passes is optional: without it the library still builds and loads."""
import pytest

from create_llm_by_cupy_b200.ops import build as B
from create_llm_by_cupy_b200.ops import native


@pytest.fixture
def elsewhere(tmp_path, monkeypatch):
    monkeypatch.setattr(B, "HOST_LIB", tmp_path / "_b200host.so")
    monkeypatch.setattr(B, "HOST_STAMP", tmp_path / "build" / "host_ops.sha1")


@pytest.mark.parametrize("command", [["false"], ["/no/such/compiler"]])
def test_library_without_extension(elsewhere, monkeypatch, command):
    monkeypatch.setattr(B, "_host_command", lambda: command)
    with pytest.warns(RuntimeWarning, match="issued from Python"):
        assert B.build().exists()
    assert B.is_current() and not B.host_current() and native._load_host() is None


def test_file_that_cannot_be_loaded(elsewhere):
    B.HOST_STAMP.parent.mkdir()
    B.HOST_LIB.write_bytes(b"not a library")
    B.HOST_STAMP.write_text(B._host_digest())
    with pytest.warns(RuntimeWarning, match="cannot load"):
        assert native._load_host() is None


def test_failed_build_leaves_nothing_current(elsewhere, monkeypatch):
    B.HOST_STAMP.parent.mkdir()
    B.HOST_LIB.write_bytes(b"an older one")
    B.HOST_STAMP.write_text(B._host_digest())
    monkeypatch.setattr(B, "HOST_FLAGS", [*B.HOST_FLAGS, "-DOTHER"])           # a flag counts like the source
    assert not B.host_current()
    monkeypatch.setattr(B, "_host_command", lambda: ["false"])
    with pytest.warns(RuntimeWarning):
        B.build()
    assert not B.host_current()


def test_built_here():
    B.build()
    assert B.host_current()
