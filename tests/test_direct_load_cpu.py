"""The library behind `call_fwd`'s short path is an extra: one that cannot be used costs a warning, not the op."""
import os
import shutil

import pytest

from flash_cuda_b200 import build, ops


@pytest.fixture
def direct_so(tmp_path, monkeypatch):
    path = str(tmp_path / "fa_b200_direct.so")
    for lib in (build.TORCH_SO, build.CAPI_SO):        # (it looks for the op's library beside itself)
        os.symlink(lib, tmp_path / os.path.basename(lib))
    monkeypatch.setattr(build, "DIRECT_SO", path)
    monkeypatch.setattr(ops, "_loaded", False)
    monkeypatch.setattr(ops, "_direct", None)
    return path


def _stamp(path):
    build._write_stamp(path, build._direct_source()[1])


def test_built_library_is_used(direct_so):
    shutil.copy(os.path.join(build.LIB, "fa_b200_direct.so"), direct_so)
    _stamp(direct_so)
    assert ops.load().fwd is not None and ops._direct is not None


def test_library_that_cannot_be_imported(direct_so):
    with open(direct_so, "wb") as f:
        f.write(b"not a library")
    _stamp(direct_so)
    with pytest.warns(UserWarning, match="dispatcher"):
        assert ops.load().fwd is not None
    assert ops._direct is None


@pytest.mark.parametrize("stamp", [None, "of another build"])
def test_library_of_another_build_is_not_executed(stamp, direct_so):
    shutil.copy(os.path.join(build.LIB, "fa_b200_direct.so"), direct_so)
    if stamp:
        build._write_stamp(direct_so, stamp)
    with pytest.warns(UserWarning, match="another Python"):
        assert ops.load().fwd is not None
    assert ops._direct is None


@pytest.mark.parametrize("works", [True, False])
def test_missing_library_is_built(works, direct_so, monkeypatch):
    asked = []

    def fake_build():
        asked.append(1)
        if not works:
            raise RuntimeError("no compiler")
        shutil.copy(os.path.join(build.LIB, "fa_b200_direct.so"), direct_so)
        _stamp(direct_so)

    monkeypatch.setattr(build, "build_direct", fake_build)
    if works:
        ops.load()
    else:
        with pytest.warns(UserWarning, match="no compiler"):
            ops.load()
    assert asked == [1] and (ops._direct is not None) == works


def test_missing_library_is_left_alone_on_request(direct_so, monkeypatch):
    monkeypatch.setattr(build, "build_direct", lambda: pytest.fail("built"))
    with pytest.warns(UserWarning, match="missing"):
        assert ops.load(build_if_missing=False).fwd is not None
    assert ops._direct is None
