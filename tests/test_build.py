"""The host module is rebuilt for another torch, whose C++ interfaces it was not compiled against."""
import torch

from nvfp4_training_b200 import _lib, build


def test_host_module_follows_the_installed_torch(monkeypatch):
    build.build_host()
    assert not build.host_is_stale()
    _lib.host()
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "9.9.9")
        assert build.host_is_stale()
        m.setattr(_lib, "_host", None)
        try:
            _lib.host()
        except _lib.Nvfp4Error as e:
            assert "9.9.9" in str(e)
        else:
            raise AssertionError("a host module of another torch was taken")
    _lib.host()
