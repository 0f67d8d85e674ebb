"""_host.so belongs to the torch and the Python it was built against."""
import pytest


def test_a_module_for_another_torch_is_rebuilt_and_not_used(monkeypatch):
    from triton_int8_b200 import build, kernels
    build.build()
    assert not build.needs_host_build()
    monkeypatch.setattr(kernels, "_host", None)
    assert kernels.host().abi == build.host_abi()
    monkeypatch.setattr(kernels, "_host", None)
    monkeypatch.setattr(build, "host_abi", lambda: "torch 1.0, cpython-30")
    assert build.needs_host_build()
    with pytest.raises(ImportError, match="built for"):
        kernels.host()
