"""Test setup: registers the ``gpu`` marker and loads the package (its
directory name is not a Python identifier) under the name ``feicar_b200``."""
import importlib.util
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG_DIR = os.path.join(ROOT, "feicar3d_3.0_febio_b200")
sys.path.insert(0, os.path.join(ROOT, "oracle"))
sys.path.insert(0, ROOT)


def _load_pkg():
    if "feicar_b200" in sys.modules:
        return sys.modules["feicar_b200"]
    spec = importlib.util.spec_from_file_location(
        "feicar_b200", os.path.join(PKG_DIR, "__init__.py"), submodule_search_locations=[PKG_DIR]
    )
    mod = importlib.util.module_from_spec(spec)
    sys.modules["feicar_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


_load_pkg()


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")
    config.addinivalue_line("markers", "slow: CPU test that takes more than a few seconds")


@pytest.fixture(autouse=True)
def _fields_written(request, monkeypatch):
    """The tests fill their device fields on torch's stream, and a handle's
    own stream is not ordered after it: the binding's functions on device
    fields start here once torch's work is done."""
    if request.node.get_closest_marker("gpu") is None:
        return
    import torch

    from feicar_b200 import fg

    def after_torch(call):
        def ordered(*args, **kw):
            torch.cuda.synchronize()
            return call(*args, **kw)
        return ordered

    for name in [n for n in vars(fg) if n.endswith("_device") and callable(getattr(fg, n))]:
        monkeypatch.setattr(fg, name, after_torch(getattr(fg, name)))
