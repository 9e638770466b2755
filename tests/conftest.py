"""Test setup: the `gpu` marker, the package import, the oracle path, and skips for the
tests against the reference's own libraries where those cannot be built.

The package directory is named `spuma-multiphysics_b200`; it is registered here
as the importable module `spuma_multiphysics_b200`.
"""
import importlib.util
import os
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))
if str(ROOT / "tests") not in sys.path:
    sys.path.insert(0, str(ROOT / "tests"))


def _register_package():
    name = "spuma_multiphysics_b200"
    if name in sys.modules:
        return
    pkg_dir = ROOT / "spuma-multiphysics_b200"
    spec = importlib.util.spec_from_file_location(name, pkg_dir / "__init__.py",
                                                  submodule_search_locations=[str(pkg_dir)])
    module = importlib.util.module_from_spec(spec)
    sys.modules[name] = module
    spec.loader.exec_module(module)


_register_package()


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")


def _reference_unavailable(e):
    """The reference library whose absence raised `e`, or None. Only where the
    reference's sources are absent too (oracle/Makefile builds the libraries from
    them): with the sources there, a missing library is a failure."""
    name = Path(str(e).split(":")[0])
    sources = Path(os.environ.get("REFERENCE", ROOT.parent / "reference"))
    if name.parent.name != "_ref" or name.parent.parent.name != "oracle" or name.exists():
        return None
    return None if (sources / "src" / "reactiveTransport" / "reactiveTransport.cpp").is_file() else name.name


def _skip_without_reference(e):
    missing = _reference_unavailable(e)
    if missing:
        pytest.skip(f"{missing}: the reference's sources are not on this machine")
    raise e


@pytest.hookimpl(wrapper=True)
def pytest_runtest_setup(item):
    try:
        return (yield)
    except OSError as e:
        _skip_without_reference(e)


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    try:
        return (yield)
    except OSError as e:
        _skip_without_reference(e)


@pytest.fixture(scope="session")
def cuda_available():
    import torch
    return torch.cuda.is_available()
