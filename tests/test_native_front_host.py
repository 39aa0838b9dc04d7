"""The native front's handling of Python objects, without a GPU: tensors on a fake CUDA device have no memory, so that
taking their pointer throws on the way."""
import gc
import importlib
import os

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode


@pytest.fixture(scope="module")
def front(pkg):
    pkg.build()
    return pkg.api.load_front()


@pytest.fixture(scope="module")
def fake(pkg):
    """(weight, x) on a fake CUDA device."""
    with FakeTensorMode():
        data, x = torch.empty(8, 16, dtype=torch.float16, device="cuda"), torch.empty(4, 16, dtype=torch.float16, device="cuda")
    return pkg.Weight(data, pkg.ScalarType.Float16, 8, 16), x


def test_an_exception_releases_the_list_of_outputs(pkg, front, fake):
    weight, x = fake

    def lists():
        gc.collect()
        return sum(type(o) is list for o in gc.get_objects())

    calls = [pkg.LinearCall(x, weight)]
    before = lists()
    for _ in range(50):
        with pytest.raises(RuntimeError):
            front.linear_grouped(0, calls, False)
    assert lists() - before < 25


def test_one_call_twice_is_left_to_the_python_path(pkg, front, fake):
    """The two have one output between them."""
    weight, x = fake
    call = pkg.LinearCall(x, weight)
    assert front.linear_grouped(0, [call, pkg.LinearCall(x, weight), call], False) is None


@pytest.mark.parametrize("state", ["absent", "not a library"])
def test_without_a_front_the_python_path_issues_the_calls(pkg, fake, monkeypatch, tmp_path, state):
    path = tmp_path / "_front.so"
    if state != "absent":
        path.write_text("no library")
    monkeypatch.setattr(pkg.api, "_front", None)
    monkeypatch.setattr(pkg.api._build, "front_path", lambda: str(path))
    with pytest.warns(RuntimeWarning, match="ctypes"):
        stand_in = pkg.api.load_front()
    weight, x = fake
    assert stand_in.linear_grouped(0, [pkg.LinearCall(x, weight)], False) is None
    assert all(getattr(stand_in, name)() is None for name in ("linear", "layer_norm", "quantize_int8", "quantize_fp8", "pack_fp8"))


def test_the_fronts_file_belongs_to_one_torch_and_python(pkg, monkeypatch):
    build = importlib.import_module(pkg.__name__ + ".build")
    here = build.front_path()
    assert os.path.exists(here)
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert build.front_path() != here
    monkeypatch.undo()
    monkeypatch.setattr(build.sysconfig, "get_config_var", lambda name: "cpython-399")
    assert build.front_path() != here


def test_a_front_that_does_not_build_leaves_the_library(pkg, monkeypatch):
    build = importlib.import_module(pkg.__name__ + ".build")
    order = []

    def no_compiler(force):
        order.append("front")
        raise RuntimeError("g++ failed")

    monkeypatch.setattr(build, "_build_library", lambda verbose: order.append("library"))
    monkeypatch.setattr(build, "build_front", no_compiler)
    with pytest.warns(RuntimeWarning, match="ctypes"):
        assert build.build(force=True) == build.LIBRARY
    assert order == ["library", "front"]
