"""The native front's handling of Python objects, without a GPU: tensors on a fake CUDA device have no memory, so that
taking their pointer throws on the way."""
import gc

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
