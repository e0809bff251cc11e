"""The Python surface of the binding: what stands in a Python function's place behaves like that function."""
import copy
import inspect
import pickle

import pytest

import llmt_b200 as L

NATIVE = ["gemm", "gemm_desc", "zero_grads", "softmax_fwd", "softmax_bwd", "gemm_softmax_fwd", "gemm_softmax_bwd", "rowdot", "head_split",
          "head_merge", "cross_entropy_fwd", "cross_entropy_bwd", "lm_head_ce_fwd", "lm_head_ce_bwd", "_group_run"]


@pytest.mark.parametrize("name", NATIVE)
def test_native_functions_keep_their_python_face(name):
    f = getattr(L, name)
    assert f is not inspect.unwrap(f), "the native form is in place"
    python = inspect.unwrap(f)
    assert inspect.signature(f) == inspect.signature(python) and len(inspect.signature(f).parameters) >= 2
    assert (f.__name__, f.__qualname__, f.__module__, f.__doc__) == (name, name, "llmt_b200", python.__doc__)
    assert f.__defaults__ == python.__defaults__ and f.__annotations__ == python.__annotations__
    assert pickle.loads(pickle.dumps(f)) is f and copy.copy(f) is f and copy.deepcopy(f) is f
    with pytest.raises(TypeError):
        f(no_such_argument=1)
    with pytest.raises(AttributeError):
        f.no_such_attribute
    holder = type("Holder", (), {"call": f})()
    assert holder.call.__self__ is holder and holder.call.__func__ is f
