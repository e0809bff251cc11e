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


class _At:
    """Stands for a tensor, or a stream, of which only the address is asked."""
    cuda_stream = 0

    def __init__(self, at=0x1000):
        self.at = at

    def data_ptr(self):
        return self.at


def test_a_descriptor_is_a_descriptor():
    """Bytes of the right length are not taken for one, a class derived from it is (m = 0: nothing is launched)."""
    import ctypes
    d = L.GemmDesc()
    d.n = d.k = d.lda = d.ldb = d.ldc = d.batch = 1
    raw = bytes(d)
    for wrong in (raw, bytearray(raw), (ctypes.c_char * len(raw))(*raw)):
        with pytest.raises((TypeError, ctypes.ArgumentError)):
            L.gemm_desc(wrong, _At(0x1000), _At(0x2000), _At(0x3000), _At())
    derived = type("Mine", (L.GemmDesc,), {}).from_buffer_copy(raw)
    for right in (d, derived):
        L.gemm_desc(right, _At(0x1000), _At(0x2000), _At(0x3000), _At())


def test_a_group_runs_the_arrays_it_has(monkeypatch):
    import ctypes
    seen = []
    monkeypatch.setattr(L, "_group_run", lambda *args: seen.append(args))
    g = L.Group([(L.GemmDesc(), _At(0x1000), _At(0x2000), _At(0x3000)), (L.GemmDesc(), _At(0x4000), _At(0x5000), _At(0x6000))])
    g.run()
    assert seen[0] == (*(ctypes.addressof(x) for x in (g.descs, g.c, g.a, g.b)), 2, None)
    g.c = (ctypes.c_void_p * 2)(0x7000, 0x8000)
    g.descs = (L.GemmDesc * 2)(*g.descs)
    g.a = ctypes.cast(g.b, ctypes.POINTER(ctypes.c_void_p))
    g.run()
    assert seen[1] == (ctypes.addressof(g.descs), ctypes.addressof(g.c), ctypes.addressof(g.b), ctypes.addressof(g.b), 2, None)
    assert list(g.c) == [0x7000, 0x8000]
    with pytest.raises(TypeError):
        g.b = [0x9000, 0xa000]


def test_the_extension_belongs_to_one_interpreter():
    import importlib.machinery
    import os
    from llmt_b200 import _native, build
    tag = importlib.machinery.EXTENSION_SUFFIXES[0]
    assert tag != ".so" and _native.__file__.endswith("_native" + tag) and os.path.samefile(_native.__file__, build.NATIVE_PATH)
    assert not os.path.exists(os.path.join(os.path.dirname(_native.__file__), "_native.so"))
