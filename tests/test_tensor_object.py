"""The Tensor object itself, on CPU: what it takes for its storage, and what it hands out.  (The ops need a GPU; the object does
not, as long as the native host side is built.)"""
import copy
import os
import pickle
import subprocess
import sys

import pytest
import torch

from irontensor_b200 import Precision, Tensor, _lib

pytestmark = pytest.mark.skipif(isinstance(_lib.host_ops(), _lib._Missing), reason="_host_ops.so is not built")
FP32, BF16 = Precision.FP32, Precision.BF16


# The declared precision decides what the bits are; integers of the same width, or bytes, carry them.
@pytest.mark.parametrize("stored,precision,held", [
    (torch.float32, FP32, torch.float32), (torch.int32, FP32, torch.float32), (torch.uint32, FP32, torch.float32),
    (torch.bfloat16, BF16, torch.bfloat16), (torch.int16, BF16, torch.bfloat16), (torch.uint16, BF16, torch.bfloat16),
])
def test_bits_of_the_declared_precision(stored, precision, held):
    values = torch.arange(12, dtype=torch.float32).to(held)
    t = Tensor(values.view(stored), [3, 4], precision)
    assert t.precision() is precision and t.byte_size() == 12 * precision.byte_size()
    assert t.torch().dtype == held and torch.equal(t.torch(), values.view(3, 4))
    assert t.data_ptr() % 4 == 0 and t.shape() == [3, 4]
    b = Tensor(values.view(torch.uint8), [3, 4], precision)
    assert b.precision() is precision and torch.equal(b.torch(), values.view(3, 4))


@pytest.mark.parametrize("stored,precision", [
    (torch.float16, FP32), (torch.float16, BF16), (torch.float64, FP32), (torch.float32, BF16), (torch.bfloat16, FP32),
    (torch.int16, FP32), (torch.int32, BF16), (torch.int64, FP32), (torch.bool, FP32), (torch.complex64, FP32),
])
def test_other_types_are_refused(stored, precision):
    with pytest.raises(TypeError):
        Tensor(torch.zeros(4, dtype=stored), [4], precision)
    with pytest.raises(TypeError):
        Tensor(torch.zeros(4), [4], None)


def test_storage_that_is_not_packed_has_no_address():
    """The kernels know packed rows only: a strided view may be held and read back, but no op gets its address."""
    x = torch.arange(12, dtype=torch.float32).view(3, 4)
    t = Tensor(x[:, :2], [3, 2], FP32)
    assert torch.equal(t.torch(), x[:, :2])
    assert torch.equal(t._data, x[:, :2].reshape(-1))
    with pytest.raises(ValueError):
        t.data_ptr()


def test_torch_views_do_not_share_their_form():
    """What torch() hands out, and what the constructor was given, share memory with the object and nothing else: changing their
    shape or strides in place leaves the object as it was."""
    x = torch.arange(6, dtype=torch.float32).view(2, 3)
    t = Tensor(x, [2, 3], FP32)
    x.t_()
    assert t.shape() == [2, 3] and t.torch().stride() == (3, 1)
    y = t.torch()
    y.t_()
    y[0, 1] = 40.0
    assert t.shape() == [2, 3] and t.torch().is_contiguous() and t.torch()[1, 0] == 40.0 and x[0, 1] == 40.0
    t.torch().unsqueeze_(0)
    assert t.shape() == [2, 3]
    w = torch.ones(4, requires_grad=True)      # a view in autograd's sense too
    Tensor(w, [4], FP32).torch().sum().backward()
    assert torch.equal(w.grad, torch.ones(4))
    v = t.torch()._version
    t.torch().add_(1.0)
    assert t.torch()._version == v + 1         # one version counter: autograd sees writes through any of them


def _lookalike(t, u):
    return u is not t and u.precision() is t.precision() and u.shape() == t.shape() and torch.equal(u.torch(), t.torch())


def test_copies_and_pickles():
    t = Tensor(torch.arange(6, dtype=torch.float32).to(torch.bfloat16), [2, 3], BF16)
    t.lse = Tensor(torch.zeros(2), [2], FP32)
    t.note = "kept"
    shallow = copy.copy(t)
    assert _lookalike(t, shallow) and shallow.data_ptr() == t.data_ptr() and shallow.lse is t.lse and shallow.note == "kept"
    deep = copy.deepcopy(t)
    assert _lookalike(t, deep) and deep.data_ptr() != t.data_ptr()
    assert _lookalike(t.lse, deep.lse) and deep.lse.data_ptr() != t.lse.data_ptr() and deep.note == "kept"
    back = pickle.loads(pickle.dumps(t))
    assert _lookalike(t, back) and _lookalike(t.lse, back.lse) and back.lse.lse is None and back.note == "kept"
    # the state of a pickle written when the object was all Python: a flat buffer, shape, precision and lse as attributes
    old = Tensor.__new__(Tensor)
    old.__setstate__({"_data": t.torch().reshape(-1), "_shape": [2, 3], "_precision": BF16, "lse": None})
    assert _lookalike(t, old) and old.lse is None


def test_a_buffer_may_be_longer_than_the_shape():
    """A pool's block is handed over whole; the shape says how much of its beginning is the tensor."""
    pool = torch.arange(20, dtype=torch.float32)
    t = Tensor(pool, [2, 3], FP32)
    assert t.shape() == [2, 3] and t.numel() == 6 and t.byte_size() == 24
    assert t.data_ptr() == pool.data_ptr() and torch.equal(t.torch(), pool[:6].view(2, 3))
    assert Tensor(pool.view(4, 5), [7], FP32).torch().tolist() == list(range(7))
    assert Tensor(torch.zeros(9, dtype=torch.int16), [2, 4], BF16).shape() == [2, 4]
    assert Tensor(torch.zeros(9, dtype=torch.uint8), [2, 2], BF16).shape() == [2, 2]
    assert Tensor(pool, [0, 3], FP32).numel() == 0 and Tensor(pool, [], FP32).torch().item() == 0.0
    for shape in ([3, 7], [-2, -3], [2 ** 40, 2 ** 40]):     # longer than the buffer, or no shape at all
        with pytest.raises(RuntimeError):
            Tensor(pool, shape, FP32)
    with pytest.raises(RuntimeError):          # a strided buffer has no such beginning
        Tensor(pool.view(4, 5)[:, :3], [2, 3], FP32)


def test_an_object_without_storage_raises():
    """Tensor.__new__ alone, as an unpickler or a subclass whose __init__ raised leaves it.  In a process of its own: a C++
    exception that nobody translates ends the process."""
    code = """
from irontensor_b200 import Tensor
t = Tensor.__new__(Tensor)
for f in (t.shape, t.numel, t.data_ptr, t.precision, t.torch, lambda: t.view([1]), t.byte_size, t.__getstate__):
    try:
        f()
    except ValueError:
        print("raised")
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=os.path.dirname(os.path.dirname(__file__)))
    assert (r.returncode, r.stdout.split()) == (0, ["raised"] * 8), r.stderr[-500:]
