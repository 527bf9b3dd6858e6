"""The front end without a GPU: which calls the extension takes itself, and what the Python forms refuse before
anything is launched."""
import ctypes
import subprocess
import sys
import textwrap
import weakref
from pathlib import Path

import pytest
import torch

import autograph_b200 as ag
from autograph_b200 import _capi

ROOT = Path(__file__).resolve().parent.parent


def _operator_calls(t):
    """Every operator with tensors made by t(shape): (name, arguments, keyword arguments)."""
    x, w, dy, b = t((2, 3, 6, 6)), t((4, 3, 3, 3)), t((2, 4, 4, 4)), t((4,))
    m, n, v = t((4, 4)), t((4, 4)), t((4,))
    labels = t((4,), torch.uint8)
    return [
        ("gemm", (1.0, m, n, 0.0, t((4, 4))), {}), ("dot", (m, n), {}),
        ("dense_forward", (m, n), dict(bias=v)), ("dense_chain_forward", (m, [n], [v]), {}),
        ("dense_chain_forward_keep", (m, [n], [v], [True]), {}),
        ("dense_chain_backward", (m, [n], [True], [t((4, 4))], [t((4, 4))], t((4, 4))), {}),
        ("conv2_forward", (x, w), dict(bias=b)), ("conv2_relu_max_pool2", (x, w), dict(bias=b)),
        ("conv2_relu_max_pool2_keep", (x, w), dict(bias=b)), ("conv2_backward_input", (w, dy, (6, 6)), {}),
        ("conv2_backward_weight", (x, dy, (3, 3)), dict(beta=1.0, dw=w)),
        ("conv_dense_chain_forward", (x, [(w, b, True, (2, 2))], [t((16, 4))], [v], [False]), {}),
        ("im2col_conv2", (x, (3, 3)), {}), ("col2im_conv2", (t((32, 27)), (4, 4), (3, 3)), {}),
        ("max_pool2", (x,), {}), ("max_pool2_backward_inplace", (x, t((2, 3, 3, 3))), {}),
        ("max_pool2_backward_from_input", (x, t((2, 3, 3, 3))), {}), ("relu_max_pool2", (x,), {}),
        ("relu_max_pool2_backward", (x, t((2, 3, 3, 3))), {}), ("relu", (x,), {}), ("relu", (x, True), {}),
        ("relu_backward", (x, t((2, 3, 6, 6))), {}), ("scaled_add", (m, 1.0, n), {}), ("bias_add", (m, v), {}),
        ("bias_grad", (m,), dict(beta=1.0, out=v)), ("scaled_cast_u8", (labels, 1.0, torch.float32), {}),
        ("cross_entropy_loss", (m, labels), {}), ("cross_entropy_loss_with_grad", (m, labels), {}),
        ("cross_entropy_loss_backward", (m, labels), {}), ("accuracy", (m, labels), {}),
        ("sgd_update", (m, n, 0.1), {}), ("sgd_update_momentum", (m, n, t((4, 4)), 0.1, 0.9), {}),
    ]


@pytest.fixture
def no_launch(monkeypatch):
    """A device object without a GPU: outputs on the CPU, a library whose operators must not be reached."""
    class Library:
        ag_conv2_output_shape = ag.lib().ag_conv2_output_shape

        def __getattr__(self, name):
            raise AssertionError(f"{name} was called")

    monkeypatch.setattr(ag, "lib", Library)
    d = ag._PyDevice.__new__(ag._PyDevice)
    d.index, d.torch_device, d._stream_ptr, d._h = 0, torch.device("cpu"), 0, None
    return d


def test_operators_refuse_host_tensors(no_launch):
    for name, args, kw in _operator_calls(lambda s, dt=torch.float32: torch.zeros(s, dtype=dt)):
        with pytest.raises(ag.AgError, match="must be in device memory"):
            getattr(ag._PyDevice, name)(no_launch, *args, **kw)


def test_operators_refuse_tensors_of_another_gpu(no_launch):
    class Elsewhere(torch.Tensor):
        is_cuda, device = True, torch.device("cuda", 1)

    make = lambda s, dt=torch.float32: torch.zeros(s, dtype=dt).as_subclass(Elsewhere)
    for name, args, kw in _operator_calls(make):
        if name.startswith("dense_chain_backward"):
            continue   # its intermediate outputs are the operator's own
        with pytest.raises(ag.AgError, match="on another GPU"):
            getattr(ag._PyDevice, name)(no_launch, *args, **kw)


def test_python_forms_hold_copies_and_refuse_strided_outputs(no_launch, monkeypatch):
    """Operands that are not contiguous reach the library as contiguous copies that are all alive during the call: freed
    before it, the memory of one was the next one's.  Tensors that are written too are refused instead."""
    copies, originals = [], set()

    class Here(torch.Tensor):
        is_cuda, device = True, torch.device("cuda", 0)

        def contiguous(self):
            if self.is_contiguous():
                return self
            t = super().contiguous()
            copies.append(weakref.ref(t))
            originals.add(self.data_ptr())
            return t

    def strided(shape, dt=torch.float32):
        if len(shape) == 1:
            return torch.zeros(2 * shape[0], dtype=dt)[::2].as_subclass(Here)
        return torch.zeros(shape[::-1], dtype=dt).permute(*reversed(range(len(shape)))).as_subclass(Here)

    def pointers(args):
        for a in args:
            if isinstance(a, ctypes.c_void_p):
                yield a.value
            elif isinstance(a, ctypes.Array) and a._type_ is ctypes.c_void_p:
                yield from a
            elif isinstance(a, ctypes.Array) and a._type_ is _capi.ConvStage:
                yield from (p for st in a for p in (st.w, st.bias))

    reached = []

    class Library:
        ag_conv2_output_shape = ag.lib().ag_conv2_output_shape

        def __getattr__(self, name):
            def call(*args):
                assert copies and all(ref() is not None for ref in copies), f"{name}: a copy was freed"
                assert not originals & set(pointers(args)), f"{name}: reads a strided tensor"
                reached.append(name)
                return 0
            return call

    library = Library()
    monkeypatch.setattr(ag, "lib", lambda: library)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda index: type("Stream", (), {"cuda_stream": 0}))
    written = {"gemm": None, "conv2_backward_weight": "dw", "max_pool2_backward_inplace": 0, "bias_add": 0, "bias_grad": "out",
               "sgd_update": 0, "sgd_update_momentum": (0, 2)}
    for name, args, kw in _operator_calls(strided):
        if name in ("gemm", "dot", "scaled_add"):
            continue   # strides are passed on; refused by an assertion
        args, outs = list(args), written.get(name, ())
        for key in outs if isinstance(outs, tuple) else (outs,):
            at = kw if isinstance(key, str) else args
            before, at[key] = at[key], torch.zeros(at[key].shape).as_subclass(Here)
            with pytest.raises(ag.AgError, match="must be contiguous"):
                at[key], plain = before, at[key]
                getattr(ag._PyDevice, name)(no_launch, *args, **kw)
            at[key] = plain
        copies.clear()
        originals.clear()
        reached.clear()
        getattr(ag._PyDevice, name)(no_launch, *args, **kw)
        assert len(reached) == 1, name


# In a process of its own: the library's functions are replaced by ones that count, and no device is needed for the
# model's host calls.  The calls that go to the Python form are counted as well.
_HARNESS = """
import ctypes, sys
import torch
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
from autograph_b200 import _front
native, python = [], []
kept = []
def counting(name):
    fn = ctypes.CFUNCTYPE(ctypes.c_int)(lambda: native.append(name) or 0)
    kept.append(fn)
    return ctypes.cast(fn, ctypes.c_void_p).value
_front.bind({{n: counting(n) for n in _front.FUNCTIONS}}, lambda status: None)
for n in _front.METHODS:
    _front.set_fallback(n, lambda self, *a, _n=n, **k: python.append(_n))
model = _front.ModelBase()
model._bind(1, 0, 0, 10)
def taken(call):
    native.clear(); python.clear()
    call()
    assert len(native) + len(python) == 1, (native, python)
    return "native" if native else "python"
x, out = torch.zeros(2, 1, 4, 4), torch.zeros(2, 10)
infer = lambda x=x, out=out: taken(lambda: model.infer(x, out))
"""


def _in_process(body):
    res = subprocess.run([sys.executable, "-c", _HARNESS.format(root=str(ROOT)) + textwrap.dedent(body)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-3000:]


def test_extension_leaves_host_tensors_to_the_python_form():
    """An operator's fast path takes tensors of its own GPU alone, whichever argument another one is."""
    _in_process("""
        from test_front import _operator_calls
        d = _front.DeviceBase()
        d._bind(1, 0, 0)
        for name, args, kw in _operator_calls(lambda s, dt=torch.float32: torch.zeros(s, dtype=dt)):
            if name in _front.METHODS:
                assert taken(lambda: getattr(d, name)(*args, **kw)) == "python", name
        """)


def test_a_default_device_keeps_the_fast_path():
    _in_process("""
        assert infer() == "native"
        with torch.device("cpu"):
            assert infer() == "native"
            with torch.device("meta"):
                assert infer() == "native"
        torch.set_default_device("meta")
        assert infer() == "native"
        torch.set_default_device(None)
        """)


def test_what_the_extension_leaves_to_the_python_form():
    """Modes that watch operations, wrappers of function transforms, subclasses, and tensors that are not what the kernels
    read; tensors that only carry a gradient or inference flag are plain."""
    _in_process("""
        from torch.overrides import TorchFunctionMode
        from torch.utils._device import DeviceContext
        from torch.utils._python_dispatch import TorchDispatchMode
        class Watching(TorchFunctionMode):
            def __torch_function__(self, f, types, args=(), kwargs=None):
                return f(*args, **(kwargs or {}))
        class Dispatching(TorchDispatchMode):
            def __torch_dispatch__(self, f, types, args=(), kwargs=None):
                return f(*args, **(kwargs or {}))
        class Context(DeviceContext):
            pass
        for mode in (Watching(), Dispatching(), Context(torch.device("cpu"))):
            with mode:
                assert infer() == "python", mode
                with torch.device("cpu"):
                    assert infer() == "python", mode
        with torch.device("cpu"), Watching():
            assert infer() == "python"
        assert infer() == "native"

        def mapped(x):
            assert infer(x=x) == "python"
            return x + 0
        torch.func.vmap(mapped)(torch.zeros(3, 2, 1, 4, 4))
        torch.func.jvp(mapped, (x,), (x,))

        class Sub(torch.Tensor):
            pass
        for other in (x.as_subclass(Sub), x.double(), x.to("meta"), x.transpose(2, 3).expand(2, 1, 4, 4)[:, :, ::2],
                      x.to_sparse(), torch.zeros(2, 4, 4), [0.0], None):
            assert infer(x=other) == "python", type(other)
        for out2 in (torch.zeros(2, 9), torch.zeros(3, 10), torch.zeros(10, 2).t(), out.double(), None):
            assert infer(out=out2) == "python"
        with torch.inference_mode():
            made = torch.zeros(2, 1, 4, 4)
            assert infer(x=made) == "native"
        assert infer(x=made) == "native"
        assert infer(x=torch.nn.Parameter(x)) == "native" and infer(x=x.requires_grad_()) == "native"
        """)
