"""The per-call binding (csrc/host_call.c, and _call_py.py, which stands in for it) on the CPU: what it hands to the library and
what it refuses.  The library's own argument checks come first, so a call with a freed handle ends in them without a GPU."""
import collections
import ctypes as C
import importlib.util
import subprocess
import sys
import types

import pytest
import torch

from muser_b200 import _call, _call_py, _lib, build, operator as op


@pytest.fixture(params=[_call, _call_py], ids=["c", "ctypes"])
def kern(request, monkeypatch):
    monkeypatch.setattr(op, "_call", request.param)

    def bind(raw, slow):
        op._call.bind(str(_lib.LIB_PATH), op._TORCH_DTYPE, torch.float32, raw, slow, op.MuserCudaError, C.ArgumentError)
    bind(lambda device: 0, lambda device: 0)
    ctx = op.Context.__new__(op.Context)
    ctx.device, ctx._h = 0, None
    yield op.CudaKernels(ctx), types.SimpleNamespace(_h=None, dtype=op.Q4_K, n_out=16)
    bind(torch._C._cuda_getCurrentRawStream, op._stream_ptr)


def test_arguments_are_refused_as_before(kern):
    k, w = kern
    x, y = torch.zeros((2, 256)), torch.zeros((2, 16))
    calls = {
        "matmul": lambda **kw: k.encode_quantized_matmul(w, kw.pop("x", x), y, kw.pop("tokens", 2), **kw),
        "group": lambda **kw: k.encode_quantized_matmul_group([w, w], kw.pop("x", x), [y, y], kw.pop("tokens", 2), epilogues=[None, kw]),
        "nvfp4": lambda **kw: k.encode_nvfp4_matmul(w, kw.pop("x", x), y, kw.pop("tokens", 2), **kw),
        "gate_up": lambda **kw: k.encode_ffn_gate_up_silu(w, w, kw.pop("x", x), y, kw.pop("tokens", 2), **kw),
    }
    for name, call in calls.items():
        with pytest.raises(op.MuserCudaError) as e:
            call(norm_weight=torch.ones(256), norm_eps=1e-5)
        assert e.value.status_name == "BAD_ARG", name  # (no context: the library's first check)
        with pytest.raises(op.MuserCudaError, match="norm_weight must be f32"):
            call(norm_weight=torch.ones(256, dtype=torch.float64))
        with pytest.raises(KeyError):
            call(x=x.to(torch.int32))
        for tokens in (2.0, "2", None):
            with pytest.raises(C.ArgumentError):
                call(tokens=tokens)
        with pytest.raises(TypeError):
            call(no_such_argument=1)
    with pytest.raises(IndexError):
        k.encode_quantized_matmul_group([w, w], x, [y, y], 2, epilogues=[None])
    for n in (1, 5, 40):  # (lists longer than the library takes)
        with pytest.raises(op.MuserCudaError):
            k.encode_quantized_matmul_group([w] * n, x, [y] * n, 2)
        with pytest.raises(op.MuserCudaError):
            k.encode_nvfp4_group_prequant([w] * n, x, x, [y] * n, 2)
    with pytest.raises(IndexError):
        k.encode_nvfp4_group_prequant([w], x, x, [y, y], 2)
    with pytest.raises(C.ArgumentError):
        k.quantize_nvfp4_activation(x, "1.0", out=(x, x))
    for eps in ("1e-5", None, x):
        with pytest.raises(Exception) as want:
            C.c_float(eps)
        for call in (lambda: k.encode_head_rms_norm(x, y, eps, 2), lambda: k.encode_fused_norm_residual_rms_norm(x, x, x[0], eps),
                     lambda: k.encode_fused_norm_residual_rms_norm(x, x, x[0], 1e-5, x, x[0], eps),
                     lambda: k.encode_nvfp4_ffn_gate_up_silu_requant(w, w, x, x, 2, eps, out_packed=x, out_scales=x)):
            with pytest.raises(want.type):
                call()
    with pytest.raises(op.MuserCudaError):
        k.quantize_nvfp4_activation(x, 1, norm_weight=torch.ones(256), norm_eps=1e-5, out=(x, x))
    for call in (lambda: k.encode_sigmoid_gate(x, x), lambda: k.encode_head_rms_norm(x, y, 1e-5, 2), lambda: k.encode_nvfp4_prequant(w, x, x, y, 2, residual=y),
                 lambda: k.encode_fused_norm_residual_rms_norm(x, x, x[0], 1e-5),
                 lambda: k.encode_nvfp4_ffn_gate_up_silu_requant(w, w, x, x, 2, 1.0, out_packed=x, out_scales=x)):
        with pytest.raises(op.MuserCudaError):
            call()
    assert k.launches == 0


def test_a_groups_arguments_may_be_what_python_takes_for_them(kern):
    """weights: len() and iteration; outputs: iteration (indexing too for NVFP4 groups); epilogues: epilogues[i], each a mapping
    or None.  The library refuses a call without a context, so BAD_ARG says that the arguments passed."""
    k, w = kern
    x, y = torch.zeros((2, 256)), torch.zeros((2, 16))
    taken = {"norm_weight": torch.ones(256), "norm_eps": 1e-5}
    wrong = {"norm_weight": torch.ones(256, dtype=torch.float64)}

    def group(weights, outputs, epilogues=None):
        k.encode_quantized_matmul_group(weights, x, outputs, 2, epilogues=epilogues)

    def nvfp4(weights, outputs):
        k.encode_nvfp4_group_prequant(weights, x, x, outputs, 2)
    two = {0: w, 1: w}
    for weights, outputs in ((two.values(), (y, y)), ((w, w), {0: y, 1: y}.values()), (collections.deque([w, w]), iter([y, y]))):
        for epilogues in (None, [None, taken], (taken, None), {0: None, 1: taken}, [types.MappingProxyType(taken), collections.UserDict(taken)],
                          collections.defaultdict(lambda: None)):
            with pytest.raises(op.MuserCudaError) as e:
                group(weights, outputs if not hasattr(outputs, "__next__") else iter([y, y]), epilogues)
            assert e.value.status_name == "BAD_ARG" and "norm_weight" not in str(e.value)
    for epilogue in (types.MappingProxyType(wrong), collections.UserDict(wrong)):
        with pytest.raises(op.MuserCudaError, match="norm_weight must be f32"):
            group([w, w], [y, y], [None, epilogue])
    with pytest.raises(op.MuserCudaError, match="norm_weight must be f32"):
        group([w, w], [y, y], {0: None, 1: wrong})
    with pytest.raises(KeyError):
        group([w, w], [y, y], {0: taken})
    for epilogue in (types.MappingProxyType({"no_such_argument": 1}), 5, [1, 2]):
        with pytest.raises(TypeError):
            group([w, w], [y, y], [None, epilogue])
    with pytest.raises(TypeError):
        group((v for v in [w, w]), [y, y])
    for weights in (two.values(), collections.deque([w, w])):
        with pytest.raises(op.MuserCudaError):
            nvfp4(weights, (y, y))
    with pytest.raises(TypeError):
        nvfp4((v for v in [w, w]), [y, y])
    for outputs in (iter([y, y]), {0: y, 1: y}.values()):
        with pytest.raises(TypeError):
            nvfp4([w, w], outputs)
    assert k.launches == 0


def test_the_stream_is_asked_for_on_every_call(kern):
    k, w = kern
    asked = []
    op._call.bind(str(_lib.LIB_PATH), op._TORCH_DTYPE, torch.float32, lambda d: asked.append(d) or 0, lambda d: asked.append(d) or 0, op.MuserCudaError, C.ArgumentError)
    x = torch.zeros((2, 256))
    for device in (0, 3):
        k.ctx.device = device
        with pytest.raises(op.MuserCudaError):
            k.encode_sigmoid_gate(x, x)
    assert asked == [0, 3]


def test_binding_needs_no_more_than_the_library(monkeypatch, tmp_path):
    """A torch without CUDA imports the operators; a Python without headers builds, and calls through ctypes; the extension
    carries the tag of the Python it was built for, so that no other loads it."""
    for hide, want in (("", "_call"), ("sys.modules['muser_b200._call'] = None\n", "_call_py")):
        prog = ("import sys, torch\n"
                "if hasattr(torch._C, '_cuda_getCurrentRawStream'): del torch._C._cuda_getCurrentRawStream\n" + hide +
                f"from muser_b200 import operator as op\nassert op._call.__name__ == 'muser_b200.{want}'\n")
        r = subprocess.run([sys.executable, "-c", prog], capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
    assert importlib.util.find_spec("muser_b200._call").origin.endswith(build.sysconfig.get_config_var("EXT_SUFFIX"))
    monkeypatch.setattr(build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    monkeypatch.setattr(build, "CALL", tmp_path / "none.so")
    assert build.build_call(force=True) is None and not (tmp_path / "none.so").exists()
