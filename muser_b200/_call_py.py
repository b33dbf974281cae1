"""csrc/host_call.c's functions over ctypes, for a Python whose headers were not there when the library was built.

Same names, arguments and refusals, some microseconds a call slower."""
from __future__ import annotations

import ctypes as C
from types import SimpleNamespace

from ._lib import Epilogue, GroupItem, MuserCudaError, lib as _L

_b = SimpleNamespace()


def bind(path, dtypes, f32, raw_stream, stream, error, argument_error) -> None:
    _b.dtypes, _b.f32, _b.stream = dtypes, f32, stream


def _ptr(tensor):
    return tensor.data_ptr() if tensor is not None else None


def epilogue(row_scale=None, residual=None, norm_weight=None, norm_eps=0.0, out_scale=1.0, softcap=0.0, all_reduce=False):
    """muser_cuda_epilogue; `norm_weight` (f32 [n_in], device) fuses rms_norm_mul(x, eps, norm_weight) in front,
    `out_scale` / `softcap` the LM-head tail y <- softcap * tanh(y * out_scale / softcap) behind."""
    if row_scale is None and residual is None and norm_weight is None and out_scale == 1.0 and softcap == 0.0 and not all_reduce:
        return None
    if norm_weight is not None and norm_weight.dtype != _b.f32:
        raise MuserCudaError(1, "norm_weight must be f32")
    return Epilogue(_ptr(row_scale), _ptr(residual), 0, float(norm_eps), _ptr(norm_weight), float(out_scale), float(softcap), int(bool(all_reduce)))


def _ref(ep):
    return C.byref(ep) if ep else None


def quantized_matmul(ctx, device, w, x, y, tokens, row_scale, residual, norm_weight, norm_eps, out_scale, softcap, all_reduce):
    ep = epilogue(row_scale, residual, norm_weight, norm_eps, out_scale, softcap, all_reduce)
    return _L.muser_cuda_quantized_matmul(ctx._h, w._h, x.data_ptr(), _b.dtypes[x.dtype], y.data_ptr(), _b.dtypes[y.dtype], tokens, _ref(ep), _b.stream(device))


def nvfp4_matmul(ctx, device, w, x, y, tokens, row_scale, residual, norm_weight, norm_eps, out_scale, softcap):
    ep = epilogue(row_scale, residual, norm_weight, norm_eps, out_scale, softcap)
    return _L.muser_cuda_nvfp4_matmul(ctx._h, w._h, x.data_ptr(), _b.dtypes[x.dtype], y.data_ptr(), _b.dtypes[y.dtype], tokens, _ref(ep), _b.stream(device))


def quantized_matmul_group(ctx, device, weights, x, outputs, tokens, epilogues):
    n = len(weights)
    items, keep = (GroupItem * n)(), []
    for i, (w, y) in enumerate(zip(weights, outputs)):
        ep = epilogue(**(epilogues[i] or {})) if epilogues else None
        keep.append(ep)
        items[i].w, items[i].y, items[i].y_dtype = getattr(w._h, "value", None), y.data_ptr(), _b.dtypes[y.dtype]
        items[i].epilogue = C.pointer(ep) if ep is not None else None
    return _L.muser_cuda_quantized_matmul_group(ctx._h, items, n, x.data_ptr(), _b.dtypes[x.dtype], tokens, _b.stream(device))


def gate_up_silu(ctx, device, gate, up, x, y, tokens, norm_weight, norm_eps):
    ep = epilogue(None, None, norm_weight, norm_eps)
    return _L.muser_cuda_ffn_gate_up_silu(ctx._h, gate._h, up._h, x.data_ptr(), _b.dtypes[x.dtype], y.data_ptr(), _b.dtypes[y.dtype], tokens, _ref(ep), _b.stream(device))


def nvfp4_prequant(ctx, device, w, packed, scales, y, tokens, row_scale, residual):
    ep = epilogue(row_scale, residual)
    return _L.muser_cuda_nvfp4_matmul_prequant(ctx._h, w._h, packed.data_ptr(), scales.data_ptr(), y.data_ptr(), _b.dtypes[y.dtype], tokens, _ref(ep), _b.stream(device))


def nvfp4_group_prequant(ctx, device, weights, packed, scales, outputs, tokens):
    n = len(weights)
    ws = (C.c_void_p * n)(*[getattr(w._h, "value", None) for w in weights])
    ys = (C.c_void_p * n)(*[y.data_ptr() for y in outputs])
    return _L.muser_cuda_nvfp4_matmul_group_prequant(ctx._h, ws, n, packed.data_ptr(), scales.data_ptr(), ys, _b.dtypes[outputs[0].dtype], tokens, _b.stream(device))


def nvfp4_gate_up_requant(ctx, device, gate, up, packed, scales, tokens, out_input_scale_inv, out_packed, out_scales):
    return _L.muser_cuda_nvfp4_ffn_gate_up_silu_requant(ctx._h, gate._h, up._h, packed.data_ptr(), scales.data_ptr(), tokens, C.c_float(out_input_scale_inv),
                                                        out_packed.data_ptr(), out_scales.data_ptr(), _b.stream(device))


def quantize_activation(ctx, device, x, tokens, n_in, input_scale_inv, norm_weight, norm_eps, packed, scales):
    head = (ctx._h, x.data_ptr(), _b.dtypes[x.dtype], tokens, n_in)
    tail = (input_scale_inv, packed.data_ptr(), scales.data_ptr(), _b.stream(device))
    if norm_weight is None:
        return _L.muser_cuda_quantize_nvfp4_activation(*head, *tail)
    return _L.muser_cuda_rmsnorm_quantize_nvfp4_activation(*head, norm_weight.data_ptr(), float(norm_eps), *tail)


def norm_residual_norm(ctx, device, hidden, src, output, weight1, weight2, tokens, n, eps1, eps2):
    return _L.muser_cuda_fused_norm_residual_rms_norm(ctx._h, hidden.data_ptr(), src.data_ptr(), _ptr(output), weight1.data_ptr(), _ptr(weight2), tokens, n,
                                                      C.c_float(eps1), C.c_float(eps2), _b.stream(device))


def sigmoid_gate(ctx, device, x, gate, count):
    return _L.muser_cuda_sigmoid_gate(ctx._h, x.data_ptr(), gate.data_ptr(), count, _b.stream(device))


def head_rms_norm(ctx, device, x, weight, eps, tokens, heads, head_dim):
    return _L.muser_cuda_head_rms_norm(ctx._h, x.data_ptr(), weight.data_ptr(), C.c_float(eps), tokens, heads, head_dim, _b.stream(device))
