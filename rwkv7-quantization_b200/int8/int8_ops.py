"""Stand-alone INT8 weight detection, loading and W8A16 projections (drop-in for the reference's int8/int8_ops.py).

Weight-info dicts (int8/int8_ops.py:22-41):
    per_tensor : {"weight" int8 [N,K], "tensor_scale", "qtype": "int8_per_tensor"}
    affine     : {"weight" uint8 [N,K], "mx", "rx", "my", "ry", "qtype": "int8_affine"}
"""
from __future__ import annotations

import torch

import rwkvq_abi as abi
from int4.int4_ops import _rows_f16, _run_rows, _f32


def is_int8_weight(z: dict, key: str) -> bool:
    return (key + ".int8_weight" in z) or (key + ".int8_w_u8" in z)


def load_int8_weight(z: dict, key: str, dev: str = "cuda"):
    if key + ".int8_weight" in z:
        return {"weight": z[key + ".int8_weight"].to(dev), "tensor_scale": z[key + ".int8_scale"].to(dev),
                "qtype": "int8_per_tensor"}
    if key + ".int8_w_u8" in z:
        info = {"weight": z[key + ".int8_w_u8"].to(dev), "qtype": "int8_affine"}
        info.update({n: z[f"{key}.int8_{n}"].to(dev) for n in ("mx", "rx", "my", "ry")})
        return info
    raise KeyError(f"No INT8 weight found for key: {key}")


TC_ROWS = 17        # rows from which the tensor-core GEMM takes over (the decode kernel takes 16 per pass over the weights)
TC_MIN_N = 512
_streams: dict = {}


def _takes_tc(m: int, n: int, k: int) -> bool:
    """Measured, us, decode kernel / tensor-core GEMM: [4096, 4096] 16 rows 6.5 / 9.9, [16384, 4096] 16 rows 17.2 / 19.3,
    [512, 4096] 16 rows 4.3 / 6.6.  Blocks too large for the decode kernel's shared memory ([2560, 10240] from 7 rows,
    [4096, 16384] from 5) run the GEMM, 11.7 and 20.4, not the row kernel, 94 and 117."""
    if n < TC_MIN_N or k % 16:
        return False
    if m >= TC_ROWS:
        return True
    fits = _streams.get((m, k))
    if fits is None:
        fits = _streams[(m, k)] = m < 1 or bool(abi.lib().rwkvq_gemv_int8_w8a16_streams(m, k))
    return not fits


def _shaped(out, x, n: int, out_dtype):
    return out if x.dim() == 2 and out.dtype is out_dtype else out.to(out_dtype).reshape(*x.shape[:-1], n)


def _tensor_core(x2, w, scale):
    abi.require_device()
    if not x2.is_cuda:
        raise RuntimeError("rwkvq: INT4 / INT8 projections run on the GPU only (no CPU fallback)")
    (m, k), n, dev = x2.shape, w.shape[0], x2.device
    out = torch.empty((m, n), dtype=torch.float16, device=dev)
    ws = torch.empty(abi.wa16_workspace_bytes(m, n, k, 8, dev), dtype=torch.uint8, device=dev)
    abi.call("rwkvq_tc_gemm_int8_w8a16", x2.data_ptr(), k, w.data_ptr(), w.stride(0), scale.data_ptr(), out.data_ptr(), n, m, n, k,
             ws.data_ptr(), ws.numel(), abi.stream_ptr())
    abi.after_call()
    return out


def linear_int8_per_tensor(x, weight_info, out_dtype=torch.float16):
    """W8A16 projection: fp16 activations times int8 weights times the scale (int8/int8_ops.py:48-78)."""
    w0, s0 = weight_info["weight"], weight_info["tensor_scale"]
    w = w0.contiguous()
    n, k = w.shape
    x2 = _rows_f16(x, k)
    scale = _f32(s0.reshape(1), x2.device)
    if w is not w0 or scale.data_ptr() != s0.data_ptr():         # copies made just now: in front of the projection
        abi.order_copies((w, w0), (scale, s0))
    if w.data_ptr() % 16 == 0 and _takes_tc(x2.shape[0], n, k):
        return _shaped(_tensor_core(x2, w, scale), x, n, out_dtype)
    out = _run_rows(x2, n, lambda xc, oc, m: abi.call(
        "rwkvq_gemv_int8_w8a16", xc.data_ptr(), k, w.data_ptr(), w.stride(0), scale.data_ptr(), oc.data_ptr(), n, m, n, k,
        abi.stream_ptr()))
    return _shaped(out, x, n, out_dtype)


def linear_int8_affine(x, weight_info, out_dtype=torch.float16):
    """MM8 projection (int8/int8_ops.py:81-110)."""
    w = weight_info["weight"].contiguous()
    n, k = w.shape
    x2 = _rows_f16(x, k)
    mx, rx, my, ry = (_f32(weight_info[v], x2.device) for v in ("mx", "rx", "my", "ry"))
    out = _run_rows(x2, n, lambda xc, oc, m: abi.call(
        "rwkvq_gemv_int8_affine", xc.data_ptr(), k, w.data_ptr(), w.stride(0), mx.data_ptr(), rx.data_ptr(), my.data_ptr(),
        ry.data_ptr(), oc.data_ptr(), n, m, n, k, abi.stream_ptr()))
    return out.to(out_dtype).reshape(*x.shape[:-1], n)


def linear_int8(x, weight_info, out_dtype=torch.float16):
    qtype = weight_info["qtype"]
    if qtype == "int8_per_tensor":
        return linear_int8_per_tensor(x, weight_info, out_dtype)
    if qtype == "int8_affine":
        return linear_int8_affine(x, weight_info, out_dtype)
    raise ValueError(f"Unknown INT8 qtype: {qtype}")
