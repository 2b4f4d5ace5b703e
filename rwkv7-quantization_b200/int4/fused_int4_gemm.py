"""INT4 GEMV entry points with the names of the reference's int4/fused_int4_gemm.py.  The reference's Triton
kernels take one activation vector [K]; these also take [M, K] (any M, processed 16 rows per launch)."""
from __future__ import annotations

import os

import torch

import rwkvq_abi as abi
from int4.int4_ops import _rows_f16, _run_rows, _f32

TRITON_AVAILABLE = False      # kept for importers; nothing here uses Triton


def _squeeze(out: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    return out.reshape(-1) if x.dim() == 1 else out.reshape(*x.shape[:-1], out.shape[-1])


def linear_int4_gemv_triton(x: torch.Tensor, packed: torch.Tensor, scale: torch.Tensor) -> torch.Tensor:
    """Per-tensor INT4 GEMV (int4/fused_int4_gemm.py:174-182)."""
    from int4.int4_ops import linear_int4_per_tensor
    return _squeeze(linear_int4_per_tensor(x.reshape(-1, x.shape[-1]), {"packed": packed, "scale": scale}), x)


def linear_int4_affine_gemv_triton(x, packed, mx, rx, my, ry) -> torch.Tensor:
    """MM4 GEMV (int4/fused_int4_gemm.py:185-194)."""
    from int4.int4_ops import linear_int4_affine
    info = {"packed": packed, "mx": mx, "rx": rx, "my": my, "ry": ry, "m_orig": x.shape[-1]}
    return _squeeze(linear_int4_affine(x.reshape(-1, x.shape[-1]), info), x)


_slices_cache: dict = {}


def _ksplit_slices(m: int, n: int, k: int) -> int:
    sl = _slices_cache.get((m, n, k))
    if sl is None:
        sl = _slices_cache[(m, n, k)] = int(abi.lib().rwkvq_gemv_int4_ksplit_slices(m, n, k))
    return sl


TC_ROWS = 17            # rows from which the tensor-core GEMM takes over from the decode kernel (which re-reads the weights every 16 rows)
TC_ROWS_LARGE = 14      # ... against matrices of this many weights, whose stream hides the GEMM's second launch
TC_LARGE = 1 << 25
TC_ROWS_WIDE = 12       # ... and against this many weight rows, where its row tiles alone fill the chip
TC_WIDE_N = 16384
TC_MIN_N = 512


def _takes_tc(m: int, n: int, k: int) -> bool:
    """Measured, us, decode kernel / tensor-core GEMM.  16 and 17 rows: [4096, 4096] 9.9 / 10.6 and 13.8 / 10.6, [2048, 2048] 5.5 /
    7.7 and 8.2 / 7.7, [512, 4096] 6.8 / 8.3 and 10.1 / 8.2 (fewer weight rows were not measured).  12, 14 and 16 rows: [8192,
    2048] 7.4 / 10.1, 7.8 / 10.1, 8.2 / 10.1; [10240, 2560] 10.6 / 12.1, 11.1 / 12.2, 11.6 / 12.1; [8192, 4096] 13.6 / 13.8, 14.3 / 13.8,
    14.2 / 13.8; [14336, 3584] 15.7 / 16.2, 16.5 / 16.0, 16.9 / 15.9; [4096, 16384] 20.1 / 20.4, 21.1 / 20.5, 21.3 / 20.9; [16384, 4096] 18.6 /
    18.1, 19.1 / 18.1, 20.0 / 18.1 (9 rows 16.9 / 17.9)."""
    first = TC_ROWS_WIDE if n >= TC_WIDE_N else (TC_ROWS_LARGE if n * k >= TC_LARGE else TC_ROWS)
    return m >= first and n >= TC_MIN_N and k % 128 == 0


def _groupwise_tc(x, packed, scales, zeros):
    """Group 128, many rows: rwkvq_tc_gemm_int4_group, or None where its alignment rules do not hold.  fp16 and bf16
    activations go in as they are (the kernel that permutes them also rounds bf16 to fp16)."""
    n, k = packed.shape[0], packed.shape[1] * 2
    if packed.stride(1) != 1 or packed.stride(0) % 16 or (packed.data_ptr() | scales.data_ptr() | (0 if zeros is None else zeros.data_ptr())) % 16:
        return None
    x2 = x if x.dim() == 2 else x.reshape(-1, k)
    if x2.dtype not in (torch.float16, torch.bfloat16):
        x2 = x2.to(torch.float16)
    x2 = x2.contiguous()
    if x2.data_ptr() % 16:
        x2 = x2.clone()
    abi.require_device()
    if not x2.is_cuda:
        raise RuntimeError("rwkvq: INT4 / INT8 projections run on the GPU only (no CPU fallback)")
    m, dev = x2.shape[0], x2.device
    out = torch.empty((m, n), dtype=torch.float16, device=dev)
    ws = torch.empty(abi.wa16_workspace_bytes(m, n, k, 4, dev), dtype=torch.uint8, device=dev)
    abi.call("rwkvq_tc_gemm_int4_group", x2.data_ptr(), abi.dtype_code(x2), k, packed.data_ptr(), packed.stride(0), scales.data_ptr(),
             abi.ptr(zeros), out.data_ptr(), n, m, n, k, ws.data_ptr(), ws.numel(), abi.stream_ptr())
    abi.after_call()
    return out


def _groupwise_rows(x, packed, scales, zeros, group_size: int) -> torch.Tensor:
    n, k = packed.shape[0], packed.shape[1] * 2
    given = scales
    if (group_size == 128 and scales.dtype != torch.float16 and x.shape[-1] == k and k and _takes_tc(x.numel() // k, n, k)
            and os.environ.get("RWKVQ_INT4", "fast") != "generic"):
        out = _groupwise_tc(x, packed, _f32(scales, x.device), None if zeros is None else _f32(zeros, x.device))
        if out is not None:
            return out
    x2 = _rows_f16(x, k)
    dev = x2.device
    scale_f16 = scales.dtype == torch.float16
    scales = scales.to(dev).contiguous() if scale_f16 else _f32(scales, dev)
    zeros_given, zeros = zeros, None if zeros is None else _f32(zeros, dev)
    if (scales is not given or zeros is not zeros_given) and x2.is_cuda:          # copies made just now: in front of the projection
        abi.order_copies((scales, given), *(() if zeros is None else ((zeros, zeros_given),)))
    generic = lambda xc, oc, m: abi.call(
        "rwkvq_gemv_int4_group_generic", xc.data_ptr(), k, packed.data_ptr(), packed.stride(0), scales.data_ptr(),
        abi.ptr(zeros), int(scale_f16), group_size, oc.data_ptr(), n, m, n, k, abi.stream_ptr())
    if os.environ.get("RWKVQ_INT4", "fast") == "generic" or group_size not in (128, 256) or k % 128:
        return _run_rows(x2, n, generic)
    if (group_size == 128 and not scale_f16 and k % 512 == 0 and scales.data_ptr() % 16 == 0
            and (zeros is None or zeros.data_ptr() % 16 == 0) and os.environ.get("RWKVQ_INT4_KSPLIT", "1") != "0"):
        # blocks too large to sit beside a deep weight ring (many rows, long rows): K in slices, fp32 partial sums, one
        # pass over the weights instead of one per block of rows
        def split(xc, oc, m):
            sl = _ksplit_slices(m, n, k)
            if sl > 1:
                ws = abi.plain_scratch(sl * m * n * 4, dev)
                abi.call("rwkvq_gemv_int4_group_ksplit", xc.data_ptr(), k, packed.data_ptr(), packed.stride(0), scales.data_ptr(),
                         abi.ptr(zeros), oc.data_ptr(), n, m, n, k, ws.data_ptr(), ws.numel(), abi.stream_ptr())
            else:
                abi.call("rwkvq_gemv_int4_group", xc.data_ptr(), k, packed.data_ptr(), packed.stride(0), scales.data_ptr(),
                         abi.ptr(zeros), 0, group_size, oc.data_ptr(), n, m, n, k, abi.stream_ptr())
        if _ksplit_slices(min(16, x2.shape[0]), n, k) >= 1:
            return _run_rows(x2, n, split, 16)
    # the streaming kernel keeps its rows of activations in shared memory: as many rows per launch as fit
    rows = 16
    while rows > 1 and abi.lib().rwkvq_gemv_int4_group_smem_bytes(rows, k) > 200 * 1024:
        rows //= 2
    if abi.lib().rwkvq_gemv_int4_group_smem_bytes(rows, k) > 200 * 1024:
        return _run_rows(x2, n, generic)
    return _run_rows(x2, n, lambda xc, oc, m: abi.call(
        "rwkvq_gemv_int4_group", xc.data_ptr(), k, packed.data_ptr(), packed.stride(0), scales.data_ptr(),
        abi.ptr(zeros), int(scale_f16), group_size, oc.data_ptr(), n, m, n, k, abi.stream_ptr()), rows)


def linear_int4_groupwise_gemv_triton(x, packed, scales, zeros, group_size: int) -> torch.Tensor:
    """Group-wise INT4 GEMV (int4/fused_int4_gemm.py:197-207)."""
    return _squeeze(_groupwise_rows(x.reshape(-1, x.shape[-1]), packed, scales, zeros, group_size), x)
