"""The tiled W8A8 GEMMs where the CTA-pair form and the single-CTA form divide the work differently: the same bits from both
(both add K in the same order), for every epilogue (plain, through bf16, relu^2 with its maxima, per-row scales, raw
accumulators), r/k/v in one launch, ragged rows and columns.  The form is chosen at the first launch of a process, so the
pairs are switched off in a child process."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# (rows, N, K): one and several waves, remainders of the 128- and 256-row tiles, N no multiple of 16 / 256
SIZES = [(129, 16384, 1024), (384, 16384, 512), (717, 10240, 2560), (300, 9000, 2064), (1025, 4104, 4096), (513, 4096, 16384)]


def results():
    import rwkvq_abi as abi
    out = []
    dev, st = "cuda", abi.stream_ptr()
    for m, n, k in SIZES:
        g = torch.Generator(device=dev).manual_seed(m + n)
        a8 = torch.randint(-127, 128, (3, m, k), generator=g, device=dev, dtype=torch.int8)
        w8 = torch.randint(-127, 128, (3, n, k), generator=g, device=dev, dtype=torch.int8)
        af = (torch.randn((3, m, k), generator=g, device=dev)).to(torch.float8_e4m3fn)
        wf = (torch.randn((3, n, k), generator=g, device=dev)).to(torch.float8_e4m3fn)
        rs = torch.rand(m, generator=g, device=dev) + 0.5
        sc = torch.rand(n, generator=g, device=dev) * 1e-4 + 1e-5
        amax = torch.full((3,), 3.0, device=dev)
        ws = abi.workspace(128, n, k, 3, torch.device(dev))
        ldo = n + 8
        y = lambda: torch.zeros((m, ldo), dtype=torch.float16, device=dev)  # noqa: E731
        for flags in (0, abi.FLAG_OUT_VIA_BF16, abi.FLAG_WSCALE_PER_ROW):
            o = y()
            abi.call("rwkvq_tc_gemm_fp8", af.data_ptr(), k, amax.data_ptr(), 1, wf.data_ptr(), k, sc.data_ptr(), o.data_ptr(), ldo, m, n, k, abi.DIV_IEEE,
                     flags, ws.data_ptr(), ws.numel(), st)
            out.append(o)
        for flags in (0, abi.FLAG_OUT_VIA_BF16 | abi.FLAG_AMAX_AFTER_BF16):
            o, h = y(), torch.zeros(2, device=dev)
            abi.call("rwkvq_tc_gemm_fp8_relu2", af.data_ptr(), k, amax.data_ptr(), 1, wf.data_ptr(), k, sc.data_ptr(), o.data_ptr(), ldo, m, n, k, abi.DIV_IEEE,
                     flags, h.data_ptr(), ws.data_ptr(), ws.numel(), st)
            out += [o, h]
            assert float(h[0]) == float((o.to(torch.bfloat16) if flags else o).max())
        for acc in (None, torch.zeros((m, n), dtype=torch.int32, device=dev)):
            o = y()
            abi.call("rwkvq_tc_gemm_int8", a8.data_ptr(), k, rs.data_ptr(), w8.data_ptr(), k, sc.data_ptr(), o.data_ptr(), ldo, abi.ptr(acc), n, m, n, k, 0,
                     ws.data_ptr(), ws.numel(), st)
            out += [o] if acc is None else [o, acc]
        want = (a8[0].double() @ w8[0].double().t()).to(torch.int32)
        assert torch.equal(out[-1], want)
        o, h = y(), torch.zeros(m, device=dev)
        abi.call("rwkvq_tc_gemm_int8_relu2", a8.data_ptr(), k, rs.data_ptr(), w8.data_ptr(), k, sc.data_ptr(), o.data_ptr(), ldo, m, n, k, 0, h.data_ptr(),
                 ws.data_ptr(), ws.numel(), st)
        out += [o, h]
        assert torch.equal(h, o.float().amax(1))
        os_ = [y() for _ in range(6)]
        abi.call("rwkvq_tc_gemm_fp8_rkv", *(t.data_ptr() for t in af), k, amax.data_ptr(), 1, *(t.data_ptr() for t in wf), k, *([sc.data_ptr()] * 3),
                 *(t.data_ptr() for t in os_[:3]), ldo, m, n, k, abi.DIV_IEEE, 0, ws.data_ptr(), ws.numel(), st)
        abi.call("rwkvq_tc_gemm_int8_rkv", *(t.data_ptr() for t in a8), k, *([rs.data_ptr()] * 3), *(t.data_ptr() for t in w8), k, *([sc.data_ptr()] * 3),
                 *(t.data_ptr() for t in os_[3:]), ldo, m, n, k, 0, ws.data_ptr(), ws.numel(), st)
        out += os_
        torch.cuda.synchronize()
        assert abi.device_status() == 0
    return [t.cpu() for t in out]


def test_pairs_and_single_ctas_give_the_same_bits(tmp_path):
    f = str(tmp_path / "single.pt")
    code = f"import sys; sys.path[:0] = [{os.path.join(ROOT, 'rwkv7-quantization_b200')!r}, {os.path.join(ROOT, 'tests')!r}]\n" \
           f"import torch, test_tiled_gemm_gpu as t; torch.save(t.results(), {f!r})"
    subprocess.run([sys.executable, "-c", code], check=True, env=dict(os.environ, RWKVQ_TC2="0"), timeout=300)
    for a, b in zip(results(), torch.load(f)):
        assert torch.equal(a, b)
