"""The tiled W8A8 GEMMs where the CTA-pair form and the single-CTA form divide the work differently: the same bits from both
(both add K in the same order), for every epilogue (plain, through bf16, relu^2 with its maxima, per-row scales, raw
accumulators), r/k/v in one launch, ragged rows and columns.  The form is chosen at the first launch of a process, so the
pairs are forced and switched off in child processes."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# (rows, N, K): one and several waves, remainders of the 128- and 256-row tiles, N no multiple of 16 / 256
SIZES = [(129, 16384, 1024), (384, 16384, 512), (717, 10240, 2560), (300, 9000, 2064), (1025, 4104, 4096), (513, 4096, 16384)]


def forms():
    import rwkvq_abi as abi
    return [int(abi.lib().rwkvq_tc_gemm_form(kind, nmat, m, n, k, 0)) for m, n, k in SIZES for kind in (abi.LINEAR_FP8, abi.LINEAR_INT8) for nmat in (1, 3)]


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


@pytest.mark.parametrize("scheme", ["fp8", "int8"])
@pytest.mark.parametrize("m,k,f,n", [(9, 1024, 4096, 1024), (13, 4096, 16384, 4096), (32, 768, 3072, 768), (20, 2560, 10240, 2560), (5, 4096, 16384, 4096),
                                     (40, 2048, 8192, 512), (200, 1024, 4096, 1024), (1, 1024, 4096, 1024), (6, 768, 3072, 768)])
def test_ffn_pair_equals_its_three_steps(scheme, m, k, f, n):
    """The FFN pair (relu_square in an epilogue or in the quantizer that follows) equals its three steps bit for bit, NaN and infinity included."""
    import fused_fp8_gemm as ff
    g = torch.Generator(device="cuda").manual_seed(m + k)
    mk = lambda a, b: (torch.randn((a, b), generator=g, device="cuda") * b ** -0.5 * 100).round().clamp(-127, 127)  # noqa: E731
    dt = torch.float8_e4m3fn if scheme == "fp8" else torch.int8
    info = [{"weight": mk(a, b).to(dt), "tensor_scale": torch.tensor(0.01, device="cuda"), "qtype": scheme} for a, b in ((f, k), (n, f))]
    pair = ff.ffn_relu2_fp8 if scheme == "fp8" else ff.ffn_relu2_int8
    for special in (None, float("inf"), float("nan")):
        x = torch.randn((m, k), generator=g, device="cuda").half()
        if special is not None:
            x[m // 2, 3] = special
        hid = ff.linear_quantized_fused(x, info[0])
        hid = (hid.float().clamp_(min=0.0) ** 2).to(torch.float16)
        want = ff.linear_quantized_fused(hid, info[1])
        got = pair(x, info[0], info[1])
        assert torch.equal(got.view(torch.int16), want.view(torch.int16)), special
        assert torch.equal(pair(x, info[0], info[1], return_hidden=True)[0].view(torch.int16), want.view(torch.int16))


def test_pairs_and_single_ctas_give_the_same_bits(tmp_path):
    """This process (the cost rule picks), one that forces the pairs and one without them; each reports the form it takes."""
    import rwkvq_abi as abi
    runs = {}
    for mode, form in (("force", abi.TC_FORM_PAIRS), ("0", abi.TC_FORM_TILED)):
        f = str(tmp_path / f"{mode}.pt")
        code = f"import sys; sys.path[:0] = [{os.path.join(ROOT, 'rwkv7-quantization_b200')!r}, {os.path.join(ROOT, 'tests')!r}]\n" \
               f"import torch, test_tiled_gemm_gpu as t; torch.save((t.forms(), t.results()), {f!r})"
        subprocess.run([sys.executable, "-c", code], check=True, env=dict(os.environ, RWKVQ_TC2=mode), timeout=300)
        forms_, runs[mode] = torch.load(f)
        # a matrix whose K is long keeps the cluster kernel at few rows; these sizes have none
        assert forms_ == [form] * len(forms_), (mode, forms_)
    here = results()
    assert len(here) == len(runs["force"]) == len(runs["0"])
    for a, b, c in zip(here, runs["force"], runs["0"]):
        assert torch.equal(a, b) and torch.equal(a, c)


@pytest.mark.parametrize("offset", [8, 16])
@pytest.mark.parametrize("m,n,k", [(40, 512, 512), (200, 1024, 512), (600, 2048, 512), (1100, 4096, 256)])
def test_results_in_a_column_range(m, n, k, offset):
    """Rows that start on 16- and on 32-byte boundaries (the epilogue's store widths) give the same bits as a result of its own, and
    leave the columns around them alone."""
    import fused_fp8_gemm as f
    import nvfp4_ops
    import rwkvq_abi as abi
    g = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn((m, k), generator=g, device="cuda").half()
    w = torch.randn((n, k), generator=g, device="cuda") * k ** -0.5
    s = w.abs().max()
    for info in ({"weight": (w / s * 448).to(torch.float8_e4m3fn), "tensor_scale": s / 448, "qtype": "fp8"},
                 {"weight": (w / s * 127).round().to(torch.int8), "tensor_scale": s / 127, "qtype": "int8"}, nvfp4_ops.quantize_to_nvfp4(w)):
        want = f.linear_quantized_fused(x, info)
        wide = torch.full((m, n + 32), 7.0, dtype=torch.float16, device="cuda")
        with abi.output_into(wide[:, offset:offset + n]):
            f.linear_quantized_fused(x, info)
        assert torch.equal(wide[:, offset:offset + n], want)
        assert bool((wide[:, :offset] == 7).all()) and bool((wide[:, offset + n:] == 7).all())


def tile_widths():
    """Every width of a pair's tile (INT8: multiples of 32, the others leave it to the plan) against the widest: halves of an odd number of 16-column pieces, columns past the last tile."""
    import rwkvq_abi as abi
    global SIZES
    sizes = [(129, 1000, 400), (300, 4104, 1040), (517, 2560, 768)]
    for SIZES in ([s] for s in sizes):
        want = None
        for bn in range(256, 127, -16):
            os.environ["RWKVQ_TC2_BN"] = str(bn)
            for (m, n, k), kind in ((s, c) for s in SIZES for c in (abi.LINEAR_FP8, abi.LINEAR_INT8)):
                assert bn % 32 and kind == abi.LINEAR_INT8 or abi.lib().rwkvq_tc_gemm_pair_width(kind, 1, m, n, k) == bn
            got = results()
            want = got if want is None else want
            assert all(torch.equal(a, b) for a, b in zip(got, want)), (SIZES, bn)
    assert abi.device_status() == 0


def test_pair_tiles_of_every_width():
    code = f"import sys; sys.path[:0] = [{os.path.join(ROOT, 'rwkv7-quantization_b200')!r}, {os.path.join(ROOT, 'tests')!r}]\n" \
           "import test_tiled_gemm_gpu as t; t.tile_widths()"
    subprocess.run([sys.executable, "-c", code], check=True, env=dict(os.environ, RWKVQ_TC2="force"), timeout=300)
