"""GEMMs on CTA pairs where every pair works on several tiles and each tile goes round the ring of operand stages more than once:
positions and phases carried from tile to tile, stages that are requested ahead for the next tile, scale columns and accumulators
that change owner between tiles, and what a pair leaves behind for the launch that follows.

Bound per element: half an fp16 ulp of the result (2^-11 relative, 2^-25 below the normal range) plus 2^-16 of the magnitudes' sum for
the 32-bit sums (sqrt(K) * 2^-23 at K = 16384)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def gen(seed, shape, std=1.0):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * std


def check(out, xd, parts):
    ref = sum(xd @ p.t() for p in parts)
    mag = sum(xd.abs() @ p.abs().t() for p in parts)
    err = (out.double() - ref).abs()
    bound = ref.abs() * 2.0 ** -11 + 2.0 ** -25 + mag * 2.0 ** -16
    assert bool((err <= bound).all()), float((err / bound).max())


def int4(n, k, zeros):
    from int4 import int4_ops, quantize_int4
    info = {a: b.cuda() if torch.is_tensor(b) else b for a, b in quantize_int4.quantize_to_int4_groupwise(gen(n, (n, k), k ** -0.5).cpu(), 128).items()}
    if not zeros:
        info["zeros"] = -8.0 * info["scales"]
    s, z = (info[v].double().repeat_interleave(128, 1) for v in ("scales", "zeros"))
    parts = [int4_ops.unpack_int4(info["packed"]).double() * s, z]
    if not zeros:
        del info["zeros"]
    info["qtype"] = "int4_groupwise"
    return lambda x: int4_ops.linear_int4(x, info), lambda x: x.double(), parts


def int8(n, k):
    from int8 import int8_ops, quantize_int8
    q, s = quantize_int8.quantize_to_int8_per_tensor(gen(n, (n, k), k ** -0.5))
    info = {"weight": q.cuda(), "tensor_scale": s.cuda(), "qtype": "int8_per_tensor"}
    return lambda x: int8_ops.linear_int8(x, info), lambda x: x.double(), [info["weight"].double() * info["tensor_scale"].double()]


def nvfp4(n, k):
    import nvfp4_ops as nf
    info = nf.quantize_to_nvfp4(gen(n, (n, k), k ** -0.5))

    def rows(x):
        codes, bs, pts = nf.quantize_activations_nvfp4(x)
        return nf.dequantize_nvfp4({"weight": codes, "block_scale": bs, "tensor_scale": pts}).double()
    return lambda x: nf.linear_nvfp4(x, info), rows, [nf.dequantize_nvfp4(info).double()]


def w8a8(scheme, n, k):
    import fused_fp8_gemm as f
    w = gen(n, (n, k), k ** -0.5)
    s = w.abs().max() / (448 if scheme == "fp8" else 127)
    info = {"weight": (w / s).to(torch.float8_e4m3fn) if scheme == "fp8" else (w / s).round().to(torch.int8), "tensor_scale": s, "qtype": scheme}
    return lambda x: f.linear_quantized_fused(x, info), None, None


@pytest.mark.parametrize("kind,m,n,k", [("int4", 1000, 16384, 1152), ("int4", 600, 10000, 2176), ("int4_symmetric", 1000, 16384, 1152), ("int4_symmetric", 600, 10000, 2176),
                                        ("w8a16", 1000, 16384, 1152), ("w8a16", 600, 10000, 2176), ("nvfp4", 1030, 5000, 1792), ("nvfp4", 2048, 4096, 4096),
                                        ("fp8", 1030, 10240, 2560), ("int8", 1030, 10240, 2560)])
def test_several_tiles_per_pair(kind, m, n, k, monkeypatch):
    import rwkvq_abi as abi
    monkeypatch.setenv("RWKVQ_NF4_BN", "pair")
    lib, slices = abi.lib(), 1
    if kind.startswith("int4") or kind == "w8a16":
        form = lib.rwkvq_tc_gemm_wa16_form(m, n, k, 8 if kind == "w8a16" else 4)
        assert form % 1000 in (1000 - 128, 1000 - 256)                  # a pair's tile of 128 or 256 tokens
        slices, tokens, width = (form + 999) // 1000, 1000 - form % 1000, 256
    elif kind == "nvfp4":
        assert lib.rwkvq_tc_gemm_nvfp4_form(m, n, k) == abi.TC_FORM_PAIRS
        tokens = width = 256
    else:
        code = abi.LINEAR_FP8 if kind == "fp8" else abi.LINEAR_INT8
        assert lib.rwkvq_tc_gemm_form(code, 1, m, n, k, 0) == abi.TC_FORM_PAIRS
        tokens, width = 256, lib.rwkvq_tc_gemm_pair_width(code, 1, m, n, k)
    tiles = -(-m // tokens) * -(-n // width) * slices
    assert tiles > torch.cuda.get_device_properties(0).multi_processor_count // 2
    run, rows, parts = int4(n, k, kind == "int4") if kind.startswith("int4") else int8(n, k) if kind == "w8a16" else nvfp4(n, k) if kind == "nvfp4" else w8a8(kind, n, k)
    xs = [gen(m + i, (m, k)).half() for i in range(2)]
    want = []
    for x in xs:
        want.append(run(x))
        torch.cuda.synchronize()
        if parts:
            check(want[-1], rows(x), parts)
    # launches that follow one another without a gap give what each gives alone
    got = [run(xs[i & 1]) for i in range(24)]
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[i & 1]) for i, y in enumerate(got))
    assert abi.device_status() == 0 and abi.workspace_status(abi.workspace(1, 1, 1, 1, torch.device("cuda", 0))) == 0
