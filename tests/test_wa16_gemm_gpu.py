"""GPU parity of the tensor-core weight-only GEMMs (gemm_wa16.cu) against the oracle's dequantized weights in 64 bits.

Bound per element: half an fp16 ulp of the result (2^-11 relative, 2^-25 below the normal range) plus the error of 32-bit
sums.  A sum of K fp32 terms errs by at most K * 2^-23 times the sum of their magnitudes when every addition truncates;
roundings of either sign grow with sqrt(K): 2^-16 of the magnitudes covers K = 16384 (sqrt(K) * 2^-23)."""
import os
import subprocess
import sys

import pytest
import torch

from oracle import rwkvq_oracle as O

pytestmark = pytest.mark.gpu


def gen(seed, shape, std=1.0):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * std


def check(out, x, parts):
    """parts: weight matrices whose sum is the dequantized weight (their magnitudes bound the intermediate sums)."""
    xd = x.to(torch.float16).double()
    ref = sum(xd @ p.double().t() for p in parts)
    mag = sum(xd.abs() @ p.double().abs().t() for p in parts)
    err = (out.double().cpu() - ref).abs()
    bound = ref.abs() * 2.0 ** -11 + 2.0 ** -25 + mag * 2.0 ** -16
    assert bool((err <= bound).all()), float((err / bound).max())


# token tiles of 32 / 64 / 96 / 128 and their remainders, row tiles with a remainder, K slices (few tiles), group counts that
# are no multiple of 4, one step of K
@pytest.mark.parametrize("m,n,k", [(17, 512, 128), (33, 640, 768), (64, 520, 4096), (65, 4096, 1152), (129, 1000, 2560),
                                   (300, 2560, 2560), (1000, 777, 640), (12, 16400, 512), (14, 8200, 4224), (40, 512, 16384),
                                   (257, 16384, 256)])
@pytest.mark.parametrize("zeros", [True, False])
def test_int4_group_many_rows(m, n, k, zeros):
    import rwkvq_abi as abi
    from int4 import int4_ops, quantize_int4
    info = quantize_int4.quantize_to_int4_groupwise(gen(n + k, (n, k), k ** -0.5), 128)
    if not zeros:
        info["zeros"] = -8.0 * info["scales"]
    u = O.unpack_int4(info["packed"]).float().reshape(n, k // 128, 128)
    parts = [(u.double() * info["scales"].double().unsqueeze(2)).reshape(n, k),
             info["zeros"].double().unsqueeze(2).expand(n, k // 128, 128).reshape(n, k)]
    d = {a: b.cuda() if torch.is_tensor(b) else b for a, b in info.items()}
    if not zeros:
        del d["zeros"]
    d["qtype"] = "int4_groupwise"
    for dtype in (torch.float16, torch.bfloat16):
        x = gen(m, (m, k)).to(dtype)
        before = abi.launch_count()
        out = int4_ops.linear_int4(x.cuda(), d)
        assert abi.launch_count() - before in (2, 3)           # activations, GEMM, sum of the K slices
        check(out, x, parts)
        assert torch.equal(out, int4_ops.linear_int4(x.cuda(), d))


# small activations: an fp16 value below 2^-10 has no exact sixteenth.  Rows from 2^-7 to 2^-20 and one row of mixed sizes; the
# group scales bring the results back into fp16's normal range, so that the bound is that of the sums.
@pytest.mark.parametrize("m,n,k,group", [(40, 640, 1024, 128), (200, 1000, 640, 128), (1, 640, 1024, 128), (7, 640, 1152, 128), (13, 640, 4096, 128),
                                         (5, 640, 16384, 128), (16, 1000, 1280, 256)])
def test_int4_group_small_activations(m, n, k, group):
    from int4 import int4_ops, quantize_int4
    info = quantize_int4.quantize_to_int4_groupwise(gen(n + k, (n, k), k ** -0.5), group)
    info["scales"], info["zeros"] = info["scales"] * 1024, info["zeros"] * 1024
    u = O.unpack_int4(info["packed"]).float().reshape(n, k // group, group)
    parts = [(u.double() * info["scales"].double().unsqueeze(2)).reshape(n, k),
             info["zeros"].double().unsqueeze(2).expand(n, k // group, group).reshape(n, k)]
    d = {a: b.cuda() if torch.is_tensor(b) else b for a, b in info.items()}
    d["qtype"] = "int4_groupwise"
    for shift in (7, 11, 14, 20):
        x = gen(m + shift, (m, k)) * 2.0 ** -shift
        x[m - 1] *= torch.exp2(-(torch.arange(k) % 14).float())
        x = x.half()
        check(int4_ops.linear_int4(x.cuda(), d), x, parts)


@pytest.mark.parametrize("m,n,k", [(17, 512, 128), (33, 640, 784), (64, 520, 4096), (65, 4096, 1168), (129, 1000, 16),
                                   (300, 2560, 2560), (1000, 777, 640), (40, 512, 16384), (257, 16384, 256)])
def test_int8_w8a16_many_rows(m, n, k):
    import rwkvq_abi as abi
    from int8 import int8_ops, quantize_int8
    q, s = quantize_int8.quantize_to_int8_per_tensor(gen(n + k, (n, k), k ** -0.5))
    d = {"weight": q.cuda(), "tensor_scale": s.cuda(), "qtype": "int8_per_tensor"}
    x = gen(m, (m, k)).half()
    before = abi.launch_count()
    out = int8_ops.linear_int8(x.cuda(), d)
    assert abi.launch_count() - before in (1, 2)               # GEMM, sum of the K slices
    check(out, x, [q.double() * s.double()])
    assert torch.equal(out, int8_ops.linear_int8(x.cuda(), d))


def narrow_plans():
    import rwkvq_abi as abi
    from int4 import int4_ops, quantize_int4
    from int8 import int8_ops, quantize_int8
    for m, n, k in ((97, 4096, 1152), (128, 640, 2560), (300, 1000, 2560), (1000, 777, 640)):
        w = gen(n + k, (n, k), k ** -0.5)
        info = quantize_int4.quantize_to_int4_groupwise(w, 128)
        u = O.unpack_int4(info["packed"]).float().reshape(n, k // 128, 128)
        parts = [(u.double() * info["scales"].double().unsqueeze(2)).reshape(n, k), info["zeros"].double().unsqueeze(2).expand(n, k // 128, 128).reshape(n, k)]
        d = {a: b.cuda() if torch.is_tensor(b) else b for a, b in info.items()}
        q, s = quantize_int8.quantize_to_int8_per_tensor(w)
        x = gen(m, (m, k)).half()
        check(int4_ops.linear_int4(x.cuda(), dict(d, qtype="int4_groupwise")), x, parts)
        check(int8_ops.linear_int8(x.cuda(), {"weight": q.cuda(), "tensor_scale": s.cuda(), "qtype": "int8_per_tensor"}), x, [q.double() * s.double()])
    assert abi.device_status() == 0


@pytest.mark.parametrize("limit", [32, 64, 96])
def test_plans_with_narrower_token_tiles(limit):
    """Every limit of the token tile (64: what a build whose wide kernels lack their registers gets); a process reads it once."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = f"import sys; sys.path[:0] = [{os.path.join(root, 'rwkv7-quantization_b200')!r}, {root!r}, {os.path.join(root, 'tests')!r}]\n" \
           "import test_wa16_gemm_gpu as t; t.narrow_plans()"
    subprocess.run([sys.executable, "-c", code], check=True, env=dict(os.environ, RWKVQ_WA16_MAX_NB=str(limit)), timeout=300)


def pair_plans():
    import rwkvq_abi as abi
    # remainders of the 256-row and 128- / 256-token tiles, zero points of an odd and of more than 16 groups, K slices, one step
    for m, n, k in ((17, 512, 128), (127, 769, 640), (129, 1000, 1152), (200, 4096, 4224), (257, 555, 2176), (300, 2560, 2560), (1000, 777, 640), (40, 512, 16384)):
        for bits in (4, 8):
            assert abi.lib().rwkvq_tc_gemm_wa16_form(m, n, k, bits) % 1000 in (1000 - 128, 1000 - 256)
        for zeros in (True, False):
            test_int4_group_many_rows(m, n, k, zeros)
        test_int8_w8a16_many_rows(m, n, k)
    test_int4_group_small_activations(200, 1000, 640, 128)
    test_int4_infinite_and_nan_activations_stay_in_their_row(200, 640, 1152)
    test_infinite_and_nan_activations_stay_in_their_row(40, 256)
    assert abi.device_status() == 0


def test_plans_on_cta_pairs():
    """Pairs wherever they are legal; a process reads the switch once."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = f"import sys; sys.path[:0] = [{os.path.join(root, 'rwkv7-quantization_b200')!r}, {root!r}, {os.path.join(root, 'tests')!r}]\n" \
           "import test_wa16_gemm_gpu as t; t.pair_plans()"
    subprocess.run([sys.executable, "-c", code], check=True, env=dict(os.environ, RWKVQ_WA16_PAIR="force"), timeout=300)


@pytest.mark.parametrize("z", [0.0, 1.0, -2.0 ** -120, 3.0e38, float("inf")])
def test_int4_zero_points_of_unusual_size_on_pairs(z):
    """The zero points' three bf16 parts: 0, a value that is one part, a tiny and a huge one, an infinity -- against the form that
    multiplies them in fp32."""
    import rwkvq_abi as abi
    from int4 import int4_ops, quantize_int4
    m, n, k = 1000, 4096, 256
    assert abi.lib().rwkvq_tc_gemm_wa16_form(m, n, k, 4) < 1000
    info = quantize_int4.quantize_to_int4_groupwise(gen(1, (n, k), k ** -0.5), 128)
    info["zeros"][5, 1] = z
    d = {a: b.cuda() if torch.is_tensor(b) else b for a, b in info.items()}
    d["qtype"] = "int4_groupwise"
    x = gen(2, (m, k)).half()
    x[:, 128:] = x[:, 128:].abs()                              # sums of one sign
    y, few = int4_ops.linear_int4(x.cuda(), d), int4_ops.linear_int4(x[:16].cuda(), d)
    assert torch.equal(y[:16, 5].isinf(), few[:, 5].isinf()) and not bool(y[:, 5].isnan().any())
    ok = few[:, 5].isfinite()
    assert bool(((y[:16, 5] - few[:, 5])[ok].abs() <= few[:, 5][ok].abs() * 2.0 ** -10 + 2.0 ** -10).all())
    assert bool(y[:, :5].isfinite().all()) and bool(y[:, 6:].isfinite().all())


# the streaming decode kernel: token tiles of 8 and their remainders, K ranges of a warp that end inside a chunk (K = 2560,
# 2320) and inside a 64-byte unit (K = 16, 336), row tiles with a remainder, blocks that no longer fit (tensor-core GEMM)
@pytest.mark.parametrize("m,n,k", [(1, 16384, 4096), (1, 40, 16), (3, 2560, 2560), (8, 1000, 336), (9, 777, 2320), (16, 4096, 4096),
                                   (6, 512, 10240), (7, 512, 10240), (5, 520, 16384)])
def test_int8_w8a16_few_rows(m, n, k):
    from int8 import int8_ops, quantize_int8
    q, s = quantize_int8.quantize_to_int8_per_tensor(gen(n + k, (n, k), k ** -0.5))
    d = {"weight": q.cuda(), "tensor_scale": s.cuda(), "qtype": "int8_per_tensor"}
    x = gen(m, (m, k)).half()
    out = int8_ops.linear_int8(x.cuda(), d)
    check(out, x, [q.double() * s.double()])
    assert torch.equal(out, int8_ops.linear_int8(x.cuda(), d))


@pytest.mark.parametrize("m,k", [(40, 256), (6, 2320), (16, 336)])
def test_infinite_and_nan_activations_stay_in_their_row(m, k):
    from int8 import int8_ops, quantize_int8
    q, s = quantize_int8.quantize_to_int8_per_tensor(gen(1, (640, k), 0.05))
    x = gen(2, (m, k)).half()
    x[3, 0], x[m - 1, k - 1] = float("inf"), float("nan")
    out = int8_ops.linear_int8(x.cuda(), {"weight": q.cuda(), "tensor_scale": s.cuda(), "qtype": "int8_per_tensor"}).cpu()
    ok = [i for i in range(m) if i not in (3, m - 1)]
    check(out[ok], x[ok], [q.double() * s.double()])
    assert not bool(out[3].isfinite().any()) and bool(out[m - 1].isnan().all())


@pytest.mark.parametrize("m,n,k", [(40, 640, 1024), (70, 1000, 640), (200, 640, 1152), (300, 4096, 2560), (20, 640, 16384)])
def test_int4_infinite_and_nan_activations_stay_in_their_row(m, n, k):
    from int4 import int4_ops, quantize_int4
    info = quantize_int4.quantize_to_int4_groupwise(gen(n + k, (n, k), k ** -0.5), 128)
    d = {a: b.cuda() if torch.is_tensor(b) else b for a, b in info.items()}
    d["qtype"] = "int4_groupwise"
    x = gen(m, (m, k)).half()
    want = int4_ops.linear_int4(x.cuda(), d)
    x[3, 0], x[m - 1, k - 1], x[m // 2, k // 2] = float("inf"), float("nan"), float("-inf")
    out = int4_ops.linear_int4(x.cuda(), d)
    special = [3, m // 2, m - 1]
    ok = [i for i in range(m) if i not in special]
    assert torch.equal(out[ok], want[ok])
    assert not bool(out[special].isfinite().any()) and bool(out[m - 1].isnan().all())


@pytest.mark.parametrize("m,n,k", [(600, 4096, 4096), (600, 4096, 16384), (1000, 4096, 2176)])
def test_int4_scales_and_zeros_that_cancel(m, n, k):
    """Activations around 8 and zeros of minus the mean weight: the scales' and the zeros' parts of a sum are thousands of times the result.
    The error before the result is rounded to fp16 may be twice that of fp32 sums that add the two parts group by group."""
    import rwkvq_abi as abi
    from int4 import int4_ops, quantize_int4
    assert abi.lib().rwkvq_tc_gemm_wa16_form(m, n, k, 4) % 1000 in (1000 - 128, 1000 - 256)
    info = quantize_int4.quantize_to_int4_groupwise(gen(n + k, (n, k), k ** -0.5) * 64, 128)
    d = {a: b.cuda() if torch.is_tensor(b) else b for a, b in info.items()}
    u = int4_ops.unpack_int4(d["packed"]).double().reshape(n, k // 128, 128)
    d["zeros"] = -(d["scales"] * u.mean(2).float())
    x = (8 + gen(m, (m, k)) * 2.0 ** -5).half().cuda()
    ref, acc = torch.zeros((m, n), dtype=torch.float64, device="cuda"), torch.zeros((m, n), device="cuda")
    for g in range(k // 128):
        xg = x[:, g * 128:(g + 1) * 128].double()
        for f, v in ((d["scales"][:, g], xg @ u[:, g].t()), (d["zeros"][:, g], xg.sum(1, keepdim=True))):
            ref += f.double() * v
            acc += f * v.float()
    rms = lambda e: float(e.double().square().mean().sqrt())  # noqa: E731
    err, sums, half = (rms(v.double() - ref) for v in (int4_ops.linear_int4(x, dict(d, qtype="int4_groupwise")), acc, ref.half()))
    assert err <= 2 * sums + half, (err, sums, half)


def test_int4_zero_points_keep_all_products_of_their_parts():
    """Zero point of the centred codes and sum of the activations both 1 + 2^-7 - 2^-23 (times a power of two), the values whose lower bf16 parts are
    largest, against a scale that cancels them exactly.  What is left are errors: half an ulp of the scales' product, the tensor core's
    sum cut to fp32 (one ulp) and its addends' alignment (one more); without zm xl and zl xm it would be 2^-21 of the product, four ulps."""
    import rwkvq_abi as abi
    from int4 import int4_ops
    m, n, k = 1000, 4096, 256
    assert abi.lib().rwkvq_tc_gemm_wa16_form(m, n, k, 4) % 1000 in (1000 - 128, 1000 - 256)
    v = 1 + 2.0 ** -7 - 2.0 ** -23
    d = {"packed": torch.full((n, k // 2), 0x88, dtype=torch.uint8, device="cuda"), "scales": torch.full((n, 2), 2 * v, device="cuda"),
         "zeros": torch.full((n, 2), -16 * v, device="cuda"), "group_size": 128, "qtype": "int4_groupwise"}
    assert float((d["scales"].double() * 8 + d["zeros"].double()).abs().max()) == 0
    x = torch.zeros((m, k), dtype=torch.float16, device="cuda")
    x[:, :128] = 65
    x[:, 0], x[:, 1] = -2.0 ** -10, 66
    assert float(x.double().sum(1).max()) == v * 2 ** 13
    y = int4_ops.linear_int4(x, d)
    assert float(y.abs().max()) <= 2.5 * 2.0 ** -10, float(y.abs().max())
