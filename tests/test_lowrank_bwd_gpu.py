"""The bf16 tensor-core products of the low-rank branch's backward against float64 on the same bf16
inputs: the generic panel product in all four operand storage orders (an operand stored with the
contraction in its rows is read as it lies, never transposed in memory), then the two entry points that
autograd's backward of `ulinear(torch.mul(s, y))` (bitlinear.py:752-757) maps onto.
Tolerance: fp32 accumulation of exact bf16 products, rel-L2 <= 1e-5 before the stated bf16 roundings."""
import pytest
import torch

from fp4_post_b200 import ops
from gpu_helpers import rel_l2

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module", autouse=True)
def _lib(built_library):
    return built_library


def _randn(rows, cols, seed, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(rows, cols, device=DEV, generator=g) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("Mg,Ng,Kg", [(128, 64, 64), (128, 128, 256), (256, 128, 1024), (200, 32, 136), (384, 256, 4096),
                                      (1000, 96, 520), (4096, 128, 2048)])
def test_panel_product_in_every_storage_order(Mg, Ng, Kg, a_mn, b_mn):
    a = _randn(Mg, Kg, seed=Mg + Kg)
    b = _randn(Ng, Kg, seed=Ng + Kg + 1, scale=Kg ** -0.5)
    want = a.double() @ b.double().t()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    got = ops.bf16_panel_gemm(a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b,
                              a_mn_major=a_mn, b_mn_major=b_mn, status=status)
    torch.cuda.synchronize()
    assert status.item() == 0
    assert got.shape == (Mg, Ng)
    assert rel_l2(got.double().cpu().numpy(), want.cpu().numpy()) <= 1e-5


def test_panel_product_reads_strided_operands_as_they_lie():
    wide = _randn(512, 1024, seed=3)
    a = wide[:, 128:640]                       # [512, 512] view with row pitch 1024
    b = _randn(64, 512, seed=4)
    got = ops.bf16_panel_gemm(a, b)
    assert rel_l2(got.double().cpu().numpy(), (a.double() @ b.double().t()).cpu().numpy()) <= 1e-5
    got = ops.bf16_panel_gemm(a, b, a_mn_major=True)      # the same memory read as [Kg = 512, Mg = 512]
    assert rel_l2(got.double().cpu().numpy(), (a.double().t() @ b.double().t()).cpu().numpy()) <= 1e-5


@pytest.mark.parametrize("M,N,r", [(256, 384, 32), (512, 1536, 64), (2048, 4096, 128), (1000, 520, 256), (16384, 4096, 128),
                                   (1120, 3584, 96), (33, 1024, 8), (9472, 640, 200)])
@pytest.mark.parametrize("s_dtype", [torch.bfloat16, torch.float32])
def test_gradient_through_ulinear_and_the_scaling(M, N, r, s_dtype):
    g = _randn(M, N, seed=M + N)
    u = _randn(N, r, seed=N + r, scale=N ** -0.5)
    yv = _randn(M, r, seed=M + r + 7)
    s = (torch.rand(r, device=DEV, generator=torch.Generator(device=DEV).manual_seed(r)) + 0.5).to(s_dtype)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    d_yv, ds = ops.lowrank_dts(g, u, yv, s, status=status)
    torch.cuda.synchronize()
    assert status.item() == 0
    # the products in float64, then the roundings autograd's bf16 ops apply
    d_ts64 = g.double() @ u.double()
    d_ts = d_ts64.to(torch.bfloat16)
    want_dyv = (d_ts.float() * s.to(torch.bfloat16).float()).to(torch.bfloat16)
    # a sum that lands within fp32 summation error of a bf16 rounding boundary rounds the other way (a few
    # elements in 1e5): d_ts then differs by one ulp, d_yv by up to two
    diff = (d_yv.float() - want_dyv.float()).abs()
    assert bool((diff <= want_dyv.float().abs() * 2.0 ** -6 + 2e-5).all())       # sums that cancel to ~1e-4 keep the absolute error of their 4096 terms
    assert float((diff == 0).float().mean()) > 0.99
    want_ds = (d_ts.float() * yv.float()).to(torch.bfloat16).double().sum(dim=0)
    assert rel_l2(ds.double().cpu().numpy(), want_ds.cpu().numpy()) <= 2e-3
    # the weight gradient of ulinear: contraction over the tokens
    ts = (yv.float() * s.to(torch.bfloat16).float()).to(torch.bfloat16)
    for out_dtype in (torch.bfloat16, torch.float32):
        du = ops.lowrank_du(g, ts, out_dtype=out_dtype, status=status)
        want = g.double().t() @ ts.double()
        tol = 1e-5 if out_dtype == torch.float32 else 4e-3
        assert du.dtype == out_dtype and du.shape == (N, r)
        assert rel_l2(du.double().cpu().numpy(), want.cpu().numpy()) <= tol
    torch.cuda.synchronize()
    assert status.item() == 0


def test_bad_shapes_are_rejected_on_the_host():
    g, u, yv = _randn(64, 64, 1), _randn(64, 12, 2), _randn(64, 12, 3)
    with pytest.raises(ValueError):
        ops.lowrank_dts(g, u, yv, torch.ones(12, device=DEV))          # rank 12: not a multiple of 8
    with pytest.raises(ValueError):
        ops.bf16_panel_gemm(_randn(64, 64, 4), _randn(300, 64, 5))     # more than 256 columns


@pytest.mark.parametrize("M,N,r", [(33, 1024, 8), (1120, 3584, 96), (9472, 640, 200), (12800, 520, 128)])
def test_ds_in_bf16_and_the_column_mean_of_d_yv(M, N, r):
    """Both finishes (sums over splits; straight from the accumulator from 9600 tokens on): ds rounded once, the mean
    that of the rounded d_yv.  Bound: fp32 sums of M terms in blocks, 2^-24 times the sum of magnitudes times the depth."""
    g, u, yv = _randn(M, N, seed=M), _randn(N, r, seed=N, scale=N ** -0.5), _randn(M, r, seed=r)
    s = torch.linspace(0.5, 1.5, r, device=DEV).to(torch.bfloat16)
    d_yv, ds32 = ops.lowrank_dts(g, u, yv, s)
    d_yv2, ds16, mean = ops.lowrank_dts(g, u, yv, s, ds_dtype=torch.bfloat16, want_mean=True)
    assert torch.equal(d_yv, d_yv2) and torch.equal(ds16, ds32.to(torch.bfloat16))
    want = d_yv.double().mean(0)
    bound = 2.0 ** -24 * 64 * d_yv.double().abs().mean(0) + 1e-30
    assert bool(((mean.double() - want).abs() <= bound).all())


def test_dequantized_in_a_ratio_of_units():
    q = ops.nvfp4_quantize(_randn(96, 272, seed=9))
    units = [torch.full((1,), v, device=DEV) for v in (0.37, 1.9, 0.011, 5.3)]
    got = ops.nvfp4_dequantize_ratio(q, torch.bfloat16, *units)
    want = ops.nvfp4_dequantize(q, torch.bfloat16, unit=(units[0] * units[1]) / (units[2] * units[3]))
    assert torch.equal(got, want)


# Bit for bit the torch expressions: more elements than one round of the grid, a row and a half, subnormal tails, a pitch.
@pytest.mark.parametrize("M,N,r,parts", [(2048, 2048, 64, 3), (16384, 8960, 64, 3), (1, 16, 8, 3), (300, 50, 128, 1)])
@pytest.mark.parametrize("s_dtype", [torch.bfloat16, torch.float32])
def test_factors_of_an_fp32_layer(M, N, r, parts, s_dtype):
    g = torch.Generator(device=DEV).manual_seed(M + r)
    store = torch.randn(M, r + 8, generator=g, device=DEV) * torch.exp(8 * torch.randn(M, 1, generator=g, device=DEV))
    yv = store[:, :r]
    u, s = torch.randn(N, r, generator=g, device=DEV), torch.rand(r, generator=g, device=DEV).to(s_dtype)
    ua, ub = torch.tensor([0.37], device=DEV), torch.tensor([1.9e-3], device=DEV)
    t, u_out = ops.lowrank_factors(yv, s, ua, ub, u, parts)
    t32 = (yv * s.float()) / (ua * ub)

    def split(v, order):
        head = v.to(torch.bfloat16)
        pieces = (head, (v - head.float()).to(torch.bfloat16))
        return torch.cat([pieces[i] for i in order], dim=1) if parts == 3 else head
    assert torch.equal(t, split(t32, (0, 1, 0))) and torch.equal(u_out, split(u, (0, 0, 1)))
