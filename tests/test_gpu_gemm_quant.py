"""Quantised-weight tcgen05 GEMMs (fp8 row-scale W8A8, nvfp4 block-scaled W4A4) against fp32 oracles."""
import pytest
import torch

from ninfer_fusion_b200._lib import StatusWord, load_native
from ninfer_fusion_b200.ops import quant as Q

pytestmark = pytest.mark.gpu
EPI_STORE, EPI_RESIDUAL, EPI_SWIGLU = 0, 1, 2


def _act_fp8(ops, x):
    T, K = x.shape
    codes = torch.empty((T, K), dtype=torch.uint8, device="cuda")
    scale = torch.empty(T, dtype=torch.float32, device="cuda")
    ops.quant_act_fp8(x, codes, scale)
    return codes, scale


def _act_nvfp4(ops, x):
    T, K = x.shape
    codes = torch.empty((T, K // 2), dtype=torch.uint8, device="cuda")
    plane = torch.zeros(int(ops.nvfp4_act_scale_bytes(T, K)), dtype=torch.uint8, device="cuda")
    ops.quant_act_nvfp4(x, codes, plane)
    return codes, plane


@pytest.mark.parametrize("T", [1, 32, 100, 300])
def test_activation_quantisers(T):
    ops = load_native()
    torch.manual_seed(T)
    K = 1024
    x = (torch.randn(T, K, device="cuda") * torch.rand(T, 1, device="cuda") * 4).bfloat16()
    codes, scale = _act_fp8(ops, x)
    deq = Q.dequant_fp8_row(codes, scale)
    assert (deq - x.float()).abs().max().item() <= 0.07 * x.float().abs().max().item()
    want_scale = x.float().abs().amax(-1) / 448.0
    assert torch.allclose(scale, want_scale, rtol=1e-6)
    c4, plane = _act_nvfp4(ops, x)
    deq4 = Q.dequant_nvfp4(c4, plane, 1.0, T, K)
    blk = x.float().reshape(T, K // 16, 16)
    err = (deq4.reshape(T, K // 16, 16) - blk).abs().amax(-1)
    assert (err <= 0.26 * blk.abs().amax(-1) + 1e-6).all()  # e2m1 step is at most amax/3 wide, plus the scale rounding


@pytest.mark.parametrize("qt", ["fp8", "nvfp4"])
@pytest.mark.parametrize("T,N,K,epi,splits", [
    (1, 256, 512, EPI_STORE, 1), (20, 384, 1024, EPI_RESIDUAL, 1), (32, 512, 2048, EPI_SWIGLU, 1),
    (64, 256, 2048, EPI_STORE, 4), (100, 640, 768, EPI_RESIDUAL, 1), (130, 256, 512, EPI_SWIGLU, 1),
    (300, 384, 1024, EPI_STORE, 1), (16, 5120, 5120, EPI_RESIDUAL, 3),
    # more tiles than SMs at prefill size: the persistent kernel (overlapped epilogue), ragged T
    (600, 8192, 768, EPI_STORE, 1), (777, 8192, 512, EPI_RESIDUAL, 1), (1000, 9984, 512, EPI_SWIGLU, 1)])
def test_gemm_quant_matches_oracle(qt, T, N, K, epi, splits):
    ops = load_native()
    status = StatusWord("cuda")
    torch.manual_seed(T + N)
    w = torch.randn(N, K, device="cuda") * 0.05
    x = torch.randn(T, K, device="cuda").bfloat16()
    resid = torch.randn(T, N, device="cuda").bfloat16() if epi == EPI_RESIDUAL else None
    w_rows = Q.interleave_gate_up(w) if epi == EPI_SWIGLU else w
    if qt == "fp8":
        wc, ws = Q.quantize_fp8_row(w_rows)
        xc, xs = _act_fp8(ops, x)
        w_deq, x_deq, div, code = Q.dequant_fp8_row(wc, ws), Q.dequant_fp8_row(xc, xs), 1.0, Q.QT_FP8_ROW
    else:
        wc, ws, div = Q.quantize_nvfp4(w_rows)
        xc, xs = _act_nvfp4(ops, x)
        w_deq, x_deq, code = Q.dequant_nvfp4(wc, ws, div, N, K), Q.dequant_nvfp4(xc, xs, 1.0, T, K), Q.QT_NVFP4
    out = torch.empty((T, N // 2 if epi == EPI_SWIGLU else N), dtype=torch.bfloat16, device="cuda")
    ops.gemm_quant(code, xc, xs, wc, ws, div, out, epi, resid, splits, status.tensor, False)
    torch.cuda.synchronize()
    status.check()
    acc = x_deq.double() @ w_deq.double().t()
    if epi == EPI_SWIGLU:
        t = acc.reshape(T, N // 128, 2, 64)   # tile-interleaved rows: [64 gate ; 64 up]
        want = (torch.nn.functional.silu(t[:, :, 0]) * t[:, :, 1]).reshape(T, N // 2)
    elif epi == EPI_RESIDUAL:
        want = acc + resid.double()
    else:
        want = acc
    err = (out.double() - want).abs().max().item()
    assert err <= 0.01 * want.abs().max().item() + 0.01, f"max err {err} vs scale {want.abs().max().item()}"


@pytest.mark.parametrize("qt", ["fp8", "nvfp4"])
@pytest.mark.parametrize("N,K", [(256, 256), (384, 2048), (19200, 512)])
@pytest.mark.parametrize("T", [65, 128, 129, 144, 256, 257, 400])
@pytest.mark.parametrize("epi", [EPI_STORE, EPI_RESIDUAL, EPI_SWIGLU])
def test_gemm_quant_token_tiles(qt, T, N, K, epi):
    """Persistent tiles of 128 and 256 tokens, ragged last ones, more and fewer tiles than SMs; nothing beside the output."""
    ops = load_native()
    status = StatusWord("cuda")
    torch.manual_seed(T + N)
    w = torch.randn(N, K, device="cuda") * 0.05
    x = torch.randn(T, K, device="cuda").bfloat16()
    if qt == "fp8":
        (wc, ws), (xc, xs), div, code = Q.quantize_fp8_row(w), _act_fp8(ops, x), 1.0, Q.QT_FP8_ROW
        w_deq, x_deq = Q.dequant_fp8_row(wc, ws), Q.dequant_fp8_row(xc, xs)
    else:
        (wc, ws, div), (xc, xs), code = Q.quantize_nvfp4(w), _act_nvfp4(ops, x), Q.QT_NVFP4
        w_deq, x_deq = Q.dequant_nvfp4(wc, ws, div, N, K), Q.dequant_nvfp4(xc, xs, 1.0, T, K)
    acc = x_deq.double() @ w_deq.double().t()
    cols = N // 2 if epi == EPI_SWIGLU else N
    wide = torch.full((T + 1, cols + 2), float("nan"), device="cuda", dtype=torch.bfloat16)
    out = wide[:T, :cols]
    if epi == EPI_RESIDUAL:
        out.copy_(torch.randn(T, N, device="cuda"))
    want = acc
    if epi == EPI_SWIGLU:
        t = acc.reshape(T, N // 128, 2, 64)
        want = (torch.nn.functional.silu(t[:, :, 0]) * t[:, :, 1]).reshape(T, cols)
    elif epi == EPI_RESIDUAL:
        want = acc + out.double()
    ops.gemm_quant(code, xc, xs, wc, ws, div, out, epi, out if epi == EPI_RESIDUAL else None, 1, status.tensor, True)
    # one rounding to bf16 (2^-9), twice that for the hardware exponential and the sums' order
    assert (out.double() - want).abs().max() <= want.abs().max() * 2.0 ** -8
    assert wide[T].isnan().all() and wide[:, cols:].isnan().all()
    status.check("persistent quantised gemm")


def test_nvfp4_codes_by_products():
    """Codes and scales bit for bit against the quotient on the host: every bf16 exponent, all ties, NaN, infinities, zeros."""
    ops = load_native()
    torch.manual_seed(5)
    K = 2048
    grid = torch.tensor([0.0, 0.25, 0.5, 0.75, 1.0, 1.25, 1.5, 1.75, 2.0, 2.5, 3.0, 3.5, 4.0, 5.0, 6.0, -0.25])
    ties = grid.repeat(K // 16)[None] * 2.0 ** torch.arange(-9, 9)[:, None]           # scales of a power of two: exact ties
    scaled = ties * (1 + torch.arange(8)[torch.arange(18) % 8, None] / 8)              # and of every mantissa
    near = torch.randn(64, K) * 2.0 ** torch.randint(-20, 12, (64, K // 16)).repeat_interleave(16, 1)
    odd = torch.randn(4, K)
    odd[0, ::7], odd[1, ::5], odd[1, 1::11], odd[2] = float("nan"), float("inf"), float("-inf"), 0.0
    x = torch.cat([ties, scaled, near, odd]).bfloat16().cuda()
    T = x.shape[0]
    codes, plane = _act_nvfp4(ops, x)
    g = x.float().reshape(T, K // 16, 16)
    amax = torch.where(g.isnan(), torch.zeros_like(g), g.abs()).amax(-1)
    sf = (amax / 6).clamp(max=448.0).to(torch.float8_e4m3fn).float()
    q = torch.where(sf[..., None] > 0, g / sf[..., None], torch.zeros_like(g))
    a = q.abs()
    bounds = ((0.25, True), (0.75, False), (1.25, True), (1.75, False), (2.5, True), (3.5, False), (5.0, True))
    mag = sum((~(a <= b) if closed else ~(a < b)).to(torch.uint8) for b, closed in bounds)
    want = (mag | ((q < 0).to(torch.uint8) << 3)).reshape(T, K)
    assert torch.equal(codes, want[:, 0::2] | (want[:, 1::2] << 4))
    got_sf = plane[Q.sf_tile_offsets(T, K, "cuda")].reshape(T, K // 16)
    assert torch.equal(got_sf, sf.to(torch.float8_e4m3fn).view(torch.uint8))
