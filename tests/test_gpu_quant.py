"""Bit-exact parity of the sm_100a blockwise quantisers with the oracle
(integer/byte outputs and IEEE-divided scales: no tolerance)."""
import numpy as np
import pytest
import torch

from helpers import fp8_sources

pytestmark = pytest.mark.gpu


def gpu_quant_1x128(capi, cuda, x):
    M, K = x.shape
    q = torch.full((M, K), 0xAA, dtype=torch.uint8, device=cuda)
    s = torch.full((K // 128, M), float("nan"), dtype=torch.float32, device=cuda)
    capi.fp8_quant_1x128(torch.from_numpy(x).to(cuda), q, s, M, K)
    torch.cuda.synchronize()
    return q.cpu().numpy(), s.cpu().numpy()


def gpu_quant_128x128(capi, cuda, w):
    R, C = w.shape
    q = torch.full((R, C), 0xAA, dtype=torch.uint8, device=cuda)
    s = torch.full((R // 128, C // 128), float("nan"), dtype=torch.float32, device=cuda)
    capi.fp8_quant_128x128(torch.from_numpy(w).to(cuda), q, s, R, C)
    torch.cuda.synchronize()
    return q.cpu().numpy(), s.cpu().numpy()


@pytest.mark.parametrize("shape", [(1, 128), (16, 2560), (33, 384), (64, 9728), (257, 1024), (1000, 512)])
def test_quant_1x128_bit_exact(capi, oracle, cuda, shape):
    x, _ = fp8_sources(30, shape[0], 128, shape[1])
    if shape[0] > 3:
        x[3, :128] = 0.0          # all-zero group
        x[2, 5] = 3.0e38          # huge value: scale near the top of fp32
        x[1, :128] *= 1e-30       # tiny group: scale is subnormal-sized
    q, s = gpu_quant_1x128(capi, cuda, x)
    oq, os_ = oracle.quant_1x128(x)
    assert (s.view(np.uint32) == os_.view(np.uint32)).all()
    assert (q == oq).all()


@pytest.mark.parametrize("shape", [(128, 128), (256, 384), (2560, 4096), (1024, 640)])
def test_quant_128x128_bit_exact(capi, oracle, cuda, shape):
    _, w = fp8_sources(31, 8, shape[0], shape[1], w_std=0.02)
    w[:128, :128] = 0.0
    q, s = gpu_quant_128x128(capi, cuda, w)
    oq, os_ = oracle.quant_128x128(w)
    assert (s.view(np.uint32) == os_.view(np.uint32)).all()
    assert (q == oq).all()


@pytest.mark.parametrize("shape", [(4096, 128), (4097, 128), (5461, 384), (5462, 384), (7711, 2176), (7710, 2176)])
def test_quant_1x128_rows_per_warp(capi, cuda, shape):
    # both sides of the group counts (4096, 16384, 131072) at which a warp takes more rows, against torch's IEEE divisions
    M, K = shape
    x = torch.randn(M, K, device=cuda, generator=torch.Generator(device=cuda).manual_seed(33))
    x[M // 2] *= 1e20
    q = torch.full((M, K), 0xAA, dtype=torch.uint8, device=cuda)
    s = torch.full((K // 128, M), float("nan"), device=cuda)
    capi.fp8_quant_1x128(x, q, s, M, K)
    b = x.view(M, K // 128, 128)
    want = b.abs().amax(dim=2) / torch.full((), 448.0, device=cuda)
    assert torch.equal(s.t(), want)
    assert torch.equal(q, (b / want[..., None]).to(torch.float8_e4m3fn).view(torch.uint8).view(M, K))


def test_quant_1x128_nan_and_infinity(capi, cuda):
    # NaN values do not enter a group's maximum unless all of them are NaN; an infinite value makes the scale infinite
    x = torch.randn(3, 256, device=cuda, generator=torch.Generator(device=cuda).manual_seed(34))
    clean = x.clone()
    x[0, 5], x[0, 6] = float("nan"), -float("nan")
    x[1, :128] = float("nan")
    x[2, 130] = float("-inf")
    q = torch.zeros(3, 256, dtype=torch.uint8, device=cuda)
    s = torch.zeros(2, 3, device=cuda)
    capi.fp8_quant_1x128(x, q, s, 3, 256)
    rest = clean.clone()
    rest[0, 5:7] = 0
    assert s[0, 0] == rest[0, :128].abs().max() / torch.full((), 448.0, device=cuda)
    assert bool(((q[0, 5:7] & 0x7F) == 0x7F).all()) and bool(((q[0, 7:128] & 0x7F) != 0x7F).all())
    assert bool(torch.isnan(s[0, 1])) and bool(((q[1, :128] & 0x7F) == 0x7F).all())
    assert bool(torch.isinf(s[1, 2])) and bool(torch.isfinite(s[1, :2]).all())


def test_full_size_quant_properties(capi, cuda):
    # 4096 x 4096 (the FP8 headline config): every group's largest code is +-448 and the
    # scale array is exactly amax/448 computed by torch in fp32
    M = K = 4096
    g = torch.Generator(device=cuda).manual_seed(32)
    x = torch.randn(M, K, device=cuda, generator=g)
    q = torch.empty(M, K, dtype=torch.uint8, device=cuda)
    s = torch.empty(K // 128, M, dtype=torch.float32, device=cuda)
    capi.fp8_quant_1x128(x, q, s, M, K)
    amax = x.view(M, K // 128, 128).abs().amax(dim=2)
    assert torch.equal(s.t().contiguous(), amax / torch.full_like(amax, 448.0))  # tensor / tensor: IEEE division
    codes = (q.view(M, K // 128, 128) & 0x7F).amax(dim=2)
    assert bool((codes == 0x7E).all())
    wq = torch.empty(M, K, dtype=torch.uint8, device=cuda)
    ws = torch.empty(M // 128, K // 128, dtype=torch.float32, device=cuda)
    capi.fp8_quant_128x128(x, wq, ws, M, K)
    bmax = x.view(M // 128, 128, K // 128, 128).abs().amax(dim=(1, 3))
    assert torch.equal(ws, bmax / torch.full_like(bmax, 448.0))
    # torch's own e4m3 conversion agrees with the bytes (same RN-even, saturating rule)
    deq_in = (x.view(M // 128, 128, K // 128, 128) / ws.view(M // 128, 1, K // 128, 1)).view(M, K)
    assert torch.equal(deq_in.to(torch.float8_e4m3fn).view(torch.uint8), wq)
    capi.check_status()


def test_quant_errors(capi, cuda):
    x = torch.zeros(4, 100, device=cuda)
    with pytest.raises(RuntimeError, match="not aligned"):
        capi.fp8_quant_1x128(x, torch.zeros(4, 100, dtype=torch.uint8, device=cuda), torch.zeros(1, 4, device=cuda), 4, 100)
