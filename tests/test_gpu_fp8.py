"""Parity of the sm_100a FP8 blockwise GEMM (through the C ABI) with the oracle.

Gates (from the task statement):
  * accumulator (fp32-output entry point): within 4e-6 * row amax of the fp64
    ground truth T0 of the quantised operands (accumulation-order noise only);
  * fused output: C_s and C_q are EXACTLY what the quantisation rule gives for
    the kernel's own accumulator (scales bit-exact from identical absmax);
  * de-quantised C: per element within (the oracle's own error against T0, which
    tests/golden pins as equal to the reference kernel's error) + 1 e4m3 ulp * scale.
"""
import re

import numpy as np
import pytest
import torch

from gpu_reference import fp8_blockwise_acc_f64
from helpers import e4m3_ulp, fp8_sources

pytestmark = pytest.mark.gpu

QWEN3_4B = [(6144, 2560), (2560, 4096), (19456, 2560), (2560, 9728)]


def to_dev(cuda, *arrs):
    return [torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in arrs]


def gpu_mm(capi, cuda, A_q, A_s, B_q, B_s, workspace=True):
    M, K = A_q.shape
    N = B_q.shape[0]
    dA, dAs, dB, dBs = to_dev(cuda, A_q, A_s, B_q, B_s)
    if workspace:
        capi.ensure_workspace(M, N, K)
    Cq = torch.full((M, N), 0xAA, dtype=torch.uint8, device=cuda)
    Cs = torch.full((N // 128, M), float("nan"), dtype=torch.float32, device=cuda)
    Cf = torch.full((M, N), float("nan"), dtype=torch.float32, device=cuda)
    capi.fp8_blockwise_mm(dA, dAs, dB, dBs, Cq, Cs, M, N, K)
    capi.fp8_blockwise_mm_f32(dA, dAs, dB, dBs, Cf, M, N, K)
    torch.cuda.synchronize()
    capi.check_status()
    return Cq.cpu().numpy(), Cs.cpu().numpy(), Cf.cpu().numpy()


def check_against_oracle(oracle, A_q, A_s, B_q, B_s, gq, gs, gf, rows=None):
    M, N = gq.shape
    r0, n = (0, M) if rows is None else rows
    t0 = oracle.fp8_blockwise_acc(A_q, A_s, B_q, B_s, exact=True, row0=r0, rows=n)
    t1 = oracle.fp8_blockwise_acc(A_q, A_s, B_q, B_s, row0=r0, rows=n)
    gq, gf, gs_rows = gq[r0:r0 + n], gf[r0:r0 + n], gs[:, r0:r0 + n]
    row_amax = np.abs(t0).max(axis=1, keepdims=True) + 1e-30
    # 1. accumulator
    assert (np.abs(gf - t0) <= 4e-6 * row_amax).all(), float((np.abs(gf - t0) / row_amax).max())
    assert (np.abs(t1 - t0) <= 4e-6 * row_amax).all()
    # 2. the fused output is the quantisation rule applied to the kernel's own accumulator, bit for bit
    q_rule, s_rule = oracle.c_quant_1x128(gf)
    assert (gs_rows.view(np.uint32) == s_rule.view(np.uint32)).all()
    assert (gq == q_rule).all()
    # 3. de-quantised values against the ground truth
    o_q, o_s = oracle.c_quant_1x128(t1)
    deq = oracle.e4m3_decode(gq) * np.repeat(gs_rows.T, 128, axis=1)
    o_deq = oracle.e4m3_decode(o_q) * np.repeat(o_s.T, 128, axis=1)
    scale_e = np.repeat(gs_rows.T, 128, axis=1).astype(np.float64)
    ulp = e4m3_ulp(oracle.e4m3_decode(gq)) * scale_e
    assert (np.abs(deq - t0) <= np.abs(o_deq - t0) + ulp + 1e-30).all()
    # scales within accumulation noise of the oracle's, bytes overwhelmingly identical
    ok = o_s > 0
    assert (np.abs(gs_rows[ok] / o_s[ok] - 1) <= 4e-6).all()
    assert (gq == o_q).mean() > 0.99


def make_case(oracle, seed, M, N, K, w_std=0.02):
    x, w = fp8_sources(seed, M, N, K, w_std=w_std)
    A_q, A_s = oracle.quant_1x128(x)
    B_q, B_s = oracle.quant_128x128(w)
    return A_q, A_s, B_q, B_s


@pytest.mark.parametrize("shape", [(128, 256, 128), (128, 128, 128), (256, 512, 512), (200, 384, 256), (129, 640, 1280),
                                   (512, 1152, 384)])
def test_general_kernel_small_shapes(capi, oracle, cuda, shape):
    M, N, K = shape
    case = make_case(oracle, 40, M, N, K)
    gq, gs, gf = gpu_mm(capi, cuda, *case)
    check_against_oracle(oracle, *case, gq, gs, gf)


@pytest.mark.parametrize("k_blocks", [1, 3, 4, 5, 17, 21])
@pytest.mark.parametrize("M", [129, 254, 387])
def test_pair_kernel_scale_ring(capi, oracle, cuda, M, k_blocks):
    # K-blocks around the chunks of four and the sixteen of the whole ring in which the pair kernel keeps its scales;
    # an odd number of rows, so that rows of A_s start at any multiple of four bytes; several tiles per pair
    case = make_case(oracle, 46 + k_blocks, M, 384, 128 * k_blocks)
    check_against_oracle(oracle, *case, *gpu_mm(capi, cuda, *case))


@pytest.mark.parametrize("M", [1, 2, 15, 16, 17, 33, 64])
@pytest.mark.parametrize("NK", [(256, 1024), (384, 128), (2560, 4096), (19072, 256), (37888, 128), (25600, 512)])
def test_decode_kernel_ragged_m(capi, oracle, cuda, M, NK):
    """Among the shapes: 149 groups x 2 K-blocks (one whole group per CTA plus one left-over group cut in two),
    296 groups x 1 (two whole groups per CTA, nothing cut), 200 groups x 4 (one whole group per CTA and 52
    left-over groups cut into pieces of one or two K-blocks that cross group boundaries)."""
    N, K = NK
    case = make_case(oracle, 41 + M, M, N, K)
    gq, gs, gf = gpu_mm(capi, cuda, *case)
    check_against_oracle(oracle, *case, gq, gs, gf)


@pytest.mark.parametrize("M", [1, 3, 9, 10, 16])
@pytest.mark.parametrize("NK", [(19072, 1024), (19072, 1152), (19072, 2048), (19072, 2176), (19200, 3328), (19072, 6400)])
def test_left_over_groups_with_many_contributors(capi, oracle, cuda, M, NK):
    # 149 or 150 groups: one or two left-over groups in pieces of one K-block, 8, 9, 16, 17, 26 and 50 contributors: both
    # sides of the choice between a warp and four warps per row, and more contributors than are in flight at a time
    N, K = NK
    case = make_case(oracle, 47 + M, M, N, K)
    gq, gs, gf = gpu_mm(capi, cuda, *case)
    check_against_oracle(oracle, *case, gq, gs, gf)
    gq2, gs2, gf2 = gpu_mm(capi, cuda, *case)  # and the words went back to zero
    assert np.array_equal(gq, gq2) and np.array_equal(gs, gs2) and np.array_equal(gf, gf2)


def ctas_with_a_row_in_two_groups(M, N, K, ctas=148):
    """CTAs of the stream-K decode kernel that finish a row in both of their cut groups with four warps to the row (more than
    eight contributors, no more rows than those), from the split rule: the left-over groups cut evenly among the CTAs."""
    groups, kb = N // 128, K // 128
    tail = (groups - groups // ctas * ctas) * kb
    n = min(tail, ctas)
    runs = [(c * tail // n, (c + 1) * tail // n) for c in range(n)]
    found = []
    for c, (lo, hi) in enumerate(runs):
        rows = 0
        for g in {lo // kb, (hi - 1) // kb}:
            part = [i for i, (a, b) in enumerate(runs) if a < (g + 1) * kb and b > g * kb]
            rows += len(part) > 8 and M <= len(part) and c - part[0] < M
        if rows == 2:
            found.append(c)
    return found


@pytest.mark.parametrize("shape", [(15, 1280, 4096), (15, 1280, 2560), (16, 1280, 9728), (13, 20480, 2560), (11, 20736, 2560), (14, 20352, 4096)])
def test_one_cta_finishes_a_row_in_two_groups(capi, oracle, cuda, shape):
    # the two rows follow one another in the same four warps: each has its own exchange of row maxima
    M, N, K = shape
    assert ctas_with_a_row_in_two_groups(M, N, K)
    case = make_case(oracle, 49, M, N, K)
    gq, gs, gf = gpu_mm(capi, cuda, *case)
    assert "stream-K" in capi.describe_plan("fp8", M, N, K)
    check_against_oracle(oracle, *case, gq, gs, gf)
    dev = to_dev(cuda, *case)
    Cq, Cs = torch.empty((M, N), dtype=torch.uint8, device=cuda), torch.empty((N // 128, M), device=cuda)
    for _ in range(50):
        capi.fp8_blockwise_mm(*dev, Cq, Cs, M, N, K)
        assert np.array_equal(Cq.cpu().numpy(), gq) and np.array_equal(Cs.cpu().numpy(), gs)


@pytest.mark.parametrize("M", [1, 16, 64])
@pytest.mark.parametrize("NK", QWEN3_4B)
def test_qwen3_4b_decode_shapes(capi, oracle, cuda, M, NK):
    N, K = NK
    case = make_case(oracle, 50, M, N, K)
    gq, gs, gf = gpu_mm(capi, cuda, *case)
    check_against_oracle(oracle, *case, gq, gs, gf)


@pytest.mark.parametrize("M", [1, 16])
@pytest.mark.parametrize("run", [(1, 0), (3, 2), (6, 0), (6, 1), (7, 0)], ids=lambda r: f"{r[0]}+{r[1]}")
def test_cluster_decode_around_the_ring_depth(capi, oracle, cuda, M, run):
    # one to seven K-blocks per CTA of a cluster, whose MMAs two threads issue in turn: odd and even runs, the six of the ring
    # and one more, in all CTAs of a cluster or in one.  (How many CTAs it has follows how many clusters the device holds.)
    N = 2560
    size = int(re.search(r"clusters of (\d) CTAs", capi.describe_plan("fp8", M, N, 4096))[1])
    K = 128 * (size * run[0] + run[1])
    case = make_case(oracle, 51 + run[0], M, N, K)
    gq, gs, gf = gpu_mm(capi, cuda, *case)
    assert f"clusters of {size} CTAs" in capi.describe_plan("fp8", M, N, K)
    check_against_oracle(oracle, *case, gq, gs, gf)
    gq2, gs2, gf2 = gpu_mm(capi, cuda, *case)
    assert np.array_equal(gq, gq2) and np.array_equal(gs, gs2) and np.array_equal(gf, gf2)


def test_decode_without_workspace_uses_general_kernel(capi, oracle, cuda):
    # no scratch registered -> the library must still compute (general kernel), never fail or fall back to a CPU
    case = make_case(oracle, 42, 16, 512, 1024)
    capi.clear_workspace()
    gq, gs, gf = gpu_mm(capi, cuda, *case, workspace=False)
    check_against_oracle(oracle, *case, gq, gs, gf)
    gq2, gs2, gf2 = gpu_mm(capi, cuda, *case, workspace=True)
    check_against_oracle(oracle, *case, gq2, gs2, gf2)
    # split-K changes only the order of the fp32 promotion sums
    assert np.abs(gf - gf2).max() <= 4e-6 * np.abs(gf).max()


def test_decode_repeated_calls_are_bitwise_stable(capi, oracle, cuda):
    # the arrival counters reset themselves and partials are summed in a fixed order
    M, N, K = 16, 2560, 9728
    A_q, A_s, B_q, B_s = make_case(oracle, 43, M, N, K)
    dA, dAs, dB, dBs = to_dev(cuda, A_q, A_s, B_q, B_s)
    capi.ensure_workspace(M, N, K)
    outs = []
    for _ in range(5):
        Cq = torch.zeros(M, N, dtype=torch.uint8, device=cuda)
        Cs = torch.zeros(N // 128, M, dtype=torch.float32, device=cuda)
        capi.fp8_blockwise_mm(dA, dAs, dB, dBs, Cq, Cs, M, N, K)
        outs.append((Cq, Cs))
    torch.cuda.synchronize()
    for Cq, Cs in outs[1:]:
        assert torch.equal(Cq, outs[0][0]) and torch.equal(Cs, outs[0][1])
    capi.check_status()


# Shapes whose last wave of 256x256 tiles is shared out K-block by K-block when scratch is registered:
# few tiles with a long K (every tile has many contributors), ragged M and N, and several full waves
# followed by a partial one.
SPLIT_SHAPES = [(256, 512, 4096), (384, 640, 4096), (300, 1280, 3584), (1024, 2048, 4096), (2304, 4352, 4096)]


@pytest.mark.parametrize("shape", SPLIT_SHAPES)
def test_split_last_wave(capi, oracle, cuda, shape):
    M, N, K = shape
    case = make_case(oracle, 44, M, N, K)
    rows = None if M <= 1024 else (M - 700, 700)
    capi.clear_workspace()
    n0 = capi.split_launch_count()
    gq, gs, gf = gpu_mm(capi, cuda, *case, workspace=False)
    assert capi.split_launch_count() == n0
    check_against_oracle(oracle, *case, gq, gs, gf, rows=rows)
    gq2, gs2, gf2 = gpu_mm(capi, cuda, *case, workspace=True)
    # the split does take place for these shapes (both entry points), otherwise this test checks nothing
    assert capi.split_launch_count() == n0 + 2
    check_against_oracle(oracle, *case, gq2, gs2, gf2, rows=rows)
    # splitting changes only the order of the fp32 promotion sums
    assert np.abs(gf - gf2).max() <= 4e-6 * np.abs(gf).max()
    # bitwise stable from call to call: counters reset themselves, pieces are added in a fixed order
    gq3, gs3, gf3 = gpu_mm(capi, cuda, *case, workspace=True)
    assert np.array_equal(gq2, gq3) and np.array_equal(gs2.view(np.uint32), gs3.view(np.uint32)) and np.array_equal(gf2, gf3)


@pytest.mark.parametrize("M", [1, 16, 64])
def test_decode_launch_chain_with_static_weights(capi, oracle, cuda, M):
    # Back-to-back launches without synchronisation, each using the previous one's stream position: with the
    # static-weights promise a launch prefetches its weights while the one before it is finishing; results
    # must be what the un-promised chain gives, bit for bit, and right.
    N, K = 2560, 4096
    cases = [make_case(oracle, 80 + i, M, N, K) for i in range(3)]
    dev = [to_dev(cuda, *c) for c in cases]
    capi.ensure_workspace(M, N, K)

    def chain():
        outs = []
        for rep in range(4):
            for dA, dAs, dB, dBs in dev:
                Cq = torch.full((M, N), 0xAA, dtype=torch.uint8, device=cuda)
                Cs = torch.full((N // 128, M), float("nan"), device=cuda)
                outs.append((Cq, Cs))
        i = 0
        for rep in range(4):
            for dA, dAs, dB, dBs in dev:
                capi.fp8_blockwise_mm(dA, dAs, dB, dBs, outs[i][0], outs[i][1], M, N, K)
                i += 1
        torch.cuda.synchronize()
        capi.check_status()
        return outs

    plain = chain()
    capi.set_static_weights(True)
    try:
        promised = chain()
    finally:
        capi.set_static_weights(False)
    for (q0, s0), (q1, s1) in zip(plain, promised):
        assert torch.equal(q0, q1) and torch.equal(s0, s1)
    for i, case in enumerate(cases):
        Cf = torch.empty(M, N, device=cuda)
        capi.fp8_blockwise_mm_f32(*dev[i], Cf, M, N, K)
        torch.cuda.synchronize()
        check_against_oracle(oracle, *case, promised[i][0].cpu().numpy(), promised[i][1].cpu().numpy(), Cf.cpu().numpy())


@pytest.mark.parametrize("M", [1, 64])
@pytest.mark.parametrize("NK", [(19456, 2560), (2560, 9728)])
def test_static_weights_written_by_the_kernel_before_the_last(capi, cuda, M, NK):
    # weight transposed or quantised, activations quantised, decode GEMM, with nothing in between: the early reads of the
    # GEMM find the new weight and its scales
    N, K = NK
    g = torch.Generator(device=cuda).manual_seed(64)
    x = torch.randn(M, K, device=cuda, generator=g)
    w = [torch.randn(N, K, device=cuda, generator=g) * s for s in (0.02, 3.0)]
    A_q, A_s = torch.empty(M, K, dtype=torch.uint8, device=cuda), torch.empty(K // 128, M, device=cuda)
    B_q, B_s = torch.empty(N, K, dtype=torch.uint8, device=cuda), torch.empty(N // 128, K // 128, device=cuda)
    B_t, B_kn = torch.empty_like(B_q), [torch.randint(0, 120, (K, N), dtype=torch.uint8, device=cuda, generator=g) for _ in range(2)]
    C = torch.empty(M, N, device=cuda)
    capi.ensure_workspace(M, N, K)

    def call(i, wait):
        outs = []
        for quantised in (True, False):
            if quantised:
                capi.fp8_quant_128x128(w[i], B_q, B_s, N, K)
            else:
                capi.transpose_aligned_128(B_t, B_kn[i], K, N)
            wait()
            capi.fp8_quant_1x128(x, A_q, A_s, M, K)
            capi.fp8_blockwise_mm_f32(A_q, A_s, B_q if quantised else B_t, B_s, C, M, N, K)
            outs.append(C.clone())
        return outs

    expected = [call(i, torch.cuda.synchronize) for i in range(2)]
    capi.set_static_weights(True)
    try:
        for rep in range(10):
            for a, b in zip(call(rep & 1, lambda: None), expected[rep & 1]):
                assert torch.equal(a, b)
    finally:
        capi.set_static_weights(False)
    capi.check_status()


# single-CTA, 128-row pair and 256-row pair kernel: K longer than the ring and the tiles requested into L2, K shorter than the
# ring, an odd number of groups (a second column half beyond the matrix), tiles and slices cut along K
@pytest.mark.parametrize("shape", [(100, 19456, 2560), (100, 19456, 256), (100, 2560, 9728), (100, 384, 256), (300, 9600, 1920), (2310, 640, 256),
                                   (2304, 4352, 2048)], ids=lambda s: "x".join(map(str, s)))
def test_static_weights_above_64_rows(capi, cuda, shape):
    # the first weight tiles are read before the quantiser of the activations has finished, the activations are not
    M, N, K = shape
    g = torch.Generator(device=cuda).manual_seed(65)
    x = [torch.randn(M, K, device=cuda, generator=g) * s for s in (1.0, 4.0)]
    w = [torch.randn(N, K, device=cuda, generator=g) * 0.02 for _ in range(2)]
    A_q, A_s = torch.empty(M, K, dtype=torch.uint8, device=cuda), torch.empty(K // 128, M, device=cuda)
    B_q, B_s = torch.empty(N, K, dtype=torch.uint8, device=cuda), torch.empty(N // 128, K // 128, device=cuda)
    C, C_q, C_s = torch.empty(M, N, device=cuda), torch.empty(M, N, dtype=torch.uint8, device=cuda), torch.empty(N // 128, M, device=cuda)
    capi.ensure_workspace(M, N, K)

    def call(i, wait):
        capi.fp8_quant_128x128(w[i], B_q, B_s, N, K)
        wait()
        capi.fp8_quant_1x128(x[i], A_q, A_s, M, K)
        capi.fp8_blockwise_mm_f32(A_q, A_s, B_q, B_s, C, M, N, K)
        capi.fp8_quant_1x128(x[1 - i], A_q, A_s, M, K)
        capi.fp8_blockwise_mm(A_q, A_s, B_q, B_s, C_q, C_s, M, N, K)
        return C.clone(), C_q.clone(), C_s.clone()

    capi.set_static_weights(False)
    expected = [call(i, torch.cuda.synchronize) for i in range(2)]
    capi.set_static_weights(True)
    try:
        for rep in range(6):
            for a, b in zip(call(rep & 1, lambda: None), expected[rep & 1]):
                assert torch.equal(a, b)
    finally:
        capi.set_static_weights(False)
    capi.check_status()


@pytest.mark.parametrize("shape", [(128, 2560, 4096), (65, 512, 2048), (100, 4096, 1024)])
def test_mid_m_few_tiles_take_the_pair_kernel_with_scratch(capi, oracle, cuda, shape):
    # 65..128 rows, tiles on at most half of the SMs: single-CTA kernel without scratch, pair kernel (whose tiles
    # are cut along K) with it; both against the oracle, and within the order of fp32 sums of each other
    M, N, K = shape
    case = make_case(oracle, 45, M, N, K)
    capi.clear_workspace()
    assert "fp8_blockwise_gemm_kernel" in capi.describe_plan("fp8", M, N, K)
    gq, gs, gf = gpu_mm(capi, cuda, *case, workspace=False)
    check_against_oracle(oracle, *case, gq, gs, gf)
    capi.ensure_workspace(M, N, K)
    assert "fp8_blockwise_gemm_pair_kernel" in capi.describe_plan("fp8", M, N, K)
    gq2, gs2, gf2 = gpu_mm(capi, cuda, *case, workspace=True)
    check_against_oracle(oracle, *case, gq2, gs2, gf2)
    assert np.abs(gf - gf2).max() <= 4e-6 * np.abs(gf).max()


@pytest.mark.parametrize("shape", [(1 + 64, 256, 1024), (127, 384, 2176), (128, 2560, 1280), (100, 6144, 1152), (65, 9472, 512),
                                   (129, 2560, 2048), (191, 640, 3200), (257, 1280, 2560), (384, 896, 1152), (641, 512, 1280), (1030, 256, 4096), (300, 512, 9344), (257, 1408, 9728), (65, 256, 16896)])
def test_pair_kernel_128_row_tiles(capi, oracle, cuda, shape):
    # one to four pairs per tile (10 to 74 tiles), rows and column groups beyond the matrix, slices of K of unequal length,
    # K-blocks that are no multiple of the scale ring's four; slices with one and two folds of the sum
    M, N, K = shape
    case = make_case(oracle, 48, M, N, K)
    capi.clear_workspace()
    gq, gs, gf = gpu_mm(capi, cuda, *case, workspace=False)
    capi.ensure_workspace(M, N, K)
    assert "pair_kernel_m128" in capi.describe_plan("fp8", M, N, K)
    gq2, gs2, gf2 = gpu_mm(capi, cuda, *case)
    check_against_oracle(oracle, *case, gq2, gs2, gf2)
    assert np.abs(gf - gf2).max() <= 4e-6 * np.abs(gf).max()
    gq3, gs3, gf3 = gpu_mm(capi, cuda, *case)
    assert np.array_equal(gq2, gq3) and np.array_equal(gs2, gs3) and np.array_equal(gf2, gf3)


@pytest.mark.parametrize("shape", [(512, 4096, 4096), (700, 2560, 4096)])
def test_long_slices_are_folded(capi, cuda, shape):
    # Whole tiles of 32 K-blocks, which the 256-row kernel would cut in two: their sums are kept in two pieces too.  Measured against the same rows of a larger problem, whose whole 256-row tiles are one chain over K: halves of a
    # chain have 1 / sqrt(2) of its random-walk error (a quarter or so of it, the block sums, is common to both).
    M, N, K = shape
    big = 4096
    A_q, A_s, B_q, B_s = full_size_case(capi, cuda, big, N, K, 63, 0.02)
    capi.ensure_workspace(M, N, K)
    assert "pair_kernel_m128" in capi.describe_plan("fp8_f32out", M, N, K)
    C, C_big = torch.empty(M, N, device=cuda), torch.empty(big, N, device=cuda)
    capi.fp8_blockwise_mm_f32(A_q[:M], A_s[:, :M].contiguous(), B_q, B_s, C, M, N, K)
    out = [(torch.empty(M, N, dtype=torch.uint8, device=cuda), torch.empty(N // 128, M, device=cuda)) for _ in range(2)]
    capi.fp8_blockwise_mm(A_q[:M], A_s[:, :M].contiguous(), B_q, B_s, *out[0], M, N, K)
    capi.fp8_blockwise_mm_gather(A_q[:M], A_s[:, :M].contiguous(), B_q, B_s, [out[1][0]], [out[1][1]], N, 0, M, N, K)
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    capi.clear_workspace()
    capi.fp8_blockwise_mm_f32(A_q, A_s, B_q, B_s, C_big, big, N, K)
    torch.cuda.synchronize()
    capi.check_status()
    exact = fp8_blockwise_acc_f64(A_q[:M], A_s[:, :M], B_q, B_s)
    err, err_big = (float((c.double() - exact).norm() / exact.norm()) for c in (C, C_big[:M]))
    assert err <= 0.9 * err_big, (err, err_big)


@pytest.mark.parametrize("shape", [(100, 512, 2176), (100, 9472, 256), (300, 384, 1664), (700, 2560, 512)])
@pytest.mark.parametrize("gather", [False, True])
def test_nan_columns_leave_the_rest_of_their_group_alone(capi, oracle, cuda, shape, gather):
    # Four adjacent weight rows of NaN codes (the four columns of one lane) and one activation row of them, on tiles that
    # are cut along K and on whole ones: every other code and scale is what it is with those weight rows zero.
    M, N, K = shape
    A_q, A_s, B_q, B_s = make_case(oracle, 50, M, N, K)
    bad = slice(N - 128 + 60, N - 128 + 64)
    A_q[M - 3] = 0x7F
    dA, dAs, dB, dBs = to_dev(cuda, A_q, A_s, B_q, B_s)
    capi.ensure_workspace(M, N, K)
    assert "pair_kernel_m128" in capi.describe_plan("fp8", M, N, K)
    outs = []
    for code in (0x00, 0x7F):
        dB[bad] = code
        Cq, Cs = torch.full((M, N), 0xAA, dtype=torch.uint8, device=cuda), torch.full((N // 128, M), -1.0, device=cuda)
        if gather:
            capi.fp8_blockwise_mm_gather(dA, dAs, dB, dBs, [Cq], [Cs], N, 0, M, N, K)
        else:
            capi.fp8_blockwise_mm(dA, dAs, dB, dBs, Cq, Cs, M, N, K)
        torch.cuda.synchronize()
        outs.append((Cq.cpu().numpy(), Cs.cpu().numpy()))
    capi.check_status()
    (q0, s0), (q1, s1) = outs
    assert np.isfinite(s1).all() and np.array_equal(s0, s1)
    assert (s1[:, M - 3] == 0).all() and ((q1[M - 3] & 0x7F) == 0x7F).all()
    assert ((q1[:, bad] & 0x7F) == 0x7F).all()
    other = np.ones(N, dtype=bool)
    other[bad] = False
    assert np.array_equal(q0[:, other], q1[:, other])


def gpu_c_quant(acc):
    """The output quantisation rule in torch fp32 on the GPU (for full-size property checks)."""
    M, N = acc.shape
    g = acc.view(M, N // 128, 128)
    amax = g.abs().amax(dim=2, keepdim=True)
    c448 = torch.full_like(amax, 448.0)  # tensor / tensor is an IEEE division; tensor / python-scalar multiplies by 1/448
    scale = amax / c448
    inv = torch.where(amax > 0, c448 / amax, torch.zeros_like(amax))
    q = (g * inv).to(torch.float8_e4m3fn).view(torch.uint8).view(M, N)
    return q, scale.squeeze(2).t().contiguous()


def full_size_case(capi, cuda, M, N, K, seed, w_std):
    g = torch.Generator(device=cuda).manual_seed(seed)
    x = torch.randn(M, K, device=cuda, generator=g)
    w = torch.randn(N, K, device=cuda, generator=g) * w_std
    A_q = torch.empty(M, K, dtype=torch.uint8, device=cuda)
    A_s = torch.empty(K // 128, M, device=cuda)
    B_q = torch.empty(N, K, dtype=torch.uint8, device=cuda)
    B_s = torch.empty(N // 128, K // 128, device=cuda)
    capi.fp8_quant_1x128(x, A_q, A_s, M, K)
    capi.fp8_quant_128x128(w, B_q, B_s, N, K)
    return A_q, A_s, B_q, B_s


@pytest.mark.parametrize("shape", [(4096, 4096, 4096, 1.0), (4096, 6144, 2560, 0.02), (4096, 2560, 9728, 0.02)])
def test_full_size_properties_and_sampled_rows(capi, oracle, cuda, shape):
    M, N, K, w_std = shape
    A_q, A_s, B_q, B_s = full_size_case(capi, cuda, M, N, K, 60, w_std)
    capi.ensure_workspace(M, N, K)
    Cq = torch.full((M, N), 0xAA, dtype=torch.uint8, device=cuda)
    Cs = torch.full((N // 128, M), float("nan"), device=cuda)
    Cf = torch.full((M, N), float("nan"), device=cuda)
    capi.fp8_blockwise_mm(A_q, A_s, B_q, B_s, Cq, Cs, M, N, K)
    capi.fp8_blockwise_mm_f32(A_q, A_s, B_q, B_s, Cf, M, N, K)
    # (a) fused output == rule(own accumulator), everywhere, bit for bit
    q_rule, s_rule = gpu_c_quant(Cf)
    assert torch.equal(Cs, s_rule)
    assert torch.equal(Cq, q_rule)
    # (b) linearity: doubling the activation scales doubles the accumulator and the output scales exactly
    Cq2 = torch.empty_like(Cq)
    Cs2 = torch.empty_like(Cs)
    capi.fp8_blockwise_mm(A_q, A_s * 2, B_q, B_s, Cq2, Cs2, M, N, K)
    assert torch.equal(Cq2, Cq) and torch.equal(Cs2, Cs * 2)
    # (c) erasure: zeroed activation rows give zero bytes and zero scales (the defined all-zero case)
    A_q0 = A_q.clone()
    A_q0[100:228] = 0
    capi.fp8_blockwise_mm(A_q0, A_s, B_q, B_s, Cq2, Cs2, M, N, K)
    assert bool((Cq2[100:228] == 0).all()) and bool((Cs2[:, 100:228] == 0).all())
    assert torch.equal(Cq2[228:], Cq[228:]) and torch.equal(Cq2[:100], Cq[:100])
    torch.cuda.synchronize()
    capi.check_status()
    # (d) sampled whole rows against the CPU oracle
    hA_q, hA_s, hB_q, hB_s = (t.cpu().numpy() for t in (A_q, A_s, B_q, B_s))
    gq, gs, gf = Cq.cpu().numpy(), Cs.cpu().numpy(), Cf.cpu().numpy()
    for r0 in (0, 127, 2049, M - 4):
        check_against_oracle(oracle, hA_q, hA_s, hB_q, hB_s, gq, gs, gf, rows=(r0, 4))


def test_reference_launcher_errors(capi, cuda):
    z8 = torch.zeros(128, 128, dtype=torch.uint8, device=cuda)
    zf = torch.zeros(128, 128, device=cuda)
    with pytest.raises(RuntimeError, match="not aligned"):
        capi.fp8_blockwise_mm(z8, zf, z8, zf, z8, zf, 128, 100, 128)
