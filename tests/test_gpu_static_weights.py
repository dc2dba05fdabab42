"""Static weights (capi.set_static_weights) in the fused forms above 64 rows, and in the plain one where the weight has fewer rows
than the activations: the first weight tiles are read before the quantiser of the activations has finished, the activations are
not.  The weight quantiser runs before that quantiser.  Results equal those of calls that read nothing early, bit for bit."""
import pytest
import torch

from llmmm_b200.host_pipeline import Fp8GemmHostPipeline

pytestmark = pytest.mark.gpu

# (form, M, columns of the output, K): the 128-row and the 256-row kernel, K shorter and longer than their rings, a ragged last row
# of tiles, several tiles per pair of CTAs
CASES = [("swiglu", 100, 1280, 256), ("swiglu", 100, 9728, 2560), ("swiglu", 300, 1280, 1920), ("swiglu", 1333, 9728, 512),
         ("rope", 100, 6144, 256), ("rope", 300, 6144, 2560), ("rope", 1333, 6144, 512),
         ("gather", 100, 1280, 256), ("gather", 300, 2560, 1920), ("gather", 1333, 6400, 1024),
         ("plain", 300, 256, 1280), ("plain", 700, 512, 1024), ("plain", 1333, 512, 6144)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_early_weights_change_nothing(capi, cuda, case):
    form, M, N, K = case
    rows = 2 * N if form == "swiglu" else N
    g = torch.Generator(device=cuda).manual_seed(66)
    x = [torch.randn(M, K, device=cuda, generator=g) * s for s in (1.0, 4.0)]
    w = [torch.randn(rows, K, device=cuda, generator=g) * 0.02 for _ in range(2)]
    A_q, A_s = torch.empty(M, K, dtype=torch.uint8, device=cuda), torch.empty(K // 128, M, device=cuda)
    B_q, B_s = torch.empty(rows, K, dtype=torch.uint8, device=cuda), torch.empty(rows // 128, K // 128, device=cuda)
    C_q, C_s = torch.empty(M, N, dtype=torch.uint8, device=cuda), torch.empty(N // 128, M, device=cuda)
    angles = torch.arange(M, device=cuda)[:, None] * 0.01 * torch.arange(1, 65, device=cuda)
    pos, cos, sin = torch.arange(M, dtype=torch.int32, device=cuda), angles.cos().contiguous(), angles.sin().contiguous()
    norm = torch.rand(128, device=cuda, generator=g) + 0.5
    n_kv = N // 128 // 6
    capi.ensure_workspace(M, rows, K)

    def call(i, wait):
        capi.fp8_quant_128x128(w[i], B_q, B_s, rows, K)
        wait()
        capi.fp8_quant_1x128(x[i], A_q, A_s, M, K)
        if form == "swiglu":
            capi.fp8_blockwise_mm_swiglu(A_q, A_s, B_q, B_s, C_q, C_s, M, N, K)
        elif form == "rope":
            capi.fp8_blockwise_mm_qk_norm_rope(A_q, A_s, B_q, B_s, C_q, C_s, pos, cos, sin, norm, norm, 1e-6, N // 128 - 2 * n_kv, n_kv, M, N, K)
        elif form == "gather":
            capi.fp8_blockwise_mm_gather(A_q, A_s, B_q, B_s, [C_q], [C_s], N, 0, M, N, K)
        else:
            capi.fp8_blockwise_mm(A_q, A_s, B_q, B_s, C_q, C_s, M, N, K)
        return C_q.clone(), C_s.clone()

    capi.set_static_weights(False)
    expected = [call(i, torch.cuda.synchronize) for i in range(2)]
    assert not torch.equal(expected[0][0], expected[1][0])
    capi.set_static_weights(True)
    try:
        for rep in range(6):
            for a, b in zip(call(rep & 1, lambda: None), expected[rep & 1]):
                assert torch.equal(a, b)
    finally:
        capi.set_static_weights(False)
    capi.check_status()


@pytest.mark.parametrize("shape", [(16, 2560, 4096), (100, 2560, 4096), (1000, 9600, 1024)], ids=lambda s: "x".join(map(str, s)))
def test_weights_copied_from_the_host_before_every_call(capi, cuda, shape):
    # the copies run on another stream and are waited for by an event: the next kernel must not start, and read, before them
    M, N, K = shape
    g = torch.Generator(device=cuda).manual_seed(67)
    calls = []
    for i in range(6):
        A_q, A_s = torch.empty(M, K, dtype=torch.uint8, device=cuda), torch.empty(K // 128, M, device=cuda)
        B_q, B_s = torch.empty(N, K, dtype=torch.uint8, device=cuda), torch.empty(N // 128, K // 128, device=cuda)
        capi.fp8_quant_1x128(torch.randn(M, K, device=cuda, generator=g), A_q, A_s, M, K)
        capi.fp8_quant_128x128(torch.randn(N, K, device=cuda, generator=g), B_q, B_s, N, K)
        calls.append((A_q, A_s, B_q, B_s))
    pipe = Fp8GemmHostPipeline(M, N, K, depth=2, device=cuda)
    expected = []
    for ops in calls:
        C_q, C_s = torch.empty(M, N, dtype=torch.uint8, device=cuda), torch.empty(N // 128, M, device=cuda)
        capi.fp8_blockwise_mm(*ops, C_q, C_s, M, N, K)
        expected.append((C_q.cpu(), C_s.cpu()))
    host = [[t.cpu().pin_memory() for t in ops] for ops in calls]
    results = [(torch.empty(M, N, dtype=torch.uint8).pin_memory(), torch.empty(N // 128, M).pin_memory()) for _ in calls]
    capi.set_static_weights(True)
    try:
        for ops, out in zip(host, results):
            pipe.submit(*ops, *out)
        pipe.drain()
    finally:
        capi.set_static_weights(False)
    for got, want in zip(results, expected):
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
