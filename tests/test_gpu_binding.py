"""The native form of the calls (csrc/binding.cpp) against the ctypes form of the same calls: the same bytes, on the
current stream, on a given stream (object or handle) and with keywords; what is not the plain case is left to ctypes."""
import pytest
import torch

from test_gpu_fp8 import full_size_case

pytestmark = pytest.mark.gpu


def calls(capi, cuda, M):
    """(name, arguments up to the stream, outputs) of every call that has a native form."""
    K, I, n_q, n_kv = 256, 256, 2, 1
    N = (n_q + 2 * n_kv) * 128
    q = full_size_case(capi, cuda, M, N, K, 5, 0.05)
    gu = full_size_case(capi, cuda, M, 2 * I, K, 6, 0.05)
    g = torch.Generator(device=cuda).manual_seed(7)
    x = torch.randn(M, K, device=cuda, generator=g)
    x2 = torch.randn(256, K, device=cuda, generator=g)
    w = torch.rand(K, device=cuda, generator=g)
    cos, sin = torch.rand(32, 64, device=cuda, generator=g), torch.rand(32, 64, device=cuda, generator=g)
    pos = torch.randint(0, 32, (M,), device=cuda, dtype=torch.int32, generator=g)
    b = lambda *s: torch.zeros(*s, dtype=torch.uint8, device=cuda)  # noqa: E731
    f = lambda *s: torch.zeros(*s, device=cuda)  # noqa: E731
    out = []
    for dt in (torch.float16, torch.bfloat16):
        A, B, C = torch.randn(M, 64, device=cuda, generator=g).to(dt), torch.randn(64, 64, device=cuda, generator=g).to(dt), f(M, 64).to(dt)
        out.append(("fp16_mm", (A, B, C, M, 64, 64), (C,)))
    C = (b(M, N), f(N // 128, M))
    out.append(("fp8_blockwise_mm", (*q, *C, M, N, K), C))
    C = (f(M, N),)
    out.append(("fp8_blockwise_mm_f32", (*q, *C, M, N, K), C))
    C = (b(M, I), f(I // 128, M))
    out.append(("fp8_blockwise_mm_swiglu", (*gu, *C, M, I, K), C))
    for weights in ((w[:128].clone(), w[128:].clone()), (None, None)):
        C = (b(M, N), f(N // 128, M))
        out.append(("fp8_blockwise_mm_qk_norm_rope", (*q, *C, pos, cos, sin, *weights, 1e-6, n_q, n_kv, M, N, K), C))
    C = (b(M, K), f(K // 128, M))
    out.append(("fp8_quant_1x128", (x, *C, M, K), C))
    C = (b(256, K), f(2, K // 128))
    out.append(("fp8_quant_128x128", (x2, *C, 256, K), C))
    C = (b(M, K), f(K // 128, M))
    out.append(("fp8_rmsnorm_quant_1x128", (x, w, 1e-6, *C, M, K), C))
    return out


@pytest.mark.parametrize("M", [1, 130])
def test_native_calls_match_ctypes(capi, cuda, monkeypatch, M):
    assert capi._native is not None
    capi.ensure_workspace(M, 512, 256)
    s = torch.cuda.Stream(device=cuda)
    for name, args, outs in calls(capi, cuda, M):
        def run(native, **kw):
            for o in outs:
                o.zero_()
            torch.cuda.synchronize()
            with monkeypatch.context() as m:
                if not native:
                    m.setattr(capi, "_native", None)
                getattr(capi, name)(*args, **kw)
            torch.cuda.synchronize()
            return [o.clone() for o in outs]

        want = run(False)
        assert any(bool(o.any()) for o in want), name
        for kw in ({}, {"stream": s}, {"stream": s.cuda_stream}):
            assert getattr(capi._native, name)(*args, kw.get("stream")) is True, name
            for got, w in zip(run(True, **kw), want):
                assert torch.equal(got, w), (name, kw)
        # not the plain case: nothing is done, ctypes decides
        first = args[0]
        for bad in (first.cpu(), first[..., ::2], "x", None):
            assert getattr(capi._native, name)(bad, *args[1:], None) is False, name
        assert getattr(capi._native, name)(*args[:-1], 1.5, None) is False
        assert getattr(capi._native, name)(*args[:-1], 2 ** 40, None) is False
        with pytest.raises(RuntimeError, match="contiguous CUDA tensor"):
            getattr(capi, name)(first[..., ::2], *args[1:])
    capi.check_status()


def test_library_errors_through_the_native_call(capi, cuda):
    z8 = torch.zeros(128, 128, dtype=torch.uint8, device=cuda)
    zf = torch.zeros(128, 128, device=cuda)
    with pytest.raises(RuntimeError, match="llmmm status .*not aligned"):
        capi._native.fp8_blockwise_mm(z8, zf, z8, zf, z8, zf, 128, 100, 128, None)
