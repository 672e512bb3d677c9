"""Few-token weight-streaming kernels ('lines', 'small') on the GPU against the CPU oracle and the reference's own CUDA library."""
import pytest
import torch

from oracle import int8_oracle as oracle
from tests import reflib
from tests.gpu_common import rand_int8, randn, rel

pytestmark = pytest.mark.gpu


def case(m, n, k, dtype, seed, residual):
    g = torch.Generator().manual_seed(seed)
    x = randn((m, k), dtype, seed)
    x[:, :4] = 1000.0 if dtype == torch.bfloat16 else 100.0  # massive-activation channels
    w = rand_int8((n, k), seed + 1)
    sw = torch.rand(n, generator=g) * 0.002 + 0.0001
    bias = randn((n,), dtype, seed + 2)
    res = randn((m, n), dtype, seed + 3, 4.0) if residual else None
    rs = torch.rand(n, generator=g).to(dtype) if residual else None
    return x, w, sw, bias, res, rs


def cuda(*tensors):
    return [None if t is None else t.cuda() for t in tensors]


@pytest.fixture(params=["planes", "converted"])
def kernel(request, wq, monkeypatch):
    """Both few-token kernels for shapes of at most 8 tokens: 'planes' (activations as INT8 digit planes, the Python module's choice) and
    'converted' (weights converted to the activation type: what wq8_gemv_lines / wq8_small of the C ABI run, and every larger shape)."""
    if request.param == "converted":
        monkeypatch.setattr(wq, "_stream_planes", lambda *args: False)
    return request.param


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("residual", [False, True], ids=["plain", "residual"])
@pytest.mark.parametrize("shape", [(1, 96, 256), (2, 100, 260), (3, 4096, 1024), (4, 520, 4096 + 64), (4, 28672, 4096), (1, 4096, 14336)], ids=str)
def test_lines(wq, kernel, shape, residual, dtype):
    m, n, k = shape
    x, w, sw, bias, res, rs = case(m, n, k, dtype, 101, residual)
    gx, gw, gsw, gbias, gres, grs = cuda(x, w, sw, bias, res, rs)
    y = wq.gemv_lines(gx, gw, gsw, gbias, gres, grs)
    expected = oracle.weight_only(x, w.numpy(), sw.numpy(), bias, res, rs, dtype)
    assert rel(y, expected) < 1e-3
    y_ref = reflib.gemv_lines(gx, gw, gsw, gbias, gres, grs)
    assert rel(y, y_ref) < 1e-3
    assert torch.equal(y, wq.gemv_lines(gx, gw, gsw, gbias, gres, grs))  # fixed-order reductions: run to run identical
    assert wq.debug_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("residual", [False, True], ids=["plain", "residual"])
@pytest.mark.parametrize("shape", [(5, 96, 256), (8, 1000, 1024), (16, 28672, 4096), (16, 4096, 14336), (32, 4096, 14336), (32, 1024, 8192), (9, 40, 64),
                                   (24, 2048, 4096)], ids=str)
def test_small(wq, kernel, shape, residual, dtype):
    m, n, k = shape
    x, w, sw, bias, res, rs = case(m, n, k, dtype, 111, residual)
    gx, gw, gsw, gbias, gres, grs = cuda(x, w, sw, bias, res, rs)
    y = wq.small(gx, gw, gsw, gbias, gres, grs)
    expected = oracle.weight_only(x, w.numpy(), sw.numpy(), bias, res, rs, dtype)
    assert rel(y, expected) < 1e-3
    y_ref = reflib.small(gx, gw, gsw, gbias, gres, grs)
    assert rel(y, y_ref) < 1e-3
    assert torch.equal(y, wq.small(gx, gw, gsw, gbias, gres, grs))  # fixed-order reductions: run to run identical
    # the split-K counters are left zeroed
    assert not wq._counters[0].any().item()
    assert wq.debug_status() == 0


def test_small_in_place_residual(wq):
    x, w, sw, bias, res, rs = case(12, 1024, 2048, torch.bfloat16, 121, True)
    gx, gw, gsw, gbias, gres, grs = cuda(x, w, sw, bias, res, rs)
    y = wq.small(gx, gw, gsw, gbias, gres, grs)
    target = gres.clone()
    wq.small(gx, gw, gsw, gbias, target, grs, out=target)
    assert torch.equal(y, target)


def test_strided_activation(wq):
    wide = randn((4, 4096), torch.bfloat16, 131).cuda()
    x = wide[:, 1024:3072]
    w = rand_int8((256, 2048), 132).cuda()
    sw = torch.full((256,), 0.001).cuda()
    assert torch.equal(wq.gemv_lines(x, w, sw), wq.gemv_lines(x.contiguous(), w, sw))
    assert torch.equal(wq.small(x, w, sw), wq.small(x.contiguous(), w, sw))


def test_planes_keep_small_values_next_to_large_ones(wq):
    """The digit planes share one power of two per 128 values: values down to 2^-14 of the largest of their run are exact, so a run that
    mixes 1000.0 with values around 0.5 still gives the FP32 result."""
    m, n, k = 4, 512, 4096
    g = torch.Generator().manual_seed(5)
    x = (torch.randn(m, k, generator=g) * 0.5).to(torch.bfloat16)
    x[:, ::128] = 1000.0
    w = rand_int8((n, k), 6)
    w[:, ::128] = 0  # the large values do not contribute: the result is made of the small ones only
    sw = torch.full((n,), 0.001)
    y = wq.gemv_lines(x.cuda(), w.cuda(), sw.cuda())
    expected = (x.double() @ w.double().T * 0.001).to(torch.bfloat16)
    assert rel(y, expected) < 2e-3
    assert wq.debug_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("tokens", [1, 4, 8])
@pytest.mark.parametrize("shape", [(28672, 4096), (4096, 14336)], ids=["up", "down"])
def test_planes_with_an_outlier_in_every_run(wq, shape, tokens, dtype):
    """The worst case of the digit-plane kernel: every run of 128 activations holds one value 2^10 times larger than the rest and all
    weights are live, so the small values carry the fewest digits.  Bar: 1e-3 against the reference's own CUDA kernels, which multiply
    the unrewritten activations; and the planes must actually be the kernel that ran."""
    n, k = shape
    g = torch.Generator().manual_seed(77)
    x = torch.randn(tokens, k, generator=g)
    x[:, 5::128] *= 1024.0
    x = x.to(dtype)
    w = rand_int8((n, k), 78)
    sw = torch.rand(n, generator=g) * 0.002 + 0.0001
    bias = randn((n,), dtype, 79)
    gx, gw, gsw, gbias = cuda(x, w, sw, bias)
    assert wq._require().wq8_stream_planes_workspace(tokens, n, k, 148) > 0
    for entry, reference in ((wq.gemv_lines, reflib.gemv_lines), (wq.small, reflib.small)):
        if entry is wq.gemv_lines and tokens > 4:
            continue
        y = entry(gx, gw, gsw, gbias)
        assert rel(y, reference(gx, gw, gsw, gbias)) < 1e-3
        exact = (x.double() @ (w.double() * sw.double()[:, None]).T + bias.double())
        assert rel(y, exact.float()) < 4e-3  # the output's own rounding to 8 or 11 bits
    assert wq.debug_status() == 0


@pytest.mark.parametrize("entry,m", [("gemv_lines", 1), ("gemv_lines", 4), ("small", 8), ("small", 9), ("small", 16), ("small", 29)])
def test_weights_straight_from_the_quantizer(wq, entry, m):
    """The few-token kernels request weights before their digits are ready: codes that the kernel right before the call writes have to be the ones
    that are used.  The buffers are the same ones over and over, with the opposite codes in them each time."""
    n, k = 6144, 4096
    g = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    w = torch.randn(n, k, device="cuda", generator=g).to(torch.bfloat16)
    weights, call = (w, -w), getattr(wq, entry)
    expected = []
    for source in weights:
        codes, _, scale = wq.quantize(source)
        torch.cuda.synchronize()
        expected.append(call(x, codes, scale))
        torch.cuda.synchronize()
    assert float((expected[0].float() + expected[1].float()).norm()) < 1e-3 * float(expected[0].float().norm())
    del codes, scale
    got = []
    for i in range(20):
        codes, _, scale = wq.quantize(weights[i % 2])
        got.append(call(x, codes, scale))
        del codes, scale  # the next round's codes go where these are
    for i, y in enumerate(got):
        assert torch.equal(y, expected[i % 2])
    assert wq.debug_status() == 0


FEW_SHAPES = [(8, 2048), (40, 2048 + 128), (1000, 4096), (16 * 148 + 24, 2048 + 384), (2304, 4096)]  # (N, K): fewer items than SMs, odd runs, partial items


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("act", [None, "swiglu", "gelu"])
@pytest.mark.parametrize("m,shape", [(m, shape) for m in (1, 2, 3, 4) for shape in FEW_SHAPES] + [(1, (520, 16384)), (1, (264, 5120)), (2, (520, 8192))], ids=str)
def test_input_operation_and_stream_in_one_launch(wq, m, shape, act, dtype):
    """wq8_few: op(x) rounded as transform_rows rounds it, then the oracle's product; the residual in place; the same bits every time."""
    n, k = shape
    assert wq._require().wq8_few_takes(m, n, k, wq.ACTS[act], 148) == 1
    _, w, sw, bias, res, rs = case(m, n, k, dtype, 141, True)
    x = randn((m, 2 * k if act == "swiglu" else k), dtype, 142)
    x[:, ::131] *= 60
    gx, gw, gsw, gbias, gres, grs = cuda(x, w, sw, bias, res, rs)
    prepared = wq.transform_rows(gx, 0, act).cpu() if act else x
    target = gres.clone()
    y = wq.linear(gx, gw, gsw, gbias, mode="lines", act=act, residual=target, residual_scale=grs, out=target)
    assert y is target
    assert rel(y, oracle.weight_only(prepared, w.numpy(), sw.numpy(), bias, res, rs, dtype)) < 1e-3
    assert torch.equal(y, wq.linear(gx, gw, gsw, gbias, mode="small" if k % 64 == 0 else "lines", act=act, residual=gres, residual_scale=grs))
    # rows of a wider matrix, and no bias or residual
    if act != "swiglu":
        wide = torch.zeros(m, k + 264, dtype=dtype, device="cuda")
        wide[:, 132:132 + k] = gx
        assert torch.equal(wq.linear(wide[:, 132:132 + k], gw, gsw, mode="lines", act=act), wq.linear(gx, gw, gsw, mode="lines", act=act))
    assert wq.debug_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("act", [None, "rms_norm", "swiglu", "gelu"])
@pytest.mark.parametrize("m,n,k", [(1, 520, 4096), (3, 1000, 4096 + 128), (4, 264, 14336), (2, 56 * 148, 16384), (4, 56 * 148 + 8, 5120), (3, 112 * 148, 4096), (3, 112 * 148 + 8, 4096),
                                   (3, 112 * 148, 5120), (3, 112 * 148 + 8, 5120)], ids=str)
def test_few_tokens_of_long_rows(wq, m, n, k, act, dtype):
    """Up to four tokens beyond one launch, on both sides of the numbers of channels at which the kernels change: op(x) rounded as transform_rows rounds
    it, and the oracle's product; wq8_small's bits on those rows where both run the planes; in place; the same bits every time and in both modes."""
    _, w, sw, bias, res, rs = case(m, n, k, dtype, 171, True)
    x = randn((m, 2 * k if act == "swiglu" else k), dtype, 172)
    x[:, ::131] *= 60
    norm = (1 + 0.1 * randn((k,), torch.float32, 173)).to(dtype) if act == "rms_norm" else None
    gx, gw, gsw, gbias, gres, grs, gnorm = cuda(x, w, sw, bias, res, rs, norm)
    prepared = wq.transform_rows(gx, 0, act, gnorm, 1e-6) if act else gx
    target = gres.clone()
    y = wq.linear(gx, gw, gsw, gbias, mode="lines", act=act, act_weight=gnorm, eps=1e-6, residual=target, residual_scale=grs, out=target)
    assert y is target
    assert rel(y, oracle.weight_only(prepared.cpu(), w.numpy(), sw.numpy(), bias, res, rs, dtype)) < 1e-3
    assert torch.equal(y, wq.linear(gx, gw, gsw, gbias, mode="small", act=act, act_weight=gnorm, eps=1e-6, residual=gres, residual_scale=grs))
    if n <= 56 * 148:  # the input operation by itself, then the streams: what linear_prepared() runs
        ready = wq.prepare(gx, 0, "lines", act, gnorm, 1e-6)
        assert torch.equal(y, wq.linear_prepared(ready, gw, gsw, gbias, gres, grs))
    assert not wq._counters[0].any().item() and wq.debug_status() == 0


@pytest.mark.parametrize("form", ["linear", "prepared"])
@pytest.mark.parametrize("m,act", [(1, "rms_norm"), (3, None), (16, "gelu")], ids=str)
def test_calls_on_several_streams_count_their_own_pieces(wq, m, act, form):
    """Tiles that several CTAs share, on streams that nothing orders and that prepare_stream() has not seen: the bits of a call alone.  The device's
    shared counters, whatever they hold, are no part of it."""
    n, k = 520, 6144
    _, w, sw, bias, _, _ = case(m, n, k, torch.float16, 161, False)
    xs = [randn((m, k), torch.float16, 162 + i).cuda() for i in range(4)]
    gw, gsw, gbias = cuda(w, sw, bias)
    assert wq._require().wq8_few_takes(m, n, k, wq.ACTS[act], 148) == 2

    def call(x):
        if form == "linear":
            return wq.linear(x, gw, gsw, gbias, mode="small", act=act, eps=1e-6)
        return wq.linear_prepared(wq.prepare(x, 0, "small", act, None, 1e-6), gw, gsw, gbias)

    alone = [call(x) for x in xs]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in xs]
    shared = wq._counters[0].clone()
    wq._counters[0].fill_(3)
    torch.cuda.synchronize()
    try:
        for _ in range(20):
            together = []
            for stream, x in zip(streams, xs):
                with torch.cuda.stream(stream):
                    together.append(call(x))
            torch.cuda.synchronize()
            assert all(torch.equal(a, b) for a, b in zip(alone, together))
        assert bool((wq._counters[0] == 3).all())
    finally:
        wq._counters[0].copy_(shared)
    assert wq.debug_status() == 0


def test_how_the_shapes_run(wq):
    takes = wq._require().wq8_few_takes
    assert [takes(m, 4096, 4096, 0, 148) for m in (1, 2, 3, 4, 5, 32, 33)] == [1, 1, 1, 1, 2, 2, 0]
    assert [takes(1, 4096, k, 0, 148) for k in (1024, 2048, 2048 + 64, 16384, 16384 + 128)] == [2, 1, 0, 1, 2]
    assert [takes(3, 4096, k, 0, 148) for k in (4096, 4096 + 128)] == [1, 2]
    assert [takes(1, 4096, 4096, act, 148) for act in (0, 1, 2, 3, 4)] == [1, 2, 1, 1, 0]
    assert [takes(9, 4096, k, act, 148) for act in (0, 1, 2, 3) for k in (128, 4096, 4096 + 64)] == [2, 2, 0] * 4


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("act", [None, "rms_norm", "swiglu", "gelu"])
@pytest.mark.parametrize("m,n,k", [(2, 264, 1024), (4, 1000, 6144 + 128), (5, 40, 128), (8, 1000, 1152), (9, 264, 4096 + 128), (16, 2048, 14336), (17, 129, 2048), (32, 520, 5120)], ids=str)
def test_input_operation_in_the_digit_split(wq, m, n, k, act, dtype, monkeypatch):
    """wq8_few in two launches: the digits of op(x) rounded as transform_rows rounds it, so the bits of wq8_small on those rows."""
    _, w, sw, bias, res, rs = case(m, n, k, dtype, 151, True)
    x = randn((m, 2 * k if act == "swiglu" else k), dtype, 152)
    x[:, ::131] *= 60
    x[1] = 0
    norm = (1 + 0.1 * randn((k,), torch.float32, 153)).to(dtype) if act == "rms_norm" else None
    gx, gw, gsw, gbias, gres, grs, gnorm = cuda(x, w, sw, bias, res, rs, norm)
    prepared = wq.transform_rows(gx, 0, act, gnorm, 1e-6) if act else gx
    monkeypatch.setattr(wq, "_stream_planes", lambda *args: False)  # wq8_small for any number of tokens
    expected = wq.small(prepared, gw, gsw, gbias, gres, grs)
    target = gres.clone()
    y = wq.linear(gx, gw, gsw, gbias, mode="small", act=act, act_weight=gnorm, eps=1e-6, residual=target, residual_scale=grs, out=target)
    assert y is target and torch.equal(y, expected)
    assert rel(y, oracle.weight_only(prepared.cpu(), w.numpy(), sw.numpy(), bias, res, rs, dtype)) < 1e-3
    if act == "rms_norm":  # without a weight
        assert torch.equal(wq.linear(gx, gw, gsw, mode="small", act=act, eps=1e-6), wq.small(wq.transform_rows(gx, 0, act, None, 1e-6), gw, gsw))
    assert not wq._counters[0].any().item() and wq.debug_status() == 0
