"""Activation preparation kernels on the GPU: bit-exact against the reference's own CUDA library, and against the CPU oracle."""
import numpy as np
import pytest
import torch

from oracle import int8_oracle as oracle
from tests import reflib
from tests.gpu_common import codes_close, randn

pytestmark = pytest.mark.gpu
ACTS = [None, "rms_norm", "swiglu", "gelu"]
# (M, K): ragged last block, register-resident rows of every size class, and a row longer than the register kernels hold
SHAPES = [(1, 8), (7, 264), (33, 2048), (5, 5120), (130, 1024 + 128 + 8), (3, 13824), (2, 16384 + 512)]


def make_x(m, k, act, dtype, seed):
    x = randn((m, 2 * k if act == "swiglu" else k), dtype, seed, 1.5)
    if m > 2:
        x[1] = 0  # an all-zero row
        x[2, ::7] *= 40  # outliers
    return x


def weight_of(k, act, dtype, seed):
    return (randn((k,), torch.float32, seed) * 0.1 + 1).to(dtype) if act == "rms_norm" else None


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("act", ACTS)
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"{s[0]}x{s[1]}")
def test_quantize_blocks_matches_reference_library(wq, shape, act, dtype):
    m, k = shape
    x = make_x(m, k, act, dtype, 11).cuda()
    w = weight_of(k, act, dtype, 12)
    w = None if w is None else w.cuda()
    q, s = wq.quantize_blocks(x, 0, act, w, 1e-6)
    q_ref, s_ref = reflib.quantize_blocks(x, 0, act, w, 1e-6)
    assert torch.equal(q, q_ref)
    assert torch.equal(s, s_ref)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("shape", [(37, 1024), (3000, 128), (3001, 1024 - 128), (3000, 1024), (1501, 1024 + 128), (300, 13824), (177, 16384 + 512), (3001, 264), (1500, 1536 + 8)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_gelu_codes_are_the_accurate_ones(wq, shape, dtype):
    """The block quantizer puts few elements through the accurate gelu; the row quantizer puts all of them.  On rows of one block both have the same
    scale to find, so codes and scales are the same bits: ordinary blocks, blocks without a value above 0.35, zeros, tiny and huge values,
    values next to nothing but one, infinities and NaN."""
    m, k = shape
    x = randn((m, k), torch.float32, 31)
    for i, change in enumerate((lambda v: v * 0.05, lambda v: -v.abs() - 0.4, lambda v: v * 0, lambda v: v * 1e-6, lambda v: v * 1e4,
                                lambda v: torch.where(v > 2.0, v, v * 1e-3))):
        x[i::7] = change(x[i::7])
    x = x.to(dtype)
    x.view(-1)[5::1009] = float("inf")
    x.view(-1)[7::1013] = -float("inf")
    x.view(-1)[9::997] = float("nan")
    q, s = wq.quantize_blocks(x.cuda(), 0, "gelu")
    rows = torch.nn.functional.pad(x, (0, -k % 128)).view(-1, 128).cuda()
    q_rows, _, s_rows = wq.quantize(rows, 0, False, "gelu")
    assert torch.equal(q, q_rows.view(m, -1)[:, :k]) and torch.equal(s, s_rows.view(m, -1))


@pytest.mark.parametrize("group", [16, 64, 256])
@pytest.mark.parametrize("act", [None, "rms_norm", "gelu"])
def test_quantize_blocks_rotated_matches_reference_library(wq, group, act):
    m, k = 9, 1024 + 256
    x = make_x(m, k, act, torch.bfloat16, 13).cuda()
    w = weight_of(k, act, torch.bfloat16, 14)
    w = None if w is None else w.cuda()
    q, s = wq.quantize_blocks(x, group, act, w, 1e-6)
    q_ref, s_ref = reflib.quantize_blocks(x, group, act, w, 1e-6)
    assert torch.equal(q, q_ref) and torch.equal(s, s_ref)


@pytest.mark.parametrize("act", ACTS)
@pytest.mark.parametrize("shape", [(7, 264), (5, 5120), (2, 16384 + 512)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_quantize_blocks_matches_oracle(wq, shape, act):
    m, k = shape
    x = make_x(m, k, act, torch.bfloat16, 15)
    w = weight_of(k, act, torch.bfloat16, 16)
    q, s = wq.quantize_blocks(x.cuda(), 0, act, None if w is None else w.cuda(), 1e-6)
    q_cpu, s_cpu = oracle.quantize_blocks(x, 0, act, w, 1e-6)
    if act in (None, "rms_norm"):  # IEEE operations only: identical
        assert codes_close(q, q_cpu, 1e-5)
        assert np.allclose(s.cpu().numpy(), s_cpu, rtol=3e-7, atol=0)
    else:  # expf / tanhf of the CUDA math library vs the host's
        assert codes_close(q, q_cpu, 2e-3)
        assert np.allclose(s.cpu().numpy(), s_cpu, rtol=2e-6, atol=0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("group", [16, 64, 256])
@pytest.mark.parametrize("k", [256, 256 * 3 + 64, 4096, 4096 + 256, 8192 + 512, 16384, 16384 + 256])
def test_rotated_codes_match_oracle(wq, k, group, dtype):
    """IEEE operations only, in the oracle's order: the same bits.  Rows in both layouts (up to 16384 values and beyond), last chunks that are not
    whole, zeros, and (BF16, FP32) values whose doubles are infinite."""
    k = k // group * group
    x = randn((6, k), torch.float32, 33)
    x[1], x[2, ::7] = 0, x[2, ::7] * 40
    x[3] *= 1e-7
    if dtype != torch.float16:
        x[4, 3] = 2.5e38
    x = x.to(dtype)
    with np.errstate(over="ignore", invalid="ignore"):
        q_cpu, s_cpu = oracle.quantize_blocks(x, group)
        hi_cpu, lo_cpu, rs_cpu = oracle.quantize_rows(x, group, True)
    ordinary = np.isfinite(rs_cpu)  # (the oracle leaves NaN where infinities meet)
    q, s = wq.quantize_blocks(x.cuda(), group)
    hi, lo, rs = wq.quantize(x.cuda(), group, True)
    only_hi, _, only_rs = wq.quantize(x.cuda(), group, False)
    assert ordinary.sum() == (6 if dtype == torch.float16 else 5)
    for got, expected in ((q, q_cpu), (s, s_cpu), (hi, hi_cpu), (lo, lo_cpu), (rs, rs_cpu), (only_hi, hi_cpu), (only_rs, rs_cpu)):
        assert np.array_equal(got.cpu().numpy()[ordinary], expected[ordinary])
    assert torch.equal(hi, only_hi) and torch.equal(rs, only_rs)
    # codes of rows that start on an 8-byte boundary only (what the entry points ask for)
    spare = torch.empty(6 * k + 8, dtype=torch.int8, device="cuda")[8:].view(6, k)
    assert wq._require().wq8_quantize(x.cuda().data_ptr(), spare.data_ptr(), None, torch.empty_like(rs).data_ptr(), 6, k, k, wq._DTYPES[dtype], group, 0, None,
                                      0.0, wq._stream(q.device)) == 0
    assert torch.equal(spare, hi)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("group", [16, 64, 256])
@pytest.mark.parametrize("k", [256, 512, 768 + 64, 1024 + 256, 2048, 13824])
def test_rotated_rows_in_many_and_in_few(wq, k, group, dtype):
    """Many rows go to the kernels with sixteen values a lane, a few to those with eight: the same bits, for ordinary values, zeros, tiny and huge ones,
    infinities and NaN, in chunks that are whole or not and an odd number of them."""
    k = k // group * group
    chunks = -(-k // 256)
    m = max(2049, 60 * 148 // chunks + 3)
    x = randn((m, k), torch.float32, 34)
    for i, change in enumerate((lambda v: v * 0, lambda v: v * 1e-7, lambda v: v * 50, lambda v: v * (1e38 if dtype != torch.float16 else 1e3))):
        x[i::11] = change(x[i::11])
    x = x.to(dtype)
    x.view(-1)[5::100003] = float("inf")
    x.view(-1)[7::100019] = -float("inf")
    x.view(-1)[9::100043] = float("nan")
    x = x.cuda()
    few = max(1, min(64, 9 * 148 // chunks))
    parts = x.split(few)
    q, s = wq.quantize_blocks(x, group)
    assert torch.equal(q, torch.cat([wq.quantize_blocks(part, group)[0] for part in parts]))
    assert torch.equal(s.view(torch.int32), torch.cat([wq.quantize_blocks(part, group)[1] for part in parts]).view(torch.int32))
    for hilo in (False, True):
        got = wq.quantize(x, group, hilo)
        expected = [torch.cat(t) for t in zip(*[[u for u in wq.quantize(part, group, hilo) if u is not None] for part in parts])]
        assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip([u for u in got if u is not None], expected))


@pytest.mark.parametrize("hilo", [False, True])
@pytest.mark.parametrize("act", ACTS)
@pytest.mark.parametrize("shape", [(1, 8), (7, 264), (5, 5120), (3, 13824), (2, 16384 + 512)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_quantize_rows_matches_reference_library(wq, shape, act, hilo):
    m, k = shape
    x = make_x(m, k, act, torch.bfloat16, 17).cuda()
    w = weight_of(k, act, torch.bfloat16, 18)
    w = None if w is None else w.cuda()
    hi, lo, s = wq.quantize(x, 0, hilo, act, w, 1e-6)
    hi_ref, lo_ref, s_ref = reflib.quantize(x, 0, hilo, act, w, 1e-6)
    assert torch.equal(hi, hi_ref) and torch.equal(s, s_ref)
    assert (lo is None) == (not hilo)
    if hilo:
        assert torch.equal(lo, lo_ref)


def test_quantize_rows_matches_oracle(wq):
    x = make_x(6, 3072, None, torch.bfloat16, 19)
    hi, lo, s = wq.quantize(x.cuda(), 0, True)
    hi_cpu, lo_cpu, s_cpu = oracle.quantize_rows(x, 0, True)
    assert np.array_equal(hi.cpu().numpy(), hi_cpu) and np.array_equal(lo.cpu().numpy(), lo_cpu)
    assert np.array_equal(s.cpu().numpy(), s_cpu)


def test_quantize_fp32_input(wq):
    x = randn((5, 520), torch.float32, 20).cuda()
    q, s = wq.quantize_blocks(x)
    q_ref, s_ref = reflib.quantize_blocks(x)
    assert torch.equal(q, q_ref) and torch.equal(s, s_ref)
    hi, lo, s = wq.quantize(x, 0, True)
    hi_ref, lo_ref, s_ref = reflib.quantize(x, 0, True)
    assert torch.equal(hi, hi_ref) and torch.equal(lo, lo_ref) and torch.equal(s, s_ref)


def test_strided_rows(wq):
    """Rows may be a column slice of a wider tensor (row stride larger than K)."""
    wide = randn((9, 1024), torch.bfloat16, 21).cuda()
    x = wide[:, 256:768]
    q, s = wq.quantize_blocks(x)
    q2, s2 = wq.quantize_blocks(x.contiguous())
    assert torch.equal(q, q2) and torch.equal(s, s2)


@pytest.mark.parametrize("group", [0, 16, 64, 256])
@pytest.mark.parametrize("act", ACTS)
def test_transform_rows_matches_reference_library(wq, act, group):
    m, k = 5, 2048 + 256
    x = make_x(m, k, act, torch.bfloat16, 22).cuda()
    w = weight_of(k, act, torch.bfloat16, 23)
    w = None if w is None else w.cuda()
    assert torch.equal(wq.transform_rows(x, group, act, w, 1e-6), reflib.transform_rows(x, group, act, w, 1e-6))


@pytest.mark.parametrize("group", [16, 64, 256])
def test_rotate_groups(wq, group):
    x = randn((6, 1280), torch.float16, 24).cuda()
    out = wq.rotate_groups(x, group)
    assert torch.equal(out, reflib.rotate_groups(x, group))
    expected = oracle.rotate_reference(x.float().cpu(), group)
    assert oracle.relative_error(out.cpu(), expected) < 1e-3


def test_large_row_count(wq):
    """More rows than the reference's per-call limit of 65535, in one call."""
    x = randn((70000, 256), torch.bfloat16, 25).cuda()
    q, s = wq.quantize_blocks(x)
    q_ref, s_ref = reflib.quantize_blocks(x)
    assert torch.equal(q, q_ref) and torch.equal(s, s_ref)


@pytest.mark.parametrize("act", [None, "rms_norm", "gelu"])
def test_quantizers_at_row_windows(wq, act):
    """wq8_quantize_at / wq8_quantize_blocks_at: for several values of the device counter the codes and scales equal the plain entry
    points' on the matching slice of input rows (the outputs always start at row 0)."""
    total, m, k, first, step = 120, 20, 1024 + 128, 3, 25
    x = make_x(total, k, act, torch.bfloat16, 21).cuda()
    w = weight_of(k, act, torch.bfloat16, 22)
    w = None if w is None else w.cuda()
    lib, stream = wq._require(), wq._stream(x.device)
    acts = {None: 0, "rms_norm": 1, "gelu": 3}
    for count in (0, 1, 3):
        counter = torch.tensor([count], dtype=torch.int64, device="cuda")
        rows = x[first + count * step:first + count * step + m]
        q, s = torch.empty((m, k), dtype=torch.int8, device="cuda"), torch.empty((m, -(-k // 128)), dtype=torch.float32, device="cuda")
        assert lib.wq8_quantize_blocks_at(x.data_ptr(), q.data_ptr(), s.data_ptr(), m, k, x.stride(0), 1, 0, acts[act], wq._ptr(w), 1e-6, None,
                                          counter.data_ptr(), first, step, stream) == 0
        q_plain, s_plain = wq.quantize_blocks(rows, 0, act, w, 1e-6)
        assert torch.equal(q, q_plain) and torch.equal(s, s_plain)
        hi, lo, rs = (torch.empty((m, k), dtype=torch.int8, device="cuda"), torch.empty((m, k), dtype=torch.int8, device="cuda"),
                      torch.empty(m, dtype=torch.float32, device="cuda"))
        assert lib.wq8_quantize_at(x.data_ptr(), hi.data_ptr(), lo.data_ptr(), rs.data_ptr(), m, k, x.stride(0), 1, 0, acts[act], wq._ptr(w), 1e-6,
                                   counter.data_ptr(), first, step, stream) == 0
        hi_plain, lo_plain, rs_plain = wq.quantize(rows, 0, True, act, w, 1e-6)
        assert torch.equal(hi, hi_plain) and torch.equal(lo, lo_plain) and torch.equal(rs, rs_plain)
    # no counter: row 0, whatever first and step say
    q, s = torch.empty((m, k), dtype=torch.int8, device="cuda"), torch.empty((m, -(-k // 128)), dtype=torch.float32, device="cuda")
    assert lib.wq8_quantize_blocks_at(x.data_ptr(), q.data_ptr(), s.data_ptr(), m, k, x.stride(0), 1, 0, acts[act], wq._ptr(w), 1e-6, None, None, 7, 9,
                                      stream) == 0
    q_plain, s_plain = wq.quantize_blocks(x[:m], 0, act, w, 1e-6)
    assert torch.equal(q, q_plain) and torch.equal(s, s_plain)
