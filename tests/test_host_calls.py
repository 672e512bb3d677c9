"""The native host side of the two whole-linear library calls: which calls it takes, and that the others go the general way with the same bits."""
from types import SimpleNamespace

import pytest
import torch

from tests.gpu_common import rand_int8, randn, rel
from wgpkernels_b200 import build as builder
from wgpkernels_b200 import int8


@pytest.fixture(scope="module")
def native():
    builder.build()
    from wgpkernels_b200.int8 import _calls
    return _calls


def test_is_bound_to_the_pytorch_it_was_built_for(native, tmp_path, monkeypatch):
    """The file says what it was compiled against; with another PyTorch or Python it is not used, and a build makes it anew."""
    assert native.BUILT_FOR == builder.built_for() and torch.__version__ in native.BUILT_FOR
    monkeypatch.setattr(int8, "built_for", lambda: "another PyTorch")
    with pytest.raises(RuntimeError, match="another PyTorch; rebuild it"):
        int8._native_calls()
    current = builder.calls_file()
    copy = tmp_path / "_calls.so"
    copy.write_bytes(current.read_bytes())
    monkeypatch.setattr(builder, "calls_file", lambda: copy)
    compiled = []
    monkeypatch.setattr(builder.subprocess, "run", lambda command, **kw: compiled.append(command) or SimpleNamespace(returncode=1, stdout="", stderr=""))
    assert builder.build_calls() == copy and not compiled
    monkeypatch.setattr(builder, "built_for", lambda: "torch of tomorrow")
    with pytest.raises(RuntimeError, match="compiler failed"):
        builder.build_calls()
    assert any('-DWQ_BUILT_FOR="torch of tomorrow"' in argument for argument in compiled[0])


def test_loads_without_the_native_side(native, monkeypatch):
    """The library is what computes: without its native callers linear() makes its calls one by one."""
    def missing():
        raise RuntimeError("the native host side is missing")

    for name in ("_lib", "_native", "_linear_address", "_few_address", "_weight_groups"):
        monkeypatch.setattr(int8, name, getattr(int8, name))
    monkeypatch.setattr(int8, "_native_calls", missing)
    with pytest.warns(RuntimeWarning, match="is missing"):
        library = int8.load_library(builder.build())
    assert int8._lib is library and int8._native is None
    monkeypatch.setattr(int8, "_plans", {("exact", 40, 8, 256, None): (1, 0, 0, 0)})
    x, w, s = torch.zeros(40, 256, dtype=torch.bfloat16), torch.zeros(8, 256, dtype=torch.int8), torch.ones(8)
    assert int8._one_call(x, w, s, None, 0, "exact", None, None, 0.0, None, None, None) is None
    assert int8._with_input_operation(x[:4], w, s, None, 0, None, None, 0.0, None, None, None) is None


def test_scratch_is_that_of_the_variant_and_library_in_use(native, monkeypatch):
    """wq8_linear is not told how large its scratch is: a size kept from another tile variant, or another library, must not be passed."""
    sizes = []
    for name, value in (("_native", SimpleNamespace(linear=lambda *a: sizes.append(a[-1]) or "done")), ("_sms", {None: 148}), ("_plans", {}), ("_scratch_sizes", {}),
                        ("_few_shapes", {"a shape": (1, 0, 0)}), ("_linear_address", 0), ("_few_address", 0), ("_weight_groups", False),
                        ("_lib", SimpleNamespace(wq8_linear_scratch=lambda m, n, k, path, variant, sms: 1000 * variant))):
        monkeypatch.setattr(int8, name, value)
    x, w, s = torch.zeros(40, 256, dtype=torch.bfloat16), torch.zeros(8, 256, dtype=torch.int8), torch.ones(8)
    for variant in (10, 20, 10):
        int8._plans["block", 40, 8, 256, None] = (variant, 0, 0, 0)
        assert int8._one_call(x, w, s, None, 0, "block", None, None, 0.0, None, None, None) == "done"
    assert sizes == [10000, 20000, 10000]
    int8.load_library(builder.build())
    assert not int8._plans and not int8._scratch_sizes and not int8._few_shapes


def test_a_build_elsewhere_makes_it_as_well(tmp_path, monkeypatch):
    made = []
    monkeypatch.setattr(builder, "build_calls", lambda *a, **kw: made.append("calls"))
    monkeypatch.setattr(builder, "_stale", lambda target, sources: False)
    assert builder.build(tmp_path / "libwgp_int8.so") == (tmp_path / "libwgp_int8.so").resolve() and made == ["calls"]


def test_takes_cuda_tensors_only(native):
    x, w, s = torch.zeros(2, 256, dtype=torch.bfloat16), torch.zeros(8, 256, dtype=torch.int8), torch.ones(8)
    tensors = (x, w, s, None, None, None, None, None)
    assert native.linear(0, *tensors, 0, 0, 0.0, 1, 1, 148, 4096) is None
    assert native.few(0, *tensors, 0, 0.0, 1, 148, 0, 0) is None
    assert native.linear(0, [x], *tensors[1:], 0, 0, 0.0, 1, 1, 148, 4096) is None  # what is no tensor


def test_wrong_arguments_are_errors(native):
    with pytest.raises(TypeError):
        native.linear(0)
    with pytest.raises(TypeError):
        native.few(0, None)
    with pytest.raises(TypeError):
        native.linear(0, *[None] * 8, "group", 0, 0.0, 1, 1, 148, 4096)


class Marked(torch.Tensor):
    pass


def test_tile_counters_lie_in_the_calls_own_scratch(monkeypatch):
    """What streams would share is no part of a few-token call: its scratch holds its counters, behind the partial sums."""
    def workspace(m, n, k, sms, sizes):
        sizes[0], sizes[1] = 1024, 64

    calls = []
    library = SimpleNamespace(wq8_few_takes=lambda *shape: 2, wq8_small_workspace=workspace)
    for name, value in (("_lib", library), ("_sms", {None: 148}), ("_few_shapes", {}), ("_native", SimpleNamespace(few=lambda *a: calls.append(a[-2:]) or "done")),
                        ("_stream", None), ("_zeroed_counters", None)):
        monkeypatch.setattr(int8, name, value)
    x, w, s = torch.zeros(2, 256, dtype=torch.bfloat16), torch.zeros(8, 256, dtype=torch.int8), torch.ones(8)
    assert int8._with_input_operation(x, w, s, None, 0, "rms_norm", None, 1e-6, None, None, None) == "done"
    assert calls == [(1024 + 64, 1024)]


@pytest.mark.parametrize("m,mode,taken", [(1, "lines", True), (4, "lines", True), (5, "lines", False), (32, "lines", False), (4, "small", True), (32, "small", True),
                                           (33, "small", False)])
def test_which_token_counts_take_the_few_token_call(m, mode, taken, monkeypatch):
    """'lines' is for one to four tokens: with more it is refused by the general way, not run as something else."""
    for name, value in (("_lib", SimpleNamespace(wq8_few_takes=lambda *shape: 1)), ("_sms", {None: 148}), ("_few_shapes", {}),
                        ("_native", SimpleNamespace(few=lambda *a: "few tokens")), ("linear_prepared", lambda *a: "general")):
        monkeypatch.setattr(int8, name, value)
    x, w, s = torch.zeros(m, 2048, dtype=torch.bfloat16), torch.zeros(8, 2048, dtype=torch.int8), torch.ones(8)
    assert int8.linear(x, w, s, mode=mode) == ("few tokens" if taken else "general")


@pytest.mark.gpu
@pytest.mark.parametrize("m", [5, 32])
def test_lines_with_more_than_four_tokens_is_an_error(wq, m):
    x, w, s = randn((m, 2048), torch.float16, 1).cuda(), rand_int8((8, 2048), 2).cuda(), torch.ones(8, device="cuda")
    for act in (None, "rms_norm"):
        with pytest.raises(RuntimeError, match="-2"):
            wq.linear(x, w, s, mode="lines", act=act, eps=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("m,mode", [(1, "lines"), (12, "small"), (40, "exact"), (40, "block")])
def test_other_forms_take_the_general_way(wq, m, mode, monkeypatch):
    n, k = 264, 2048
    x, w, s, b = randn((m, k), torch.float16, 1).cuda(), rand_int8((n, k), 2).cuda(), (torch.rand(n) * 0.01 + 0.001).cuda(), randn((n,), torch.float16, 3).cuda()
    res = randn((m, n), torch.float16, 4).cuda()
    wq.linear(x, w, s, b, mode=mode)  # (the tile variant is known from here on)
    expected, added = wq.linear(x, w, s, b, mode=mode), wq.linear(x, w, s, b, mode=mode, residual=res)
    taken = []
    native = wq._native
    monkeypatch.setattr(wq, "_native", type("Counted", (), {name: staticmethod(lambda *a, f=getattr(native, name): taken.append(f(*a)) or taken[-1]) for name in ("linear", "few")}))
    assert torch.equal(wq.linear(torch.nn.Parameter(x, requires_grad=False), w, s, b, mode=mode), expected) and taken.pop() is not None
    out = torch.empty_like(res)
    assert wq.linear(x, w, s, b, mode=mode, residual=res, out=out) is out and torch.equal(out, added) and taken.pop() is out
    general = wq.linear(x.as_subclass(Marked), w, s, b, mode=mode)
    assert taken.pop() is None and torch.equal(general.as_subclass(torch.Tensor), expected)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        elsewhere = wq.linear(x, w, s, b, mode=mode)
    side.synchronize()
    assert torch.equal(elsewhere, expected)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = wq.linear(x, w, s, b, mode=mode)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(captured, expected)


@pytest.mark.gpu
@pytest.mark.parametrize("act", [None, "rms_norm"])
@pytest.mark.parametrize("m,mode", [(1, "lines"), (12, "small"), (40, "exact"), (40, "block"), (300, "row")])
def test_the_calls_one_by_one(wq, m, mode, act, monkeypatch):
    """Without the native side: the same bits, but for one to four tokens behind rms_norm, whose sums are formed in another order."""
    n, k = 264, 2048
    x, w, s = randn((m, k), torch.float16, 1).cuda(), rand_int8((n, k), 2).cuda(), (torch.rand(n) * 0.01 + 0.001).cuda()
    res = randn((m, n), torch.float16, 4).cuda()
    call = lambda: wq.linear(x, w, s, None, mode=mode, act=act, eps=1e-6, residual=res)
    call()
    expected = call()
    monkeypatch.setattr(wq, "_native", None)
    assert rel(call(), expected) < 1e-4 if (m, act) == (1, "rms_norm") else torch.equal(call(), expected)
    assert wq.debug_status() == 0


@pytest.mark.gpu
def test_library_errors_are_raised(wq):
    x, w, s = torch.zeros(12, 2048 + 8, dtype=torch.float16, device="cuda")[:, 4:2052], torch.zeros(8, 2048, dtype=torch.int8, device="cuda"), torch.ones(8, device="cuda")
    with pytest.raises(RuntimeError):  # rows that are not 16-byte aligned
        wq.linear(x, w, s, mode="small")
