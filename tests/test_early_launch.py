"""Order of the two halves of programmatic dependent launch in the kernels' source (no GPU): a kernel that may itself have been started early
waits for the kernels before it BEFORE it lets the next one start, so that whatever starts finds everything but its direct predecessor finished."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "wgpkernels_b200" / "csrc"


def kernels():
    """{kernel name: body} of every __global__ function."""
    found = {}
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for start in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
            begin = text.index("{", text.index(")", start.end()))
            depth, end = 1, begin + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            found[start.group(1)] = text[begin:end]
    return found


BODIES = kernels()


def launched_early():
    """The kernels that the host code launches with programmatic stream serialization, directly or through a local name."""
    names = set()
    for path in CSRC.glob("*.cu"):
        text = path.read_text()
        for match in re.finditer(r"(?:launch_after_previous|cudaLaunchKernelEx)\(\s*(?:&config,\s*)?(\w+)", text):
            name = match.group(1)
            names.add(name if name in BODIES else re.findall(rf"auto {name} = (\w+)", text[:match.start()])[-1])
    return names


def test_the_sources_are_understood():
    assert {"gemm_i8_tc", "stream_tc", "stream_planes", "split_digits", "split_planes", "regroup_weight_scales", "quantize_rows"} <= set(BODIES)
    assert {"gemm_i8_tc", "stream_tc", "stream_planes", "split_digits", "split_planes", "regroup_weight_scales"} <= launched_early()


@pytest.mark.parametrize("name", sorted(launched_early()))
def test_waits_before_it_lets_the_next_one_start(name):
    body = BODIES[name]
    assert "dependency_wait()" in body
    if "dependents_may_start()" in body:
        assert body.index("dependency_wait()") < body.index("dependents_may_start()")


@pytest.mark.parametrize("name", ["gemm_i8_tc", "regroup_weight_scales", "split_digits", "split_planes"])
def test_reads_what_the_kernel_before_it_may_have_written_with_ordinary_loads(name):
    """These start behind any kernel, a quantizer that wrote the weights and their scales included.  The read-only path is for data that nobody
    writes while the kernel runs, and its loads may be moved ahead of the wait."""
    assert not re.search(r"__ldg\(|(?<!\w)load_eight\(|ld\.global\.nc", BODIES[name])


@pytest.mark.parametrize("name", ["gemm_few_rows", "stream_few"])
def test_kernels_of_few_rows_and_tokens_read_with_ordinary_loads(name):
    assert name in launched_early() and not re.search(r"__ldg\(|(?<!\w)load_eight\(|ld\.global\.nc|__restrict__", BODIES[name])


@pytest.mark.parametrize("name", sorted(n for n, body in BODIES.items() if "dependents_may_start()" in body))
def test_lets_the_next_one_start_only_where_everything_before_it_has_finished(name):
    assert "dependency_wait()" in BODIES[name] or name not in launched_early()
