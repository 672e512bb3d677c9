"""The build's check of ptxas' report, and how it puts a new library in place (no GPU)."""
from wgpkernels_b200 import build as builder


def report(kernel, stored, loaded):
    return (f"ptxas info    : Compiling entry function '{kernel}' for 'sm_100a'\nptxas info    : Function properties for {kernel}\n"
            f"    {8 if stored else 0} bytes stack frame, {stored} bytes spill stores, {loaded} bytes spill loads\nptxas info    : Used 96 registers\n")


def test_spills_around_tensor_memory_loads_are_refused():
    row, block = "_ZN2wq10gemm_i8_tcI13__nv_bfloat16Li0ELi128ELb0ELb0ELi4ELb0EEEv", "_ZN2wq10gemm_i8_tcI6__halfLi2ELi256ELb1ELb0ELi4ELb0EEEv"
    eight_warps, few = "_ZN2wq10gemm_i8_tcI6__halfLi2ELi256ELb0ELb0ELi2ELb0EEEv", "_ZN2wq9stream_tcI6__halfLi16EEEv"
    quantizer = "_ZN2wq13quantize_rowsI6__halfLi16ELb1ELi3ELi4EEEv"
    fine = report(row, 0, 0) + report(block, 8, 4) + report(few, 0, 0) + report(quantizer, 48, 48)
    assert builder.spills(fine) == []
    bad = fine + report(row, 8, 4) + report(block, 16, 4) + report(eight_warps, 8, 8) + report(few, 4, 4)
    assert builder.spills(bad) == [(row, 8, 4), (block, 16, 4), (eight_warps, 8, 8), (few, 4, 4)]


def test_a_new_file_takes_the_old_ones_place(tmp_path):
    """Not its bytes: a process that has the old library mapped goes on with it."""
    target, built = tmp_path / "library.so", tmp_path / "new"
    target.write_bytes(b"old")
    built.write_bytes(b"new and longer")
    with open(target, "rb") as mapped:
        builder._install(built, target)
        assert mapped.read() == b"old" and target.read_bytes() == b"new and longer"
    assert sorted(path.name for path in tmp_path.iterdir()) == ["library.so", "new"]
