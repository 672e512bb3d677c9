"""Ahead-of-time build of libwgp_int8.so for B200 (sm_100a), written next to the package's `int8` module:

    python -m wgpkernels_b200.build [--output PATH] [--verbose] [--jobs N] [--force]

A second, tiny library, libwgp_int8_probe.so, is built beside it: the tensor-pipe issue-rate probe that only the benchmark loads.  And the native
host side of the Python module, _calls.so, with the C++ compiler against the PyTorch at hand.

One architecture only: the GEMM uses tcgen05 / tensor-memory instructions that exist on sm_100a alone, so there is no PTX fallback.
The CUDA runtime is linked statically and only the C ABI is exported, so the library depends on the driver alone (the same properties
as the reference's build, wgpkernels/build.py:55-65 of WGPKernels).
"""
import argparse
import os
import re
import shutil
import subprocess
import sys
import sysconfig
import tempfile
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PACKAGE = Path(__file__).resolve().parent
SOURCES = ("api.cu", "quantize.cu", "stream.cu", "stream_few.cu", "stream_tc.cu", "gemm_rows.cu", "gemm_tc.cu")
PROBE_SOURCES = ("probe.cu",)
HEADERS = ("common.cuh", "tc_ptx.cuh")
ARCH_FLAGS = ("-gencode", "arch=compute_100a,code=sm_100a")


# Kernels whose loads from tensor memory are in flight while other work goes on: a register that such a load is still to fill must not be spilled
# (the copy would be taken before the load has delivered, and columns come out wrong now and then).  So these kernels do not spill at
# all, but for one value of 'block' on 256 channels with sixteen drain warps (gemm_i8_tc<T, 2, 256, *, 0, 4, 0>): it belongs to the write-out,
# behind the last such load -- the same kernels without their write-out spill nothing, and with half the registers for those loads as much.
NO_SPILLS = re.compile(r"gemm_i8_tc|gemm_few_rows|stream_tc|split_digits")
SPILLS_ALLOWED = {r"gemm_i8_tcI(13__nv_bfloat16|6__half)Li2ELi256ELb[01]ELb0ELi4ELb0EE": (8, 4)}  # mangled name: bytes stored, loaded


def spills(report):
    """[(kernel, bytes stored, bytes loaded)] of the kernels in ptxas' report that spill where they must not."""
    found = re.findall(r"Function properties for (\S+)\s+\d+ bytes stack frame, (\d+) bytes spill stores, (\d+) bytes spill loads", report)
    wrong = []
    for kernel, stored, loaded in found:
        most = next((limit for pattern, limit in SPILLS_ALLOWED.items() if re.search(pattern, kernel)), (0, 0))
        if NO_SPILLS.search(kernel) and (int(stored) > most[0] or int(loaded) > most[1]):
            wrong.append((kernel, int(stored), int(loaded)))
    return wrong


def library_file():
    return PACKAGE / "int8" / "libwgp_int8.so"


def probe_library_file():
    return PACKAGE / "int8" / "libwgp_int8_probe.so"


def calls_file():
    return PACKAGE / "int8" / "_calls.so"


def built_for():
    """The PyTorch and the Python at hand, as the native host side names those it was compiled against: it reads tensors through PyTorch's inline
    functions, so with others it may import and read wrong offsets."""
    import torch
    return f"torch {torch.__version__} {torch.version.git_version}, {sys.implementation.cache_tag}, C++11 ABI {int(torch._C._GLIBCXX_USE_CXX11_ABI)}"


def build_calls(nvcc="nvcc", verbose=False, force=False):
    """Compiles the native host side of the Python module (a CPython extension) against the PyTorch that imports it."""
    import torch
    source, target, root = PACKAGE / "csrc" / "host_calls.cpp", calls_file(), Path(torch.__file__).resolve().parent
    identity = built_for()
    if not force and not _stale(target, [source]) and identity.encode() in target.read_bytes():
        return target
    toolkit = Path(shutil.which(nvcc) or "/usr/local/cuda/bin/nvcc").resolve().parents[1]
    includes = [root / "include", root / "include" / "torch" / "csrc" / "api" / "include", sysconfig.get_paths()["include"], toolkit / "include"]
    with tempfile.TemporaryDirectory(prefix="wgpkernels-b200-") as work:
        built = Path(work) / target.name
        done = subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
                               f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DWQ_BUILT_FOR="{identity}"', *[f"-I{path}" for path in includes], str(source), f"-L{root / 'lib'}",
                               "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", "-o", str(built)], capture_output=True, text=True)
        if verbose or done.returncode:
            print(done.stdout + done.stderr)
        if done.returncode:
            raise RuntimeError(f"the C++ compiler failed on {source.name}")
        _install(built, target)
    return target


def _install(built, target):
    """Puts a new file in the old one's place: a process that has the old one mapped keeps it whole."""
    beside = target.with_name(f"{target.stem}.{os.getpid()}.so")
    shutil.copyfile(built, beside)
    beside.chmod(0o755)
    os.replace(beside, target)


def _stale(target, sources):
    if not target.exists():
        return True
    newest = max(p.stat().st_mtime for p in sources)
    return target.stat().st_mtime < newest


def build(output=None, nvcc="nvcc", verbose=False, jobs=None, force=False, sources=SOURCES):
    """Compiles `sources` into the shared library `output` (default: the product library; the probe library is built with it)."""
    if sources is SOURCES:
        build_calls(nvcc, verbose, force)  # (whichever library the module is to load, these lie beside the module)
        if output is None:
            build(probe_library_file(), nvcc, verbose, jobs, force, PROBE_SOURCES)
    target = Path(output or library_file()).resolve()
    csrc = PACKAGE / "csrc"
    inputs = [csrc / name for name in sources] + [csrc / name for name in HEADERS]
    if not force and not _stale(target, inputs):
        return target
    target.parent.mkdir(parents=True, exist_ok=True)
    common = [nvcc, "-O3", "-std=c++17", "-lineinfo", *ARCH_FLAGS, "-Xcompiler", "-fPIC,-fvisibility=hidden", "--cudart", "static", "-Xptxas", "-v"]
    with tempfile.TemporaryDirectory(prefix="wgpkernels-b200-") as work:
        def compile_one(name):
            obj = Path(work) / (name + ".o")
            done = subprocess.run([*common, "-c", str(csrc / name), "-o", str(obj)], capture_output=True, text=True)
            if verbose or done.returncode:
                print(done.stdout + done.stderr)
            if done.returncode:
                raise RuntimeError(f"nvcc failed on {name}")
            wrong = spills(done.stdout + done.stderr)
            if wrong:
                raise RuntimeError(f"{name}: registers that loads from tensor memory may still have to fill are spilled: {wrong}")
            return obj
        with ThreadPoolExecutor(max_workers=jobs or min(len(sources), os.cpu_count() or 1)) as pool:
            objects = list(pool.map(compile_one, sources))
        built = Path(work) / target.name
        subprocess.run([nvcc, "-shared", *ARCH_FLAGS, "--cudart", "static", "-Xcompiler", "-fPIC,-fvisibility=hidden",
                        *map(str, objects), "-o", str(built)], check=True)
        _install(built, target)
    return target


def main():
    parser = argparse.ArgumentParser(description=__doc__)
    parser.add_argument("--output", type=Path, default=None)
    parser.add_argument("--nvcc", default="nvcc")
    parser.add_argument("--verbose", action="store_true", help="print register and shared memory usage (-Xptxas -v)")
    parser.add_argument("--jobs", type=int, default=None)
    parser.add_argument("--force", action="store_true")
    args = parser.parse_args()
    print(f"Built {build(args.output, args.nvcc, args.verbose, args.jobs, args.force)}")


if __name__ == "__main__":
    main()
