"""Host code of the native library against fakes of the CUDA runtime, and what the
compiler says of its kernels, without a GPU.

Each program of tests/native is compiled with nvcc against the library's headers and
linked to the shared runtime, some of whose functions its .cpp file replaces.
"""

import glob
import os
import re
import shutil
import subprocess

import pytest

from conftest import PKG_DIR, REPO

HERE = os.path.dirname(os.path.abspath(__file__))


def _nvcc():
    return shutil.which("nvcc") or (os.path.exists("/usr/local/cuda/bin/nvcc") and "/usr/local/cuda/bin/nvcc") or None


def _flags(nvcc):
    return [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-diag-suppress", "177,550,1886",
            "-I", os.path.join(REPO, "include"), "-I", os.path.join(PKG_DIR, "csrc")]


def run_native(tmp_path, name):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc is not installed")
    lib = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "lib64")
    exe = str(tmp_path / name)
    subprocess.run([*_flags(nvcc), "-cudart", "shared", "-Xlinker", "-rpath", "-Xlinker", lib, "-o", exe,
                    *sorted(glob.glob(os.path.join(HERE, "native", name + "*.c*"))), "-lpthread"], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, (out.returncode, out.stdout, out.stderr)
    return out.stdout.split()


def test_shared_memory_limit_never_falls(tmp_path):
    """Two threads that opt one kernel in for two grids leave it with room for both."""
    e0, e1, limit, larger = map(int, run_native(tmp_path, "opt_in_threads"))
    assert (e0, e1) == (0, 0)
    assert limit >= larger


def test_sgs_block_kernels_do_not_spill(tmp_path):
    """The values that the block Smagorinsky kernels carry from layer to layer fit their
    registers in double precision (three and four points a thread)."""
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("nvcc is not installed")
    out = subprocess.run([*_flags(nvcc), "-O3", "-lineinfo", "-Xptxas", "-v", "-c", "-o", str(tmp_path / "k.o"),
                          os.path.join(HERE, "native", "sgs_block_registers.cu")], check=True, capture_output=True, text=True)
    spills = re.findall(r"k_sgs_x\w*\n\s*\d+ bytes stack frame, (\d+) bytes spill stores", out.stderr)
    assert spills == ["0"] * 3, out.stderr


def test_row_kernel_radices(tmp_path):
    """The radices of the in-place x kernels follow from the lanes they use: a second radix
    that leaves lanes of a warp idle has no alternative of 16 that the rule allows (it is not
    for the Smagorinsky model in double precision), and the larger radix is within a third of
    the smallest there is.  The blocks per SM ask for no
    more registers than there are."""
    codelets = (2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16, 18, 24, 32)
    shapes = [line.split(",") for line in run_native(tmp_path, "row_shapes")]
    assert len(shapes) > 120
    for kind, *numbers in shapes:
        points, fp32, a, b, rows, threads, blocks = map(int, numbers)
        multiple = 2 if kind == "sgs" else 3 if points % 3 == 0 else 1
        pairs = [(points // q, q) for q in codelets
                 if points % q == 0 and points // q in codelets and points // q % multiple == 0]
        smallest = min(map(max, pairs))
        assert (a, b) in pairs and 3 * max(a, b) <= 4 * smallest, (kind, points, fp32, a, b)
        if 32 % b and (kind == "adv" or fp32):
            assert all(q != 16 or 3 * max(p, q) > 4 * smallest for p, q in pairs), (kind, points, fp32, a, b)
        # as many registers as radix-a or radix-b values take (2 or 4 each) have to remain
        assert 65536 // (threads * blocks) >= max(a, b) * (2 if fp32 else 4), (kind, points, fp32, threads, blocks)


def test_host_copy_without_memory_for_threads(tmp_path):
    """A staged copy that cannot start all its threads does their parts itself."""
    assert run_native(tmp_path, "hostcopy_no_memory") == ["0"]


def test_autotuner_launches(tmp_path):
    """A candidate costs at most 16 launches, and a second round only where the first was
    short and for about as long as that round has to last."""
    rows = [tuple(map(int, line.split(","))) for line in run_native(tmp_path, "tune_launches")]
    for us, again in rows:
        assert 1 + 3 + again <= 16, (us, again)
        assert again == 0 if 3 * us >= 100 else 3 <= again and again * us <= 200, (us, again)
