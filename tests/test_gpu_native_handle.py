"""Checks of a handle through a host program linked with the library's objects
(native_handle.cu): what the C ABI alone cannot set up."""
import glob
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    import build as B  # the package's own build script
    exe = str(tmp_path_factory.mktemp("native") / "native_handle")
    objs = sorted(glob.glob(os.path.join(B.BUILD, "*.cu.o")))
    assert objs, "the library's objects are not built"
    wrap = ["-Xlinker", ",".join("--wrap=" + f for f in ("cudaFuncSetAttribute", "cudaLaunchKernelExC",
                                                         "cudaMallocHost", "cudaMalloc"))]
    subprocess.check_call([B.nvcc()] + B.NVCC_FLAGS + [os.path.join(HERE, "native_handle.cu")] + objs + wrap +
                          ["-o", exe])
    return exe


def _check(program, name):
    r = subprocess.run([program, name], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_small_handles_on_a_second_device(program):
    """The resident kernel's attributes belong to the device they were set on: a
    handle made on another one (played by the program's wrapped calls) runs too,
    with the same bits."""
    _check(program, "devices")


def test_an_export_reports_its_own_timeout(program):
    """A look-back wait of the neighbour lists that gives up (bounded, a few seconds)
    is the export's error, not the state's."""
    _check(program, "lookback")


def test_an_export_after_a_failed_allocation(program):
    """The export's two buffers are had one by one: the next call gets the missing one."""
    _check(program, "pinned")


def test_a_total_without_room_for_the_entries(program):
    """The call for the total succeeds when the entries' buffer cannot be had; the
    one that asks for the entries reports it."""
    _check(program, "count_only")


def test_launch_counts(program):
    """sphg_launches_per_step and SPHG_DBG_RESORT[2] against the launches made."""
    _check(program, "launches")
