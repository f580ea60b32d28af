"""The host side of large host-device copies (psb_host.cuh), compiled against
a stand-in for the CUDA runtime (host_copies/cuda_runtime.h) whose streams run
nothing before somebody waits for them: what a call may leave to be read or
written after its return shows up every time, without a GPU."""
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent / "host_copies"
CSRC = HERE.parent.parent / "psacking_b200" / "csrc"


def _build(tmp_path_factory, *flags):
    out = tmp_path_factory.mktemp("host_copies") / "main"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{HERE}", f"-I{CSRC}", *flags, "-x", "c++",
                    str(HERE / "main.cpp"), "-o", str(out)], check=True, capture_output=True, text=True)
    return str(out)


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    return _build(tmp_path_factory)


def _run(program, *args):
    r = subprocess.run([program, *map(str, args)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (args, r.stdout, r.stderr)


# below the staged sizes, the smallest staged one, odd sizes, above a block
@pytest.mark.parametrize("size", [4, 100_000, (3 << 19) - 4, 3 << 19, (5 << 20) + 12, (64 << 20) + 4])
@pytest.mark.parametrize("memory", ["pageable", "locked"])
def test_upload_source_may_be_reused_on_return(program, size, memory):
    _run(program, "upload", size, "p" if memory == "locked" else "h")


@pytest.mark.parametrize("memory", ["pageable", "locked"])
def test_upload_without_a_free_block(program, memory):
    _run(program, "upload_no_block", "p" if memory == "locked" else "h")


@pytest.mark.parametrize("device", [0, 1])
@pytest.mark.parametrize("size", [100_000, (4 << 20) + 12, 40 << 20])
def test_download_waits_on_the_callers_device(program, size, device):
    _run(program, "download", size, device)


def test_staging_blocks_of_several_devices(program):
    _run(program, "two_devices")


@pytest.mark.parametrize("threads", [0, 2])
def test_without_threads_the_caller_does_the_work(tmp_path_factory, threads):
    few = _build(tmp_path_factory, f"-DTHREADS={threads}")
    for n in (1, 10, 11, 5000):
        _run(few, "chunks", n)
    _run(few, "upload", 5 << 20, "h")
    _run(few, "download", 5 << 20, 0)
