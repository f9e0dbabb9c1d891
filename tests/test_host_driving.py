"""Host code that drives the device, run against a CUDA runtime on the host.

tests/fake_cuda holds the runtime: work queued on a stream runs only when
something waits for it, so a missing wait, or a resource handed on while work
that uses it is still queued, shows on the CPU.
"""
import os
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
FAKE = ROOT / "tests" / "fake_cuda"
CSRC = ROOT / "gnss-1_b200" / "csrc"
CUDA_INC = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"

pytestmark = pytest.mark.skipif(not (CUDA_INC / "cuda_runtime.h").exists() or shutil.which("g++") is None,
                                reason="needs g++ and the CUDA headers")


def _compile(out: Path, *sources: Path, flags=()) -> Path:
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", *flags, f"-I{CUDA_INC}", f"-I{ROOT / 'include'}",
                    f"-I{CSRC}", f"-I{FAKE}", "-o", str(out), *map(str, sources), str(FAKE / "fake_cuda.cpp")],
                   check=True)
    return out


def _run(exe: Path, *args: str):
    return subprocess.run([str(exe), *args], capture_output=True, text=True, timeout=60)


def test_table_upload_has_arrived_on_return(tmp_path):
    r = _run(_compile(tmp_path / "upload", FAKE / "upload.cpp"))
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.fixture(scope="module")
def server(tmp_path_factory):
    return _compile(tmp_path_factory.mktemp("server") / "server", FAKE / "server.cpp", FAKE / "fake_ctx.cpp",
                    CSRC / "batch.cpp")


@pytest.mark.parametrize("scenario", ["failed_request", "idle_contexts", "device_of_reuse"])
def test_server(server, scenario):
    r = _run(server, scenario)
    assert r.returncode == 0, r.stdout + r.stderr
