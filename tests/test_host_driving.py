"""Host code that drives the device, run against a CUDA runtime on the host.

tests/fake_cuda holds the runtime: work queued on a stream runs only when
something waits for it, so a missing wait, or a resource handed on while work
that uses it is still queued, shows on the CPU.
"""
import os
import shutil
import subprocess
from pathlib import Path

import numpy as np
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


@pytest.mark.parametrize("scenario", ["failed_request", "idle_contexts", "device_of_reuse", "large_state"])
def test_server(server, scenario):
    r = _run(server, scenario)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("nx,ny,nz,alias", [(96, 96, 96, 0.75), (64, 128, 48, 15 / 32), (48, 48, 48, 1.0)])
def test_sphere_tables_do_not_depend_on_fma(tmp_path, nx, ny, nz, alias):
    """Bounds compiled with contraction to fused multiply-adds allowed equal those of numpy, which rounds every
    operation, in boxes that put modes like (2 2 1) k exactly on the sphere but for rounding."""
    fma = ["-mfma"] if " fma " in Path("/proc/cpuinfo").read_text() else []
    exe = _compile(tmp_path / "sphere", FAKE / "sphere.cpp", flags=["-O3", "-ffp-contract=fast", *fma])
    for scale in (1.0, 0.31, 0.36, 0.42, 0.44):
        l = 2 * np.pi * scale
        r = _run(exe, *(repr(v) for v in (nx, ny, nz, l, l, l, alias)))
        assert r.returncode == 0, r.stderr
        bounds, tiles, counts = (np.array(line.split(), dtype=int) for line in r.stdout.splitlines())
        dk, kmax = 2 * np.pi / l, alias * (nx * np.pi / l)
        kx = dk * np.arange(nx // 2 + 1)
        ky = dk * np.where(np.arange(ny) < ny // 2, np.arange(ny), np.arange(ny) - ny)
        kz = dk * np.array([*range(nz // 2), -nz // 2])
        inside = ~((kx * kx + (ky * ky)[:, None, None]) + (kz * kz)[:, None] > kmax * kmax)   # [ky][kz][kx]
        want = inside.sum(axis=2) - 1                                     # the kept |kx| are 0 .. bound
        y = np.arange(ny // 2 + 1) * dk
        want_y = (~((y * y) + (kz * kz)[:, None] > kmax * kmax)).sum(axis=1) - 1
        assert np.array_equal(bounds, np.concatenate([want.ravel(), want_y]))
        rows = np.where(2 * want >= nx, nx, 2 * want + 1)   # modes +-kx of a column
        first = rows[:, ::8]
        assert list(counts) == [rows[want >= 0].sum(), (want >= 0).sum(), 8 * (first > 0).sum(),
                                8 * first[first > 0].sum()]
        assert np.array_equal(tiles, [i << 8 | k for i in range(ny) for k in range(nz // 2 + 1) if want[i, k] >= 0])
