"""The serving loop's turns on the device, on the CPU: with the engine calls
replaced by stand-ins that count CTAs, the cooperative grids of all passes in
progress (Step 1 among them) always fit on the GPU together."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "mosp-cuda_b200")


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("turns") / "server_turns")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT}/include", f"-I{SRC}/include", f"-I{SRC}/csrc/host",
                    f"-I{cuda}/include", os.path.join(ROOT, "tests", "server_turns.cpp"),
                    os.path.join(SRC, "csrc", "host", "server.cpp"), "-o", exe, "-lpthread"], check=True)
    return exe


@pytest.mark.parametrize("workers,overlap", [(1, 1), (2, 1), (4, 1), (2, 0), (4, 0)])
def test_grids_of_all_passes_fit(driver, workers, overlap):
    out = subprocess.run([driver, str(workers), str(overlap)], check=True, capture_output=True, text=True,
                         timeout=120).stdout.split()
    ctas, launches = int(out[0]), int(out[1])
    assert ctas <= 148
    assert launches > 1 if workers > 1 and overlap else launches == 1
