"""The library's host paths on the CPU: vx_api.cpp over a made-up CUDA runtime
(tests/c/host_paths.cpp) that knows what every enqueued piece of work follows,
counts what is allocated, and fails any one call on request."""
import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    cuda = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"
    out = tmp_path_factory.mktemp("host_paths") / "host_paths"
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", f"-I{cuda}", f"-I{ROOT / 'include'}",
                    f"-I{ROOT / 'voxelg_b200' / 'csrc'}", str(ROOT / "tests/c/host_paths.cpp"),
                    "-x", "c++", str(ROOT / "voxelg_b200/csrc/vx_api.cpp"), "-o", str(out),
                    "-lpthread", "-ldl"], check=True)
    return out


# batch_memory: pick batches over host arrays return what each ray gives,
#   allocate nothing on later calls, whether results are kept or dropped, and
#   leave the world with buffers of a bounded size
# batch_beside_others: a batch under way holds up neither single picks nor
#   other threads' batches
# batch_errors: whichever CUDA call of a batch fails, it reports an error and
#   the next batch is right
# frame_sizes: host frames of every split into bands and streams return every
#   row and leave no access unordered
# frame_handles, update_handles: whichever stream, event or buffer a host frame
#   or an update of bricks could not make on first use, the next one makes it
# frame_errors: whichever CUDA call of a host frame fails, the next frames are
#   right and touch no buffer that work of the failed one may still use
@pytest.mark.parametrize("scenario", ["batch_memory", "batch_beside_others", "batch_errors",
                                      "frame_sizes", "frame_handles", "update_handles", "frame_errors"])
def test_scenario(exe, scenario):
    r = subprocess.run([str(exe), scenario], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
