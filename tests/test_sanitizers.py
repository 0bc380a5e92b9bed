"""Host-side native code under sanitizers (no GPU): AddressSanitizer + UBSan over the plan compiler and the CPU
executor for every algorithm, ThreadSanitizer over the threads-as-ranks MPI stand-in.  The reference is built
with default flags only (CMakeLists.txt:5) and has no such checks."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "rbruck_alltoallv_b200" / "csrc"

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


def _build_and_run(tmp_path, name, sources, flags, includes, env=None):
    exe = tmp_path / name
    cmd = ["g++", "-std=c++17", "-O1", "-g", "-fno-omit-frame-pointer", *flags, *[f"-I{i}" for i in includes],
           *[str(s) for s in sources], "-o", str(exe), "-pthread"]
    b = subprocess.run(cmd, capture_output=True, text=True)
    if b.returncode != 0 and "sanitize" in (b.stderr or "") and "cannot find" in b.stderr:
        pytest.skip("sanitizer runtime not installed")
    assert b.returncode == 0, b.stderr[-2000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600, env=env)
    assert r.returncode == 0, (r.stdout[-1500:], r.stderr[-3000:])
    return r.stdout


def test_plan_compiler_and_executor_under_asan_ubsan(tmp_path):
    out = _build_and_run(tmp_path, "plan_asan",
                         [ROOT / "tests" / "native" / "plan_sanitize_main.cpp", CSRC / "plan" / "plan.cpp"],
                         ["-fsanitize=address,undefined", "-fno-sanitize-recover=undefined"], [CSRC / "include"])
    assert " 0 bad" in out


def test_mpi_stand_in_under_tsan(tmp_path):
    out = _build_and_run(tmp_path, "shim_tsan",
                         [ROOT / "tests" / "native" / "shim_tsan_main.cpp", ROOT / "baseline" / "mpi_shim" / "mpi_shim.cpp"],
                         ["-fsanitize=thread"], [ROOT / "baseline" / "mpi_shim"])
    assert "bad 0" in out


def test_device_byte_copy_stays_inside_its_block(tmp_path):
    """The warp copy of the alltoallv kernels with lanes as fibers: for every alignment and every size around the limits of
    its rounds, each load touches the source block, each store lies inside the destination, and the bytes are right."""
    out = _build_and_run(tmp_path, "warp_copy", [ROOT / "tests" / "native" / "warp_copy_main.cpp"], [], [CSRC])
    assert " 0 bad" in out


def test_static_tables_deliver_every_block(tmp_path):
    """Every schedule resolved for one, two and four processes against a stand-in for the CUDA runtime, and its items executed
    on the host: chains, flags between hops, wide items, chunk sizes given and chosen."""
    from rbruck_alltoallv_b200.parallel.plan import ALGOS
    include = Path("/usr/local/cuda/include")
    if not (include / "cuda_runtime.h").exists():
        pytest.skip("needs the CUDA headers")
    exe = tmp_path / "static_table"
    b = subprocess.run(["g++", "-std=c++17", "-O1", "-g", f"-I{include}", f"-I{CSRC / 'include'}", f"-I{CSRC}",
                        str(ROOT / "tests" / "native" / "static_table_main.cpp"), "-x", "c++", str(CSRC / "comm" / "comm.cu"),
                        str(CSRC / "plan" / "plan.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert b.returncode == 0, b.stderr[-2000:]
    r = subprocess.run([str(exe), str(len(ALGOS))], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and " 0 bad" in r.stdout, (r.stdout[-1500:], r.stderr[-1500:])
