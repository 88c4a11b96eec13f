"""One context per host thread: two threads solving at different orders at the
same time.  A kernel's shared-memory limit belongs to the function, not to the
context, so a limit lowered for one thread's launch would fail the other's.
Every call must succeed and repeat its first result bit by bit (the solves are
deterministic; the mixed form's autotuned splits are fixed by a context's first
solves)."""
import os
import subprocess
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parent / "cpp" / "threads.cpp"


def cuda_home():
    for p in (os.environ.get("CUDA_HOME"), "/usr/local/cuda"):
        if p and (Path(p) / "include" / "cuda_runtime.h").exists():
            return Path(p)
    pytest.skip("no CUDA headers")


@pytest.fixture(scope="module")
def threads_bin(lib_path, tmp_path_factory):
    out, cuda = tmp_path_factory.mktemp("cpp") / "threads", cuda_home()
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", str(lib_path.parent.parent / "include"), "-I",
                    str(cuda / "include"), str(SRC), "-L", str(lib_path.parent), "-llfmm", "-L", str(cuda / "lib64"),
                    "-lcudart", "-ldl", "-pthread", f"-Wl,-rpath,{lib_path.parent}", "-o", str(out)], check=True)
    return out


def test_threads_compiles_and_links(threads_bin):
    assert threads_bin.exists()


# orders that share kernel instances and differ in shared memory: the factored
# translations (13-16, 17-18), the evaluation kernels (all orders), the 2D M2L
# (17-24); a plan's graph beside solves of another order
@pytest.mark.gpu
@pytest.mark.parametrize("dim,form,N0,N1,depth,max_leaf", [
    (3, 0, 13, 16, 4, 0), (3, 0, 17, 18, 4, 0), (3, 0, 8, 18, 6, 24), (3, 1, 13, 16, 6, 24), (3, 1, 9, 12, 6, 24),
    (3, 2, 16, 13, 6, 24), (2, 0, 17, 24, 5, 0)])
def test_threads_at_different_orders(threads_bin, dim, form, N0, N1, depth, max_leaf):
    r = subprocess.run([str(threads_bin), *map(str, (dim, form, N0, N1, depth, max_leaf, 200))], capture_output=True,
                       text=True, timeout=100)
    assert r.returncode == 0, r.stdout + r.stderr
