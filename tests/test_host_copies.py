"""Copies between device state and ordinary host buffers (csrc/hostcopy.cu): what is set is what
is read back, around the sizes where the copy changes its form (the driver's staging alone below
1 MB or into mapped pages, then behind threads that map the pages in parts of 512 KB), from several
threads at once, and with the particles equal to those of the pinned-buffer path."""
import os
import subprocess
import threading

import numpy as np
import pytest

from ariel_b200 import _abi as A
from ariel_b200.flipsim import Batch

from helpers import dambreak, params


def _handle(n):
    d = A.scene_dambreak(n)
    d.n_liquid = 0
    b = Batch([d], params())
    b.init()
    return b


def _round_trip(n, seed):
    rng = np.random.default_rng(seed)
    b = _handle(n)
    d = rng.standard_normal((n, n, n)).astype(np.float32)
    p = rng.standard_normal((n, n, n))
    a = rng.integers(0, 3, (n, n, n)).astype(np.int32)
    b.set_grid(A.GRID_D, d)
    b.set_grid(A.GRID_P64, p)
    b.set_grid(A.GRID_A, a)
    for _ in range(2):
        np.testing.assert_array_equal(b.get_grid(A.GRID_D), d)
        np.testing.assert_array_equal(b.get_grid(A.GRID_P64), p)
        np.testing.assert_array_equal(b.get_grid(A.GRID_A), a)
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 36, 37, 50, 51, 64, 81, 128])
def test_grids_round_trip(n):
    _round_trip(n, n)


@pytest.mark.gpu
def test_handles_copy_from_several_threads():
    errors = []

    def work(i):
        try:
            for k in range(3):
                _round_trip(60 + 7 * i, 10 * i + k)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    t = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert not errors, errors


@pytest.mark.gpu
@pytest.mark.parametrize("n", [8, 20, 48])
def test_particles_equal_the_pinned_path(n):
    b = Batch([dambreak(n), dambreak(n + 3, seed=4)], params(precision=A.PREC_MIXED, stop=A.STOP_REL))
    b.init()
    b.step(3)
    for s in range(2):
        m = b.count(s)
        pos, vel = np.empty((m, 3), np.float32), np.empty((m, 3), np.float32)
        b.download_state(pos, vel, s)
        q = b.get_particles(s)
        np.testing.assert_array_equal(q["pos"], pos)
        np.testing.assert_array_equal(q["vel"], vel)
        assert (q["mass"] == 1).all() and (q["type"] == A.FLUID).all()
        assert np.isfinite(q["density"]).all()
    b.close()


def _run_cpp(tmp_path, name):
    from ariel_b200 import build as B
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    libdir = os.path.join(root, "ariel_b200", "_lib")
    exe = str(tmp_path / name)
    subprocess.run([B.host_compiler(), "-std=c++17", "-O1", "-I", os.path.join(root, "include"),
                    os.path.join(root, "tests", "cpp", name + ".cpp"), "-L", libdir, "-lariel_b200",
                    "-Wl,-rpath," + libdir, "-rdynamic", "-ldl", "-pthread", "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr)


@pytest.mark.gpu
def test_host_threads_of_a_copy(tmp_path):
    """tests/cpp/host_copies.cpp: as many threads as the caller may use CPUs, at most."""
    _run_cpp(tmp_path, "host_copies")


@pytest.mark.gpu
def test_copies_without_host_memory(tmp_path):
    """tests/cpp/host_copy_memory.cpp: a failed allocation in a copy is a status, or no matter."""
    _run_cpp(tmp_path, "host_copy_memory")
