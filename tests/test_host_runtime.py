"""The engine's host code on the CPU, against a stand-in for the CUDA runtime
(fake_runtime.cpp) that records what the host asks for: launches, streams, pinned
buffers, graphs.  It has two devices, which a one-GPU machine does not."""
import ctypes as C
import glob
import os
import shutil
import subprocess

import numpy as np
import pytest

from remd_b200 import engine as E
from remd_b200 import systems as S

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    """The engine linked against the stand-in, in place of the engine library."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no CUDA headers")
    E.build_library()
    out = str(tmp_path_factory.mktemp("fake") / "libremd_fake.so")
    objects = [o for o in sorted(glob.glob(os.path.join(os.path.dirname(E.__file__), "csrc", "_build", "*.o")))]
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-o", out,
                    "-I" + os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include"),
                    os.path.join(HERE, "fake_runtime.cpp"), *objects, "-lpthread", "-ldl", "-lrt"], check=True)
    kept = E._LIB, E.LIB_PATH
    E._LIB, E.LIB_PATH = None, out
    L = E.lib()
    L.fake_launch.restype = C.c_char_p
    L.fake_count.restype = C.c_long
    yield L
    E._LIB, E.LIB_PATH = kept


@pytest.fixture(autouse=True)
def device_zero(fake):
    fake.cudaSetDevice(0)
    fake.fake_reset()


def _grid(nmol, nrep, model="tip4p", confined=0, interval=3, wall=7.0):
    e = S.small_ensemble(model, confined, nmol=nmol, ntemp=nrep, npress=1, seed=5, interval=interval, wall=wall)
    return e


def test_state_is_read_whatever_device_is_current(fake):
    """The copies of an earlier read-back worked whatever device was current; a kernel
    launch does only with the stream's own."""
    eng = E.REMDGPU([_grid(64, 2)], device=0)
    other = E.REMDGPU([_grid(64, 1)], device=1)   # leaves device 1 current
    eng.ConvertVariablesToHost(1)
    now = C.c_int(-1)
    fake.cudaGetDevice(C.byref(now))
    assert now.value == 1   # the caller's device is left as it was
    fake.cudaSetDevice(0)   # as on a host thread that never chose a device
    other.ConvertVariablesToHost(0)
    fake.cudaGetDevice(C.byref(now))
    assert now.value == 0
    eng.close(), other.close()


def test_read_back_buffer_is_made_once(fake):
    """One pinned buffer for the handle's largest replica, also where replicas are read
    from the smallest to the largest."""
    eng = E.REMDGPU([_grid(n, 1) for n in (64, 100, 200)])
    fake.fake_reset()
    for k in range(3):
        eng.ConvertVariablesToHost(k)
    assert fake.fake_count(b"host_allocs") == 1
    eng.close()


def _launches(fake):
    """(kernel, grid, block, programmatic, stream) of every launch since the last reset."""
    g, b, p, s = C.c_int(), C.c_int(), C.c_int(), C.c_int()
    out = []
    for k in range(fake.fake_count(b"launches")):
        name = fake.fake_launch(k, C.byref(g), C.byref(b), C.byref(p), C.byref(s)).decode()
        out.append((name, g.value, b.value, p.value, s.value))
    return out


def _interval(fake, eng):
    """The launches of one more interval."""
    fake.fake_reset()
    eng.ExecuteSteps(eng.T, eng.P)
    return _launches(fake)


def _steps(launches):
    return [x for x in launches if any(k in x[0] for k in ("k_integrate", "k_replica_head", "k_force"))]


@pytest.mark.parametrize("nmol,nrep,expected", [(128, 16, 1), (512, 8, 1), (512, 16, 0), (512, 64, 0), (900, 64, 0)])
def test_programmatic_launch_follows_the_work_of_all_chains(fake, nmol, nrep, expected):
    """Chains run side by side: what one chain launches programmatically must depend on
    the work of all of them, not on how many chains share it."""
    eng = E.REMDGPU([_grid(nmol, nrep)])
    steps = _steps(_interval(fake, eng))
    assert len(steps) >= 3 * 4 and all(x[3] == expected for x in steps)
    eng.close()


@pytest.mark.parametrize("nmol,nrep,extra", [(128, 16, 32), (729, 96, 0)])
def test_chain_warp_only_where_all_chains_leave_room(fake, nmol, nrep, extra):
    """The integrate kernel's extra warp: 2208 tiles of 64 threads are more than the GPU
    holds at once, however they are split over chains."""
    eng = E.REMDGPU([_grid(nmol, nrep)])
    assert all(x[2] == 32 + extra for x in _interval(fake, eng) if "k_integrate" in x[0])
    eng.close()


def _chains(launches):
    return len({x[4] for x in _steps(launches)})


def test_first_interval_is_cheap_to_set_up(fake):
    """Streams are made with the handle, not inside its first timed call, and the first
    interval's graph holds four chains however large the batch is."""
    for n, nrep in ((128, 16), (512, 64)):
        eng = E.REMDGPU([_grid(n, nrep)])
        first = _interval(fake, eng)
        assert fake.fake_count(b"streams_made") == 0
        assert fake.fake_count(b"nodes") == 4 * 4 * 3 + 2 == len(first)   # chains x kernels x steps, start and end
        assert _chains(first) == 4 and eng.launches_per_interval() == len(first)
        eng.close()


@pytest.mark.parametrize("nmol,nrep,later", [(512, 64, 8), (128, 16, 4), (512, 4, 4), (64, 1, 1)])
def test_eight_chains_come_once_they_pay(fake, nmol, nrep, later):
    """A handle that keeps running goes over to a second graph, once, where eight chains
    are faster; every replica is in exactly one chain of it."""
    eng = E.REMDGPU([_grid(nmol, nrep)])
    for _ in range(32):
        assert _chains(_interval(fake, eng)) == min(4, nrep)
    second = _interval(fake, eng)
    assert _chains(second) == later and eng.launches_per_interval() == len(second)
    for kernel, per in (("k_integrate", nrep * -(-nmol // 32)), ("k_replica_head", nrep), ("k_force_pairs", nrep * -(-nmol // 16))):
        assert sum(x[1] for x in second if kernel in x[0]) == 3 * per
    fake.fake_reset()
    eng.ExecuteSteps(eng.T, eng.P)
    assert fake.fake_count(b"instantiated") == 0
    eng.set_tuning(64, 1.0)   # a new layout keeps the chains
    assert _chains(_interval(fake, eng)) == later
    eng.close()


def test_no_room_for_the_second_graph(fake):
    """Where the second graph cannot be made the handle goes on with the first one, and
    does not try again every interval."""
    eng = E.REMDGPU([_grid(512, 64)])
    for _ in range(32):
        _interval(fake, eng)
    fake.fake_fail_instantiations(1)
    assert _chains(_interval(fake, eng)) == 4 and fake.fake_count(b"instantiated") == 1
    assert _chains(_interval(fake, eng)) == 4 and fake.fake_count(b"instantiated") == 0
    fake.fake_fail_instantiations(0)
    eng.close()


def test_serving_loop_updates_its_graph_in_place(fake):
    """A batch that grows and shrinks keeps one graph topology, so the executable graph
    is updated and not made anew, also after many rounds."""
    srv = E.Server(budget_bytes=1 << 33)
    e = _grid(200, 64)
    srv.submit(e, 40)
    for _ in range(36):
        srv.step()
    fake.fake_reset()
    srv.submit(_grid(400, 64), 20)
    srv.step()
    assert fake.fake_count(b"instantiated") == 0 and fake.fake_count(b"updated") == 1
    assert _chains(_launches(fake)) == 4
    srv.close()


@pytest.mark.parametrize("model", ["tip3p", "tip5p"])
@pytest.mark.parametrize("nmol,nrep", [(2, 1), (64, 16), (100, 64), (128, 16), (129, 4), (900, 3)])
def test_job_bytes_cover_what_the_batch_allocates(fake, model, nmol, nrep):
    """The serving loop admits jobs by these bytes: they are no less than the device
    memory that the job's batch takes, and not far above it."""
    e = _grid(nmol, nrep, model)
    said = E.Server.job_bytes(e)
    srv = E.Server(budget_bytes=said)   # and exactly that budget admits it
    srv.submit(e, 2)
    fake.fake_reset()
    srv.step()
    used = fake.fake_count(b"device_bytes")
    assert used <= said <= 1.25 * used + 20000
    srv.close()
