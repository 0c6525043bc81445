"""The order of the host code's copies, waits and launches, on stand-ins for
the CUDA runtime that run a stream's work as late as a GPU may."""
import ctypes
import struct
import threading

import numpy as np
import pytest

import host_runtime
from sph_gb300 import LearnedModel, Simulation, SphError, _lib, scenes


@pytest.fixture(scope="module")
def host_lib(tmp_path_factory):
    return host_runtime.load(tmp_path_factory.mktemp("host"))


@pytest.fixture
def host(host_lib, monkeypatch):
    monkeypatch.setattr(_lib, "_lib", host_lib)
    host_lib.host_reset()
    return host_lib


def copies_in(log):
    """(destination, bytes) of the log's host-to-device copies."""
    return [tuple(map(int, line.split()[1:])) for line in log.decode().splitlines()
            if line.startswith("h2d ")]


@pytest.mark.parametrize("first,second", [(1, 1), (20000, 300), (300, 20000), (200000, 131073)])
def test_forward_calls_of_two_threads_keep_apart(host, first, second):
    """While one call of the network is on its way, another thread's call on
    the same model neither writes its rows over the first one's nor takes
    its buffers away."""
    with LearnedModel(0, seed=1) as m:
        m.forward(np.ones((10, LearnedModel.IN), np.float32))
        host.host_log()
        threads = [threading.Thread(target=m.forward, args=(np.ones((n, LearnedModel.IN), np.float32),))
                   for n in (first, second)]
        host.host_hold()
        threads[0].start()
        assert host.host_wait_held()
        mine = copies_in(host.host_log())
        threads[1].start()
        threads[1].join(1.0)
        log = host.host_log()
        host.host_release()
        for t in threads:
            t.join()
    assert len(mine) == 1
    assert not any(line.startswith(b"free ") for line in log.splitlines()), log
    a, size = mine[0]
    assert not any(b < a + size and a < b + k for b, k in copies_in(log)), (mine, log)


def simulation(n=1000):
    sc = scenes.config2(n)
    return Simulation(sc.params.as_dict(), sc.config(), sc.n)


def test_empty_checkpoint_restores_its_counters(host, tmp_path):
    """The step count of a checkpoint without particles is written after the
    upload's clearing of the counters."""
    path = tmp_path / "empty.ckpt"
    path.write_bytes(struct.pack("<8sIiiIQI12x", b"SPHCKPT1", 1, 0, 1, 1, 77,
                                 ctypes.sizeof(_lib.FluidParticle)))
    with simulation() as sim:
        sim.load_state(path)
        assert sim.counters()["steps"] == 77


def test_rebuild_is_refused_in_a_capture(host):
    with simulation() as sim:
        _lib.check(host.sph_cuda_set_stream(sim.handle, host.host_stream(1)))
        host.host_log()
        with pytest.raises(SphError, match="(?i)captur"):
            sim.rebuild_neighbors()
        assert b"launch" not in host.host_log()


@pytest.mark.parametrize("call", ["cudaGraphInstantiate", "cudaStreamBeginCapture"])
def test_steps_go_on_without_the_multi_step_graph(host, call):
    with simulation() as sim:
        x = np.linspace(1.0, 2.0, 100, dtype=np.float32)
        sim.upload(x, x)
        sim.step(None, 4)
        host.host_log()
        host.host_fail(call.encode(), 0, 2)  # cudaErrorMemoryAllocation
        for _ in range(9):
            sim.step(None, 4)
        log = host.host_log().splitlines()
        assert sum(line.startswith(b"graph ") for line in log) == 9 * 4
        # the graph of a single step is not optional
        host.host_fail(call.encode(), 0, 2)
        sim.upload(x[:50], x[:50])
        with pytest.raises(SphError):
            sim.step(None, 4)


@pytest.mark.parametrize("interrupted", ["step", "upload"])
def test_upload_after_an_interrupted_build_clears_the_counters(host, interrupted):
    """A key producer that ran without its cell starts leaves counters that a
    later build would add its own to."""
    sc = scenes.config2(1000)
    size = 4 * (sc.size_x * sc.size_y + 1)
    x = np.linspace(1.0, 2.0, 100, dtype=np.float32)

    def cleared(sim):
        host.host_log()
        sim.upload(x, x)
        return any(line.startswith(b"memset ") and int(line.split()[2]) == size
                   for line in host.host_log().splitlines())

    with Simulation(sc.params.as_dict(), sc.config(), 200) as sim:
        assert not cleared(sim)
        host.host_fail(b"launch", 1, 701)  # the cell starts: cudaErrorLaunchOutOfResources
        with pytest.raises(SphError):
            if interrupted == "step":
                sim.step_split(None, sc.params.as_dict())
            else:
                sim.upload(x, x)
        assert cleared(sim)
        assert not cleared(sim)
