"""The C ABI's host code on a CUDA runtime that runs on the host
(fake_device.cpp): which device a call works on, what it allocates and what a
call that runs out of device memory leaves behind."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from dugks_b200 import case as cs
from dugks_b200 import lib as dl

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "libdugks_fake.so")
    csrc = os.path.join(ROOT, "psp-vst_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-w", "-I", csrc, "-I", os.path.join(ROOT, "include"),
                    "-I", "/usr/local/cuda/include", "-o", so, os.path.join(ROOT, "tests", "fake_device.cpp"),
                    os.path.join(csrc, "dugks_abi.cpp"), os.path.join(csrc, "dugks_host.cpp"), "-Wl,-Bsymbolic", "-ldl"],
                   check=True)
    lib = dl.load(so)
    lib.path = so
    lib.fake_used.restype = C.c_size_t
    lib.fake_capacity.argtypes = [C.c_int, C.c_size_t]
    return lib


@pytest.fixture
def memory(fake):
    yield fake
    for d in (0, 1):
        fake.fake_capacity(d, 1 << 40)


def test_a_handles_state_is_read_whatever_device_is_current(memory):
    s = dl.Solver(cs.cavity_case(4, 6), device=1, lib_path=memory.path)
    memory.fake_current(0)
    g, h = s.state()
    assert np.all(g == 1.0) and not np.any(h)
    assert memory.fake_device() == 0
    s.set_state(2.0 * g, h, 1e-6)
    assert memory.fake_device() == 0 and np.all(s.state()[0] == 2.0)


def test_a_set_state_that_finds_no_memory_changes_nothing(memory):
    # 3-D, KInner 0: the first nonzero h~ needs two more arrays, one at a time
    c = cs.cube_case(3, 6)
    s = dl.Solver(c, lib_path=memory.path)
    g, h = s.state()
    used = memory.fake_used(0)
    s.step(1, c.dt)
    assert memory.fake_last_hzero() == 1
    for spare in (0, 8 * 32 * 216 + 20000):      # neither array fits, only the first does
        memory.fake_capacity(0, used + spare)
        passes = memory.fake_passes()
        with pytest.raises(dl.DugksError) as e:
            s.set_state(2.0 * g, h + 1.0, c.dt)
        assert e.value.code == 3
        g1, h1 = s.state()
        assert np.array_equal(g1, g) and np.array_equal(h1, h)
        assert memory.fake_used(0) == used and memory.fake_passes() == passes
        s.step(1, c.dt)
        assert memory.fake_last_hzero() == 1
    memory.fake_capacity(0, 1 << 40)
    with pytest.raises(dl.DugksError) as e:
        s.set_state(2.0 * g, h, 0.0)             # dt_prev 0
    assert e.value.code == 1 and np.array_equal(s.state()[0], g)
    s.set_state(2.0 * g, h + 1.0, c.dt)
    s.step(1, c.dt)
    assert memory.fake_last_hzero() == 0 and np.all(s.state()[1] == 1.0)


@pytest.mark.parametrize("n,n_dv,scale", [(120, 12, 1), (120, 12, 2), (40, 20, 1), (40, 20, 3), (4, 6, 1)])
def test_reported_chunks_give_the_handle_they_were_read_from(fake, n, n_dv, scale):
    c = cs.cavity_case(n, n_dv)

    def chunks(dv_chunks):
        s = dl.Solver(c, dv_chunks=dv_chunks, lib_path=fake.path)
        s.step(1, c.dt)
        return s.layout()["dv_chunks"], fake.fake_last_chunks(0), fake.fake_last_chunks(1)

    auto = chunks(0)
    assert auto[0] == auto[1]
    got = chunks(scale * auto[0])
    assert got[0] == got[1] == min(scale * auto[0], n_dv)
    assert got == chunks(got[0])
    if scale == 1:
        assert got == auto


def _run(fake, s, *mib):
    sizes = (C.c_size_t * len(mib))(*[m << 20 for m in mib])
    return fake.fake_run(s.h, sizes, len(mib))


def test_memory_kept_between_runs_is_bounded_and_given_back(memory):
    c = cs.cavity_case(4, 6)
    a, b = (dl.Solver(c, lib_path=memory.path) for _ in range(2))
    other = dl.Solver(c, device=1, lib_path=memory.path)
    bare = memory.fake_used(0)
    kept = lambda: (memory.fake_used(0) - bare) >> 20   # noqa: E731
    assert _run(memory, a, 500, 300) == 0 and kept() == 800
    # a small run in between, another handle's run and another device's: the
    # blocks are there for the next run
    assert _run(memory, a, 1) == 0 and _run(memory, b, 500, 300) == 0 and kept() == 801
    assert _run(memory, other, 7) == 0 and kept() == 801
    # 2 GiB a device at most, over all handles
    for m in (600, 700, 900, 3000):
        assert _run(memory, b, m) == 0 and kept() <= 2048
    # a block over the bound takes no other's place
    at = kept()
    assert _run(memory, b, 3000) == 0 and kept() == at
    # no allocation of any handle fails while memory is kept
    assert _run(memory, a, 1000, 900) == 0
    memory.fake_capacity(0, memory.fake_used(0))
    d = dl.Solver(cs.cavity_case(40, 20), lib_path=memory.path)
    assert kept() < 100
    d.close()
    memory.fake_capacity(0, bare + (500 << 20))
    assert _run(memory, a, 400) == 0 and kept() == 400
    assert _run(memory, b, 450) == 0 and kept() == 450
    assert _run(memory, b, 600) == 3
    a.step(1, c.dt)                                      # the failure leaves no error behind
    memory.fake_capacity(0, 1 << 40)
    # a call for it, and the last handle of the device
    assert _run(memory, a, 300) == 0 and kept() == 300
    assert memory.dugks_release_memory(0) == 0 and kept() == 0 and memory.dugks_release_memory(-1) == 1
    assert _run(memory, a, 300) == 0
    a.close()
    assert kept() >= 299
    b.close()
    assert memory.fake_used(0) == 0 and memory.fake_used(1) > 7 << 20
    other.close()
    assert memory.fake_used(1) == 0


def _with_nodes(c, n_dv):
    c.xis, c.weights, c.xi_max = np.linspace(-1600.0, 1600.0, n_dv), np.full(n_dv, 3200.0 / n_dv), 1600.0
    return c


@pytest.mark.parametrize("n_dv", [8, 40])
def test_the_half_steps_arrays_take_what_memory_is_left(memory, n_dv):
    # 2-D: gbar+ and hbar+ are two of eight reals a cell and DV; with a
    # quarter of them (whole rows of DVs at least) a handle still fits
    c = _with_nodes(cs.cavity_case(24, 6), n_dv)
    s = dl.Solver(c, lib_path=memory.path)
    whole = memory.fake_used(0)
    bars = 2 * 8 * 576 * n_dv * n_dv
    s.close()
    assert memory.fake_used(0) == 0
    memory.fake_capacity(0, whole - bars * 3 // 4 + 20000)
    s = dl.Solver(c, lib_path=memory.path)
    assert memory.fake_used(0) <= whole - bars * 3 // 4 + 20000
    g, h = s.state()
    s.set_state(g + np.arange(g.size).reshape(g.shape), h + 2.0, 1e-6)     # in parts of gbar+'s size
    assert np.array_equal(s.state()[0], 1.0 + np.arange(g.size).reshape(g.shape)) and np.all(s.state()[1] == 2.0)
    s.close()
    memory.fake_capacity(0, whole - bars)
    with pytest.raises(dl.DugksError) as e:
        dl.Solver(c, lib_path=memory.path)
    assert e.value.code == 3 and memory.fake_used(0) == 0


def test_large_half_step_arrays_leave_memory_free(memory):
    # 2 x 284 MB of gbar+ and hbar+: whole on a large device, cut where they are
    # more than a quarter of what is free
    c = _with_nodes(cs.cavity_case(150, 6), 40)
    s = dl.Solver(c, lib_path=memory.path)
    whole = memory.fake_used(0)
    s.close()
    bars = 2 * 8 * 22528 * 1600
    memory.fake_capacity(0, whole + bars)
    s = dl.Solver(c, lib_path=memory.path)
    assert memory.fake_used(0) <= whole - bars // 2 + 40000
    s.close()


def test_chunks_follow_the_devices_multiprocessors(fake):
    # 3,721 cells, 28 x 28 DVs: one wave of CTAs is 5 chunks on 148
    # multiprocessors (device 0) and 2 on 74 (device 1)
    c = cs.cavity_case(61, 28)
    assert [dl.Solver(c, device=d, lib_path=fake.path).layout()["dv_chunks"] for d in (0, 1)] == [5, 2]
