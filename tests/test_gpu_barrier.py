"""The bounded grid barrier of the persistent list step (sph_barrier_check):
barriers among resident blocks open; a barrier that waits for more blocks
than were launched -- an arrival that never comes -- gives up after its time
limit with SPH_ERR_TIMEOUT, and the device stays usable.  A list rebuild whose
barriers give up (a time limit of 0 s): the steps return the error with the
state as it was, on every path that reports it, until the next upload."""
import copy
import time

import numpy
import pytest

import cases
from sphere_b200 import _abi, scenes
from sphere_b200.runner import SphereError, Stepper

pytestmark = pytest.mark.gpu

OK, INPUT, TIMEOUT = 0, 1, 9


def test_barriers_open_among_resident_blocks():
    lib = _abi.load_library()
    for blocks in (1, 7, 64):
        assert lib.sph_barrier_check(blocks, blocks, 200, 1.0) == OK


def test_a_barrier_missing_an_arrival_times_out_and_the_device_stays_usable():
    lib = _abi.load_library()
    t0 = time.perf_counter()
    rc = lib.sph_barrier_check(8, 9, 1, 0.25)
    dt = time.perf_counter() - t0
    assert rc == TIMEOUT
    assert 0.2 < dt < 10.0
    # the context is still good: a step runs and gives results
    s = cases.make("periodic_xy_wall_stress")[0]
    st = Stepper([s], precision="mixed")
    st.set_variant(4)
    st.upload()
    st.step(3)
    hp, _ = st.download()
    assert numpy.isfinite(hp.x).all()
    st.close()


def test_barrier_check_refuses_bad_arguments():
    lib = _abi.load_library()
    assert lib.sph_barrier_check(0, 1, 1, 1.0) == INPUT
    assert lib.sph_barrier_check(100000, 100000, 1, 1.0) == INPUT
    assert lib.sph_barrier_check(4, 4, 1, 0.0) == INPUT
    assert lib.sph_barrier_check(4, 4, 1, 100.0) == INPUT


def _state(st):
    hp, _ = st.download()
    c, h, _ = st.contacts()
    b = st.boxes()
    return [getattr(hp, k) for k in ("x", "vel", "angvel", "force", "es", "ev", "xyzsum")] + \
        [c, h, numpy.array([[q.t_current] + list(q.walls.nx[0]) + list(q.walls.mvfd[0]) for q in b])]


@pytest.mark.parametrize("warm", [0, 7])
@pytest.mark.parametrize("precision,variant,shape,radii", [
    ("fp64", 3, 0, 1.0),      # k_touch
    ("fp64", 3, 0, 1.15),     # spheres wider than a cell: k_search, k_contacts
    ("mixed", 3, 0, 1.0), ("mixed", 4, 0, 1.0), ("mixed", 4, 5, 1.0), ("mixed", 4, 9, 1.0),
    ("mixed", 4, 12, 1.0)])
def test_a_rebuild_that_gives_up_leaves_the_state(precision, variant, shape, radii, warm):
    """3,000 spheres: 12 blocks, none of which but the last to arrive passes a
    barrier with no time to wait."""
    s = scenes.lattice_pack(3000, seed=2, periodic=1, nw=1, wmode=1)
    s.radius = s.radius * radii
    if radii > 1.0:
        s.k_n[0] = s.k_t[0] = 1.0e4   # overlaps of a quarter radius: soft contacts
    s.angvel = s.angvel.astype(numpy.float32).astype(numpy.float64)   # as the list step holds them

    def fresh():
        st = Stepper([copy.deepcopy(s)], precision=precision)
        st.set_variant(variant)
        st.set_launch_shape(shape)
        st.upload()
        st.step(warm)
        return st

    st = fresh()
    before = _state(st)
    st.set_rebuild_limit(0.0)
    st.set_neighbor_lists(48)     # asks for a rebuild
    for k in (5, 1):
        with pytest.raises(SphereError) as e:
            st.step(k)
        assert e.value.status == TIMEOUT
        for u, v in zip(before, _state(st)):
            assert numpy.array_equal(u, v)
    # the pipelined path: the snapshot reports and clears the error word
    for _ in range(2):
        st.step_async(3)
        st.snapshot()
        with pytest.raises(SphereError) as e:
            st.snapshot_read()
        assert e.value.status == TIMEOUT
    # time to wait again does not bring the half-built lists back
    st.set_rebuild_limit(1.0)
    with pytest.raises(SphereError):
        st.step(1)
    assert all(numpy.array_equal(u, v) for u, v in zip(before, _state(st)))
    # an upload does
    st.upload()
    st.step(warm + 9)
    ref = fresh()
    ref.step(9)
    for u, v in zip(_state(ref), _state(st)):
        assert numpy.array_equal(u, v)
    st.close()
    ref.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_rebuild_that_gives_up_leaves_the_bonds(precision):
    s = scenes.bonded_pack(3000, nbonds=4500, seed=1, device=0)
    st = Stepper([s], precision=precision)
    st.set_variant(3)
    st.upload()
    st.step(7)
    before = st.download()
    st.set_rebuild_limit(0.0)
    st.set_neighbor_lists(48)
    with pytest.raises(SphereError) as e:
        st.step(4)
    assert e.value.status == TIMEOUT
    after = st.download()
    for name in ("pairs", "delta_n", "delta_t", "omega_n", "omega_t"):
        assert getattr(before[1], name).any()
        assert numpy.array_equal(getattr(before[1], name), getattr(after[1], name)), name
    assert numpy.array_equal(before[0].x, after[0].x) and numpy.array_equal(before[0].force, after[0].force)
    st.close()


def test_tuning_reports_a_rebuild_that_gave_up():
    """Steps that return at once are the fastest of all: the tuner does not take
    their times for a choice."""
    s = scenes.lattice_pack(3000, seed=2, periodic=1, nw=1, wmode=1)
    st = Stepper([s], precision="fp64")
    st.upload()
    st.step(3)
    x = st.download()[0].x
    st.set_rebuild_limit(0.0)
    with pytest.raises(SphereError) as e:
        st.autotune(steps=3)
    assert e.value.status == TIMEOUT
    assert numpy.array_equal(st.download()[0].x, x)
    st.set_rebuild_limit(1.0)
    st.upload()
    st.autotune(steps=3)
    st.step(3)
    assert numpy.array_equal(st.download()[0].x, x)
    st.close()
