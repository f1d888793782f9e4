"""Calls that find no device memory: they report it or do without, and leave
nothing behind that a later call would take for an error of its own.  What a
handle allocates that it does not need."""
import numpy
import pytest

import torch

from sphere_b200 import scenes
from sphere_b200.runner import SphereError, Stepper

pytestmark = pytest.mark.gpu

NOMEM = 6


def test_a_failed_allocation_is_reported_once():
    """Adjoint checkpoints of 4e5 steps, some 700 GB, do not fit; the calls
    after it, which end by asking for launch errors, run."""
    s = scenes.loose_pack(1000, seed=0)
    st = Stepper([s], precision="fp64", length="fp64")
    st.upload()
    st.step(3)
    with pytest.raises(SphereError) as e:
        st.adjoint_forward(400000, ckpt=1)
    assert e.value.status == NOMEM
    assert st.relax(1, alpha=0.1, z_top=float(s.L[2])) >= 0.0
    assert st.count_contacts() >= 0
    st.close()


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _fill():
    """All but a few MB of the device's free memory."""
    return torch.empty((_free() // (2 << 20) - 2) * (2 << 20), dtype=torch.uint8, device="cuda")


def _give_back():
    torch.cuda.empty_cache()


def _lattice(n, **kw):
    return scenes.lattice_pack(n, seed=1, periodic=1, nw=1, wmode=1, **kw)


def test_split_step_buffers_by_need():
    """The default variant's buffers, taken by the first upload with lists on:
    84 bytes a sphere, and 260 more for spheres wider than a cell."""
    n = 400000
    s = _lattice(n)
    st = Stepper([s], precision="fp64")
    st.set_neighbor_lists(0)
    st.upload()
    st.set_neighbor_lists(48)
    free = [_free()]
    for r in (1.0, 1.15):
        st.sims[0].radius = s.radius * r
        st.upload()
        assert st.tuning()[0] == 3
        free.append(_free())
    assert free[0] - free[1] <= 84 * n + (4 << 20)
    assert 256 * n <= free[1] - free[2] <= 260 * n + (4 << 20)   # (the counts may fit a chunk)
    st.close()


def test_default_upload_without_room_for_the_split_step():
    s = _lattice(150000)
    ref = Stepper([s], precision="fp64")
    ref.set_variant(1)
    st = Stepper([s], precision="fp64")
    st.set_neighbor_lists(0)      # no split step, so none of its buffers yet
    for q in (ref, st):
        q.upload()
    ref.step(3)
    st.set_neighbor_lists(48)
    pad = _fill()
    before = _free()
    st.upload()
    assert st.tuning()[0] == 1 and _free() == before
    assert st.count_contacts() == 0
    st.step(3)
    del pad
    _give_back()
    out = [st.download()[0]]
    st.upload()
    assert st.tuning()[0] == 3
    st.step(3)
    out.append(st.download()[0])
    want = ref.download()[0]
    for o in out:
        for name in ("x", "vel", "force"):
            assert numpy.array_equal(getattr(o, name), getattr(want, name)), name
    st.close()
    ref.close()


def test_small_handles_take_little_memory():
    """100 spheres: 0.2 MB of arrays, allocated in steps of up to 2 MB."""
    s = _lattice(100)
    free = _free()
    many = []
    for _ in range(40):
        many.append(Stepper([s], precision="fp64"))
        many[-1].upload()
    assert free - _free() <= 40 * (2 << 20) + (4 << 20)
    for st in many:
        st.step(1)
        st.close()


def test_scratch_of_an_analysis_call_gives_way():
    """The image buffer kept from a large image (27 MB) is given back when
    the tuner's state snapshot, 15 MB, finds no other room."""
    s = _lattice(10000)
    st = Stepper([s], precision="fp64")
    st.upload()
    img = st.render(width=3000, height=3000)
    pad = _fill()
    st.autotune(steps=1)
    del pad
    _give_back()
    assert numpy.array_equal(st.render(width=3000, height=3000), img)
    st.close()


def test_bonds_come_back_from_a_full_device():
    s = scenes.bonded_pack(200000, nbonds=300000, seed=0, device=0)
    out = []
    for full in (False, True):
        st = Stepper([s], precision="fp64")
        st.upload()
        st.step(3)
        pad = _fill() if full else None
        out.append(st.download()[1])     # 19 MB of staging on the device
        del pad
        _give_back()
        st.close()
    a, b = out
    for name in ("pairs", "delta_n", "delta_t", "omega_n", "omega_t"):
        assert getattr(a, name).any() and numpy.array_equal(getattr(a, name), getattr(b, name)), name


def test_sort_products_of_the_list_step_from_a_full_device():
    s = _lattice(1300000)
    st = Stepper([s], precision="mixed")
    st.set_variant(4)
    st.upload()
    st.step(2)
    a = st.sort_products()
    pad = _fill()
    b = st.sort_products()
    del pad
    _give_back()
    st.step(2)
    for u, v in zip(a, b):
        assert numpy.array_equal(u, v)
    assert (numpy.diff(a[0][a[1]].astype(numpy.int64)) >= 0).all()
    st.close()


def test_list_step_that_does_not_fit_gives_back_what_it_got():
    """2.7 kB a sphere of 300,000 with room for a third of it."""
    s = _lattice(300000)
    st = Stepper([s], precision="mixed")
    st.upload()
    pad = torch.empty(((_free() - (300 << 20)) // (2 << 20)) * (2 << 20), dtype=torch.uint8,
                      device="cuda")
    before = _free()
    for _ in range(3):
        with pytest.raises(SphereError) as e:
            st.set_variant(4)
        assert e.value.status == NOMEM and _free() == before
    st.step(2)
    del pad
    _give_back()
    st.set_variant(4)
    st.step(2)
    assert st.tuning()[0] == 4
    st.close()
