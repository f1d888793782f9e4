"""The split step with its sort and list rebuild on demand (k_resort) and the
search in the contact kernel (k_touch), FP64, bit for bit: against the CPU
oracle at sphere counts around a warp's and a block's share; against the
fused kernel (which sorts at every step) at the counts where the spheres per
warp change, with spheres in random order; and over changes of launch
variant, contact rows set by the caller and the sort products read in
between.  The list step in random sphere order against the FP64 form.  What
a handle runs that chooses no variant: the split step in the FP64 form, the
fused kernel, bit for bit, in the mixed form.  Captured steps when the state
they were captured for changes: radii that no longer fit the cells, and
graphs captured before there was a state."""
import copy

import numpy
import pytest

import cases
import oracle as O
from sphere_b200 import scenes
from sphere_b200.runner import Stepper
from test_gpu_parity import check_same

pytestmark = pytest.mark.gpu


def _pack(n, seed=5, order="lattice"):
    s = scenes.lattice_pack(n, seed=seed, periodic=1, nw=1, wmode=1)
    if order == "random":
        p = numpy.random.default_rng(seed).permutation(n)
        for name in ("x", "radius", "vel", "angvel", "fixvel"):
            setattr(s, name, numpy.ascontiguousarray(getattr(s, name)[p]))
    return s


def _stepper(s, variant, **kw):
    st = Stepper([s], precision="fp64", **kw)
    st.set_variant(variant)
    st.upload()
    return st


def _state(st):
    hp, _ = st.download()
    c, h, d = st.contacts()
    return [getattr(hp, k) for k in ("x", "vel", "angvel", "force", "torque", "es", "ev", "p")] + [c, h, d]


def _same(a, b):
    for u, v in zip(_state(a), _state(b)):
        assert numpy.array_equal(u, v)


@pytest.mark.parametrize("length", ["reference", "fp64"])
@pytest.mark.parametrize("n", [27, 64, 65, 127, 343])
def test_touch_step_matches_oracle(n, length):
    s = _pack(n, order="random")
    cpu = O.CpuRun(s, "oracle", length_mode=0 if length == "reference" else 1)
    st = _stepper(s, 3, length=length)
    for k in (1, 2, 40):
        st.step(k)
        cpu.step(k)
        check_same(st, cpu, s)
    st.close()


@pytest.mark.parametrize("n", [11840, 11841, 23681, 47361])
def test_touch_step_matches_fused_kernel(n):
    s = _pack(n, order="random")
    a, b = _stepper(s, 1), _stepper(s, 3)
    for k in (1, 30):
        a.step(k)
        b.step(k)
        _same(a, b)
        for u, v in zip(a.sort_products(), b.sort_products()):
            assert numpy.array_equal(u, v)
    a.close()
    b.close()


@pytest.mark.parametrize("name", ["fast_spheres", "periodic_xy_wall_stress", "adaptive_grid"])
def test_variant_changes_keep_the_bits(name):
    s, _, _ = cases.make(name)
    a, b = _stepper(s, 1), _stepper(s, 1)
    for variant, lists, k in ((3, 48, 7), (1, 48, 3), (3, 48, 1), (3, 3, 9), (3, 0, 2), (3, 48, 6)):
        b.set_variant(variant)
        b.set_neighbor_lists(lists)
        a.step(k)
        b.step(k)
        _same(a, b)
        # the rows handed back through the caller: k_touch must take them anew
        c, h, _ = b.contacts()
        b.set_contacts(c, h)
        a.set_contacts(c, h)
    a.close()
    b.close()


def test_list_step_in_random_order_matches_fp64_form():
    """One step from the same state: the mixed form's force bound (1e-5), the
    same contact sets, the caller's sphere numbering throughout."""
    n = 3000
    s = _pack(n, order="random")
    a = _stepper(s, 1)
    m = Stepper([s], precision="mixed", length="reference")
    m.set_variant(4)
    m.upload()
    a.step(1)
    m.step(1)
    ha, hm = a.download()[0], m.download()[0]
    assert numpy.linalg.norm(hm.force - ha.force) <= 1e-5 * numpy.linalg.norm(ha.force)
    # a position moves by (2/3) F / m dt^2 in the step
    m_s = 4.0 / 3.0 * numpy.pi * s.radius ** 3 * float(s.rho[0])
    move = numpy.linalg.norm(ha.force / m_s[:, None]) * float(s.time_dt[0]) ** 2
    assert numpy.linalg.norm(hm.x - ha.x) <= 1e-5 * move + 1e-15 * numpy.linalg.norm(ha.x)
    ca, cm = (numpy.sort(q.contacts()[0].reshape(n, -1), axis=1) for q in (a, m))
    assert numpy.array_equal(ca, cm)
    cid, perm, start, _ = m.sort_products()
    assert numpy.array_equal(numpy.sort(perm), numpy.arange(n))
    assert (numpy.diff(cid[perm].astype(numpy.int64)) >= 0).all()
    for u, v in zip(a.sort_products(), (cid, perm, start, _)):
        assert numpy.array_equal(u, v)
    a.close()
    m.close()


@pytest.mark.parametrize("length", ["reference", "fp64"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_default_variant_keeps_the_fused_kernel_bits(precision, length):
    """Against variant 1 over 60 steps of a pack in contact and of a bonded
    one.  In the mixed form the split step's contractions need not be the
    fused kernel's, so only the fused kernel itself gives its bits."""
    bonded = scenes.bonded_pack(2000, nbonds=3000, seed=1, device=0)
    for s in (_pack(3000, order="random"), bonded):
        a, b = (Stepper([s], precision=precision, length=length) for _ in range(2))
        a.set_variant(1)
        for st in (a, b):
            st.upload()
            st.step(60)
        assert b.tuning()[0] == (3 if precision == "fp64" else 1)
        _same(a, b)
        a.close()
        b.close()


@pytest.mark.parametrize("profile", [False, True])
def test_upload_of_radii_wider_than_a_cell_on_the_same_handle(profile):
    """k_touch asks for cells wider than the largest diameter; the second
    upload's spheres are wider, so that pairs two cells apart overlap which
    the +-1 cell search does not visit; the third's fit again."""
    s = scenes.gravity_settling(400, seed=3)
    wide = copy.deepcopy(s)
    wide.radius = s.radius * 1.6
    cell = numpy.asarray(s.L) / numpy.asarray(s.num)
    assert (2.0 * s.radius.max() < cell).all() and (cell < 2.0 * wide.radius.max()).all()
    c = numpy.floor(s.x / cell)
    apart = numpy.abs(c[:, None] - c[None]).max(-1) > 1
    dist = numpy.linalg.norm(s.x[:, None] - s.x[None], axis=-1)
    assert (apart & (dist < wide.radius[:, None] + wide.radius[None])).any()
    st = Stepper([s], precision="fp64")
    st.set_variant(3)
    if profile:
        st.profile(True)
    for q in (s, wide, s):
        st.sims[:] = [q]
        st.upload()
        ref = _stepper(q, 1)
        for k in (1, 5, 20):
            st.step(k)
            ref.step(k)
            _same(ref, st)
            for u, v in zip(ref.sort_products(), st.sort_products()):
                assert numpy.array_equal(u, v)
        ref.close()
    st.close()


@pytest.mark.parametrize("precision,variant", [("fp64", 3), ("mixed", 4)])
def test_graphs_captured_before_the_first_upload(precision, variant):
    """sph_profile captures its steps; before an upload these cannot be the
    lazily sorted step or the list step, which the handle then runs."""
    s = _pack(343)
    out = []
    for early in (True, False):
        st = Stepper([s], precision=precision)
        st.set_variant(variant)
        if early:
            st.profile(True)
        st.upload()
        st.step(2)
        st.profile(False)
        st.step(9)
        out.append(_state(st))
        st.close()
    for u, v in zip(*out):
        assert numpy.array_equal(u, v)


@pytest.mark.parametrize("sweeps", [0, 1])
def test_sort_products_after_packing_sweeps(sweeps):
    """Those of the last sweep, or with no sweep of the last step, as from the
    kernel that sorts at every step."""
    s = scenes.gravity_settling(3000, seed=3)
    s.vel[:] = numpy.random.default_rng(0).normal(0.0, 1.0, s.vel.shape)
    out = []
    for variant in (1, 3):
        st = _stepper(s, variant)
        st.step(60)
        if sweeps:
            st.relax(sweeps, alpha=0.5, z_top=float(s.L[2]))
        else:
            st._check(st.lib.sph_relax(st.h, 0, 0.5, float(s.L[2]), None), "sph_relax")
        out.append(st.sort_products())
        st.close()
    for u, v in zip(*out):
        assert numpy.array_equal(u, v)
