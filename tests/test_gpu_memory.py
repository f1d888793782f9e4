"""Calls that find no device memory: they report it or do without, and leave
nothing behind that a later call would take for an error of its own."""
import numpy
import pytest

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
