"""The kernels that bench.py counts as the interact stage, as sph_profile names
them in each kind of step, and its reference arm where the reference's kernels
are not built: a line that says so, not a measurement of something else."""
import json
import os
import subprocess
import sys

import pytest

import bench


@pytest.mark.parametrize("profiled,stage", [
    (["k_resort", "k_touch", "k_finish", "k_block_sums", "k_box_step"], ["k_touch", "k_finish"]),
    (["k_resort", "k_search", "k_contacts", "k_finish", "k_box_step"],
     ["k_search", "k_contacts", "k_finish"]),
    (["k_hash", "k_scan(3)", "k_scatter", "k_place", "k_vlist", "k_interact", "k_box_step"],
     ["k_interact"]),
    (["k_pair_resort", "k_pair_step", "k_pair_walls"], ["k_pair_step"])])
def test_interact_stage(profiled, stage):
    assert bench.interact_stage(dict.fromkeys(profiled, 0.1)) == stage


@pytest.mark.gpu
def test_interact_stage_names_are_the_profiled_ones():
    from sphere_b200 import scenes
    from sphere_b200.runner import Stepper
    s = scenes.lattice_pack(500, seed=1, periodic=1, nw=1, wmode=1)
    for precision, variant in (("fp64", 1), ("fp64", 3), ("mixed", 3), ("mixed", 4)):
        st = Stepper([s], precision=precision)
        st.set_variant(variant)
        st.upload()
        st.profile(True)
        st.step(8)
        kernels = st.profile_read()
        assert all(k in kernels for k in bench.interact_stage(kernels)), sorted(kernels)
        st.close()


def test_reference_arm_without_the_reference():
    import oracle
    if oracle.available("ref"):
        pytest.skip("the reference's kernels are built here")
    out = subprocess.run([sys.executable, os.path.abspath(bench.__file__), "--impl", "reference", "--steps",
                          "1", "--warmup", "1"], capture_output=True, text=True, timeout=300)
    line = json.loads(out.stdout.strip().splitlines()[-1])
    assert out.returncode == 0 and line["impl"] == "reference"
    assert line["unavailable"] and "value" not in line
