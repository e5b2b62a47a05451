"""Stage launches of small FP64 2+1D events run as programmatic dependents of
one another: a launch's blocks are resident while the one before still writes
the state that they read after its end."""
import os
import re

import numpy as np
import pytest

import vahlib as V

vah = V.product

FIELDS = list(range(16)) + [V.E, V.PP, V.UT, V.UX, V.UY, V.UN]
CSRC = os.path.join(V.ROOT, "gpu-vah_b200", "csrc")


@pytest.mark.parametrize("name", ["vah_march.cuh", "vah_stage.cuh", "vah_tile_cell.cuh"])
def test_stage_code_has_no_read_only_loads(name):
    """ld.global.nc is defined for memory that is constant for the kernel's
    lifetime, which the state is not: no __ldg, nor its wrapper, in stage code."""
    with open(os.path.join(CSRC, name)) as f:
        code = re.sub(r"//.*", "", f.read())
    assert not re.search(r"\b(__)?ldg\(", code)


@pytest.mark.gpu
@pytest.mark.parametrize("flux", [vah.VAH_FLUX_PER_CELL, vah.VAH_FLUX_SHARED])
@pytest.mark.parametrize("nx,ny,steps", [(1, 1, 50), (14, 2, 50), (61, 61, 200), (200, 197, 50), (435, 435, 20)])
def test_dependent_stages_give_the_bits_of_separate_ones(nx, ny, steps, flux):
    """With the event's timing on, event records stand between the stages, which
    then run one after the other."""
    e = V.product.optical_glauber(nx, ny, 0.1, 0.1, b=4.0, e_peak=150.0) + 1e-3
    out = []
    for timing in (False, True):
        ev = vah.Event(nx, ny, 1, 0.1, 0.1, 0.1, 0.16, table=V.eos_table(), t0=0.25, flux=flux)
        ev.init_from_e(0.25, e, vah.VAH_PL_ISOTROPIC)
        ev.set_timing(timing)
        ev.run(0.25, 0.005, steps)
        ev.sync()
        out.append([ev.get_field(f) for f in FIELDS])
        ev.close()
    for f, a, b in zip(FIELDS, *out):
        assert np.array_equal(a, b, equal_nan=True), f
