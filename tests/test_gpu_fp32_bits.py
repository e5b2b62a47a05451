"""The FP32 form's bits: the sums whose fused product the compiler chose kernel
by kernel, and the events whose dilute edge cells make such a choice visible."""
import ctypes as C
import os

import numpy as np
import pytest

import vahlib as V

pytestmark = pytest.mark.gpu
vah = V.product

PHYSICS = {"ideal": 0, "shear": 1, "bulk": 2}
FIELDS = {"ideal": list(range(5)), "shear": list(range(15)), "bulk": list(range(16))}
PRIMITIVES = [V.E, V.PP, V.UT, V.UX, V.UY, V.UN]


def spots(n, seed, e_peak=350.0, dx=0.1):
    """Gaussian deposits of width 0.5 fm in a box that is mostly dilute, over the floor."""
    rng = np.random.default_rng(seed)
    x = (np.arange(n) - 0.5 * (n - 1)) * dx
    c = rng.normal(scale=2.0, size=(60, 2)) * (0.6, 1.2)
    v = np.exp(-0.5 * ((x[None] - c[:, 1:]) / 0.5) ** 2).T @ np.exp(-0.5 * ((x[None] - c[:, :1]) / 0.5) ** 2)
    return e_peak * v / v.max() + 1e-3


def form(physics, eos):
    table = eos == "table"
    return dict(physics=PHYSICS[physics], table=V.eos_table() if table else None, precision=vah.VAH_FP32,
                eos=vah.VAH_EOS_TABLE if table else vah.VAH_EOS_CONFORMAL,
                zeta=vah.VAH_ZETA_CROSSOVER if table else vah.VAH_ZETA_REFERENCE)


def event_fields(e, dx, t0, dt, steps, ids, **opt):
    nz, ny, nx = e.shape
    ev = vah.Event(nx, ny, nz, dx, dx, dx, 0.16, t0=t0, **opt)
    ev.init_from_e(t0, e, vah.VAH_PL_ISOTROPIC)
    ev.run(t0, dt, steps)
    out = [ev.get_field(f, False).reshape(e.shape) for f in ids]
    ev.close()
    return out


def batch_fields(e, dx, t0, dt, steps, ids, **opt):
    nz, ny, nx = e.shape
    b = vah.Batch(capacity_bytes=4 << 30, **opt)
    slot = b.add(nx, ny, nz, dx, dx, dx, t0, dt, 0.16, e, vah.VAH_PL_ISOTROPIC)
    b.step(steps)
    out = []
    for f in ids:
        a = np.zeros(e.size)
        vah.check(b.L.vah_batch_get_field(b.b, slot, f, a.ctypes.data_as(C.POINTER(C.c_double)), 0), "get_field")
        out.append(a.reshape(e.shape))
    b.close()
    return out


@pytest.mark.parametrize("run", [event_fields, batch_fields])
def test_edge_cells_of_a_2d_event_hold_the_recorded_velocities(run):
    """50 steps of a 161x161 event whose edge cells amplify a last bit about 1e8
    times, against u recorded on a B200 from the tiled FP32 kernels that the
    flux and cell launches replaced, in the 41x41 cells around the worst one.
    The FP64 parts of the form (inversions, closure fits) round a float
    differently in one cell of 4e5 per step, which reaches u at about 1e-6;
    10 times that is allowed. A sum fused another way comes to 1e-3 here."""
    gold = np.load(os.path.join(os.path.dirname(__file__), "golden", "fp32_2d_edge_cell_u.npy"))
    y, x = 108, 22
    u = run(spots(161, 29)[None], 0.1, 0.25, 0.01, 50, [V.UT, V.UX, V.UY], **form("bulk", "table"))
    for m in range(3):
        assert np.max(np.abs(u[m][0, y:y + 41, x:x + 41] - gold[m])) < 1e-5, m


@pytest.mark.parametrize("eos", ["table", "conformal"])
@pytest.mark.parametrize("physics", ["ideal", "shear", "bulk"])
@pytest.mark.parametrize("nz", [1, 21])
def test_event_and_batch_kernels_round_alike(physics, eos, nz):
    """Bit for bit after 20 steps (times and steps exact in binary, so that both
    clocks agree)."""
    eta = np.exp(-0.5 * ((np.arange(nz) - 0.5 * (nz - 1)) * 0.25) ** 2) if nz > 1 else np.ones(1)
    e = spots(65 if nz == 1 else 33, 3)[None] * eta[:, None, None] + 1e-3
    ids = FIELDS[physics] + PRIMITIVES
    args = (np.ascontiguousarray(e), 0.125 if nz == 1 else 0.25, 0.25, 2.0 ** -7, 20, ids)
    a, b = (run(*args, **form(physics, eos)) for run in (event_fields, batch_fields))
    for f, p, q in zip(ids, a, b):
        assert np.array_equal(p, q, equal_nan=True), (f, np.count_nonzero(p != q))
