"""The flux and cell launches (vah_march.cuh) where their division of the
lattice can go wrong: rows and columns around the warps' widths (14 / 16 cells
for FP64, 30 / 32 for FP32), single rows and planes, and lattices whose flux
differences do not fit the scratch at once."""
import numpy as np
import pytest

import vahlib as V

pytestmark = pytest.mark.gpu
vah = V.product

STATE = list(range(16)) + [V.E, V.PP, V.UT, V.UX, V.UY, V.UN]


def lumps(nx, ny, nz, seed, e_peak=40.0):
    """A few smooth lumps over a floor, off centre, so that no face is trivial."""
    rng = np.random.default_rng(seed)
    z, y, x = np.meshgrid(*(np.arange(n, dtype=float) for n in (nz, ny, nx)), indexing="ij")
    e = np.full(z.shape, 0.5)
    for _ in range(4):
        c = rng.random(3) * (nz, ny, nx)
        e += e_peak * rng.random() * np.exp(-((x - c[2]) ** 2 + (y - c[1]) ** 2 + (z - c[0]) ** 2) / (2 * 4.0 ** 2))
    return e


@pytest.mark.parametrize("shape", [(1, 1, 1), (13, 1, 1), (14, 2, 1), (15, 16, 1), (17, 3, 2), (29, 33, 1), (30, 5, 3),
                                   (31, 31, 2), (32, 15, 5), (3, 47, 6), (64, 2, 17)])
def test_fp64_steps_match_the_oracle_around_the_warp_widths(shape):
    """Three steps against the CPU oracle: normwise 1e-11 per field, the bound
    the fixture tests hold a few steps to (rounding of a step times its growth)."""
    nx, ny, nz = shape
    tab = V.eos_table()
    g = V.Grid(nx, ny, nz, 0.3, 0.25, 0.2, 0.16, physics="pimunu_pi", eos="table", zeta="crossover", table=tab)
    e = lumps(nx, ny, nz, seed=nx + 7 * ny + 31 * nz)
    ev = V.Event(g, t0=0.5)
    ev.init_from_e(0.5, e.ravel(), vah.VAH_PL_ISOTROPIC)
    o = V.Oracle(g)
    V.load_state(o, {f: ev.get_field(f) for f in STATE})
    o.set_conserved(0.5, 1)
    o.set_ghost_cells()
    o.run(0.5, 0.01, 3)
    ev.run(0.5, 0.01, 3)
    ev.sync()
    scale = 1e-3 * np.max(g.interior(o.field(V.E)))  # of the viscous fields where they are analytically ~0
    for f in STATE:
        a, b = g.interior(o.field(f)), g.interior(ev.get_field(f))
        size = max(np.max(np.abs(a)), scale if 5 <= f < 16 else 0.0, 1e-6)
        assert np.max(np.abs(a - b)) / size < 1e-11, f
    ev.close()


@pytest.mark.parametrize("shape", [(1, 1, 1), (29, 3, 1), (30, 31, 1), (31, 2, 4), (33, 32, 3), (5, 65, 7)])
def test_fp32_steps_track_the_fp64_shared_form(shape):
    """Three FP32 steps against the FP64 shared-face form, the same scheme: e
    and u within 1e-5 normwise (some hundred FP32 roundings; an indexing error
    is of order 1)."""
    nx, ny, nz = shape
    tab = V.eos_table()
    e = lumps(nx, ny, nz, seed=nx + ny + nz).ravel()
    got = []
    for precision, flux in ((vah.VAH_FP32, vah.VAH_FLUX_PER_CELL), (vah.VAH_FP64, vah.VAH_FLUX_SHARED)):
        ev = vah.Event(nx, ny, nz, 0.3, 0.25, 0.2, 0.16, table=tab, t0=0.5, precision=precision, flux=flux)
        ev.init_from_e(0.5, e)
        ev.run(0.5, 0.01, 3)
        ev.sync()
        got.append({f: ev.get_field(f, False) for f in (V.E, V.UT, V.UX, V.UY)})
        ev.close()
    for f in got[0]:
        assert np.max(np.abs(got[0][f] - got[1][f])) / max(np.max(np.abs(got[1][f])), 1e-2) < 1e-5, f


def test_lattice_stepped_in_slabs_matches_the_fused_stage():
    """161 x 161 x 451 needs more than 4 GB of flux differences, so a stage runs
    slab by slab; the fused stage keeps none. Same face semantics: 1e-12."""
    nx, ny, nz = 161, 161, 451
    tab = V.eos_table()
    e = lumps(nx, ny, nz, seed=5).ravel()
    got = []
    for flux in (vah.VAH_FLUX_PER_CELL, vah.VAH_FLUX_PER_CELL_FUSED):
        ev = vah.Event(nx, ny, nz, 0.2, 0.2, 0.2, 0.16, table=tab, t0=0.5, flux=flux)
        ev.init_from_e(0.5, e)
        ev.run(0.5, 0.01, 2)
        ev.sync()
        got.append({f: ev.get_field(f, False) for f in (V.E, V.PL, V.UX, V.UN)})
        ev.close()
    for f in got[0]:
        assert np.max(np.abs(got[0][f] - got[1][f])) < 1e-12 * np.max(np.abs(got[1][f])), f


def test_batch_in_groups_equals_each_event_alone():
    """Two events of 2.3 GB of flux differences each do not share the scratch
    and step as two groups: bit for bit as alone."""
    tab = V.eos_table()
    nx, ny, nz = 161, 161, 227
    es = [lumps(nx, ny, nz, seed=s).ravel() for s in (11, 12)]

    def run(which):
        b = vah.Batch(table=tab, capacity_bytes=24 << 30)
        slots = [b.add(nx, ny, nz, 0.2, 0.2, 0.2, 0.5, 0.01, 0.16, es[k]) for k in which]
        b.step(2)
        out = [{f: b.get_field(s, f, False) for f in (V.E, V.UX)} for s in slots]
        b.close()
        return out

    both = run((0, 1))
    for k in (0, 1):
        alone = run((k,))[0]
        for f in alone:
            np.testing.assert_array_equal(both[k][f], alone[f])


@pytest.mark.parametrize("precision", [0, 1])
def test_field_reads_and_writes_across_staging_runs(precision):
    """A field of more values than the 8 MB staging holds goes through in runs
    of rows, interior and ghosted, and comes back as written."""
    nx, ny, nz = 131, 127, 75
    tab = V.eos_table()
    ev = vah.Event(nx, ny, nz, 0.2, 0.2, 0.2, 0.16, table=tab, t0=0.5, precision=precision)
    rng = np.random.default_rng(2)
    full = rng.random((nz + 4, ny + 4, nx + 4)).astype(np.float32).astype(np.float64)
    ev.set_field(V.E, full.ravel())
    np.testing.assert_array_equal(ev.get_field(V.E), full.ravel())
    np.testing.assert_array_equal(ev.get_field(V.E, False), full[2:-2, 2:-2, 2:-2].ravel())
    inner = rng.random((nz, ny, nx)).astype(np.float32).astype(np.float64)
    ev.set_field(V.E, inner.ravel(), False)
    full[2:-2, 2:-2, 2:-2] = inner
    np.testing.assert_array_equal(ev.get_field(V.E), full.ravel())
    ev.close()
