"""A batch's capacity bounds its device memory up to a constant, the scratch of
the flux differences included, and any set of events that is admitted can be
stepped: in groups and slabs of planes where the scratch is short (256 MB where
the events leave less), with the same results."""
import ctypes as C

import numpy as np
import pytest

import vahlib as V

pytestmark = pytest.mark.gpu
vah = V.product

FIELDS = list(range(16)) + [V.E, V.PP, V.UT, V.UX, V.UY, V.UN]


def lump(nx, ny, nz, seed):
    rng = np.random.default_rng(seed)
    z, y, x = np.meshgrid(*((np.arange(n) - 0.5 * (n - 1)) for n in (nz, ny, nx)), indexing="ij")
    c = rng.normal(size=3) * 2
    return np.ascontiguousarray(0.05 + 40.0 * np.exp(-((x - c[0]) ** 2 + (y - c[1]) ** 2) / 50 - (z - c[2]) ** 2 / 40))


def fields(b, slot, n):
    out = np.zeros(n)
    res = []
    for f in FIELDS:
        vah.check(b.L.vah_batch_get_field(b.b, slot, f, out.ctypes.data_as(C.POINTER(C.c_double)), 0), "get_field")
        res.append(out.copy())
    return res


def run(capacity, shapes, steps, **opt):
    tab = V.eos_table()
    b = vah.Batch(table=tab, capacity_bytes=capacity, **opt)
    slots = [b.add(*s, 0.2, 0.2, 0.2, 0.5, 0.005, 0.16, lump(*s, seed=k), vah.VAH_PL_ISOTROPIC)
             for k, s in enumerate(shapes)]
    assert all(s is not None for s in slots)
    top = b.max_energy_density(len(slots))  # before any step
    b.step(steps)
    b.sync()
    out = [fields(b, s, int(np.prod(shape))) for s, shape in zip(slots, shapes)]
    info = [(b.info(s).steps, b.info(s).face_fallbacks, b.info(s).cell_fallbacks) for s in slots]
    obs = np.array(b.observables(len(slots)))
    b.close()
    return top, out, info, obs


@pytest.mark.parametrize("precision,shapes", [
    # FP64: differences of 477 MB (an event in two slabs), of 190 MB, and of small ones
    (vah.VAH_FP64, [(121, 119, 81), (97, 95, 49), (33, 35, 1), (16, 9, 2)]),
    # a 2+1D event whose one plane takes 305 MB, more than the scratch may take of itself
    (vah.VAH_FP64, [(1091, 1087, 1), (61, 57, 21)]),
    # FP32: 279 MB, in two slabs
    (vah.VAH_FP32, [(127, 125, 90), (41, 43, 12)]),
])
@pytest.mark.parametrize("flux", [vah.VAH_FLUX_PER_CELL, vah.VAH_FLUX_SHARED])
@pytest.mark.parametrize("room", [0.0, 0.8])
def test_a_full_batch_steps_with_the_same_results(precision, shapes, flux, room):
    """room: what the events leave of the capacity, in footprints of the first."""
    opt = dict(precision=precision, flux=flux)
    probe = vah.Batch(table=V.eos_table(), **opt)
    per = [probe.event_bytes(*s) for s in shapes]
    probe.close()
    full = run(sum(per) + int(room * per[0]), shapes, 2, **opt)
    wide = run(16 << 30, shapes, 2, **opt)
    assert np.array_equal(full[0], wide[0])
    assert full[2] == wide[2]
    for a, b in zip(full[1], wide[1]):
        for f, x, y in zip(FIELDS, a, b):
            assert np.array_equal(x, y), f
    # sums of a cell item's block, added item by item: in another grouping, to rounding
    assert np.allclose(full[3], wide[3], rtol=1e-11, atol=1e-14)


def test_device_memory_stays_within_the_capacity():
    """FP32 events of 131 MB whose differences would take as much again: beside
    the capacity, the scratch's 256 MB, and 128 MB for the lists and what the
    pool rounds up (it maps 32 MB pieces)."""
    torch = pytest.importorskip("torch")
    shape, n = (97, 97, 65), 8
    tab, e = V.eos_table(), lump(97, 97, 65, seed=1)
    probe = vah.Batch(table=tab, precision=vah.VAH_FP32)
    per = probe.event_bytes(*shape)
    probe.close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    b = vah.Batch(table=tab, capacity_bytes=n * per, precision=vah.VAH_FP32)
    slots = [b.add(*shape, 0.2, 0.2, 0.2, 0.5, 0.005, 0.16, e, vah.VAH_PL_ISOTROPIC) for _ in range(n)]
    assert all(s is not None for s in slots)
    assert b.add(*shape, 0.2, 0.2, 0.2, 0.5, 0.005, 0.16, e, vah.VAH_PL_ISOTROPIC) is None
    b.step(2)
    b.sync()
    used = before - torch.cuda.mem_get_info()[0]
    b.close()
    assert used < n * per + (256 << 20) + (128 << 20)


def test_scratch_makes_way_for_events():
    """Events admitted one by one, with steps between: the scratch grown for the
    first ones gives way as the capacity fills, and events leave again."""
    tab = V.eos_table()
    shape = (101, 99, 61)  # 247 MB of differences each
    probe = vah.Batch(table=tab)
    per = probe.event_bytes(*shape)
    probe.close()
    b = vah.Batch(table=tab, capacity_bytes=4 * per)
    alone = vah.Batch(table=tab, capacity_bytes=1 << 30)
    e = [lump(*shape, seed=k) for k in range(5)]
    live = []
    for k in range(4):
        live.append(b.add(*shape, 0.2, 0.2, 0.2, 0.5, 0.005, 0.16, e[k], vah.VAH_PL_ISOTROPIC))
        assert live[-1] is not None
        b.step(1)
    b.remove(live[1])
    live[1] = b.add(*shape, 0.2, 0.2, 0.2, 0.5, 0.005, 0.16, e[4], vah.VAH_PL_ISOTROPIC)
    b.step(3)
    b.sync()
    for slot, k, steps in ((live[0], 0, 7), (live[3], 3, 4), (live[1], 4, 3)):
        r = alone.add(*shape, 0.2, 0.2, 0.2, 0.5, 0.005, 0.16, e[k], vah.VAH_PL_ISOTROPIC)
        alone.step(steps)
        n = int(np.prod(shape))
        for f, x, y in zip(FIELDS, fields(b, slot, n), fields(alone, r, n)):
            assert np.array_equal(x, y), (k, f)
        alone.remove(r)
    b.close()
    alone.close()
