"""Events that the device can hold, but not with all of their flux differences."""
import numpy as np
import pytest

import vahlib as V

pytestmark = pytest.mark.gpu
vah = V.product


def test_event_is_created_where_its_flux_differences_do_not_fit():
    """An FP32 event of 2.2 GB with 2.8 GB of device memory free, of which all its
    differences would take another 2.2: it is stepped in slabs of planes, with
    the results of an event that has room."""
    torch = pytest.importorskip("torch")
    nx, ny, nz = 301, 301, 121
    z, y, x = np.meshgrid(*((np.arange(n) - 0.5 * (n - 1)) for n in (nz, ny, nx)), indexing="ij", sparse=True)
    e = np.ascontiguousarray(0.1 + 40.0 * np.exp(-(x * x + y * y) / 2000 - z * z / 400))

    def fields():
        ev = vah.Event(nx, ny, nz, 0.2, 0.2, 0.2, 0.16, table=V.eos_table(), t0=0.5, precision=vah.VAH_FP32)
        ev.init_from_e(0.5, e, vah.VAH_PL_ISOTROPIC)
        ev.run(0.5, 0.005, 1)
        ev.sync()
        out = [ev.get_field(f, False) for f in (0, 3, 7, 14, V.E, V.UT, V.UX, V.UN)]
        ev.close()
        return out

    want = fields()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - (2800 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = fields()
    finally:
        del hold
        torch.cuda.empty_cache()
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
