"""The work that is timed: what a user of the VAH time step has it do, through
the library's public entry points (include/vah.h, reached by ctypes as the
Python binding gpu-vah_b200/vah.py does).

Four kinds of case, each a whole call sequence of a user's program:

  event    one event: its initial state from an energy density on the host
           (vah_event_init_from_e), `steps` RK2 steps (vah_run), and every
           field of its state read back (vah_event_get_field);
  batch    several events of uneven size admitted together (vah_batch_add),
           `steps` steps of all of them (vah_batch_step), every field of every
           event read back, and the events removed again;
  host     one RK2 step on host arrays in place (vah_rk2_step_host), as a
           program that keeps its own driver calls it in its time loop;
  buffers  one RK2 step (two vah_stage_noalloc calls) on device buffers that
           the caller owns.

The initial energy densities are MC-Glauber-like: participants of two
Woods-Saxon nuclei, Gaussian deposits, a plateau with Gaussian flanks along
eta, the 1e-3 fm^-4 floor. exact() restates the whole scheme in torch, FP64.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-vah_b200"))
import vah  # noqa: E402

HBARC = 0.197326938
EOS_FACTOR = 13.8997
PHYSICS = {"ideal": 0, "shear": 1, "bulk": 2}
NQ = {"ideal": 5, "shear": 15, "bulk": 16}
FLUX = {"per_cell": vah.VAH_FLUX_PER_CELL, "shared": vah.VAH_FLUX_SHARED}
TABLE_N = 4096


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # the headline event: rhic-conf's spacing and step, lattice of the benchmark; the evolution between
        # two readings of the state
        dict(name="event_fp64_121x121x81", kind="event", nx=121, ny=121, nz=81, dx=0.1, dz=0.1, steps=40, dt=0.005,
             physics="bulk", eos="table", precision="fp64", flux="per_cell", pl="reference", T0=0.6, b=7.0),
        # the same event in the FP32 form
        dict(name="event_fp32_121x121x81", kind="event", nx=121, ny=121, nz=81, dx=0.1, dz=0.1, steps=60, dt=0.005,
             physics="bulk", eos="table", precision="fp32", flux="per_cell", pl="reference", T0=0.6, b=7.0),
        # a parameter scan's event: middling 3+1D lattice with ragged sides, shear only, conformal gas
        dict(name="event_fp64_61x57x21", kind="event", nx=61, ny=57, nz=21, dx=0.2, dz=0.2, steps=40, dt=0.01,
             physics="shear", eos="conformal", precision="fp64", flux="per_cell", pl="isotropic", T0=0.5, b=5.0),
        # the same size of event in the FP32 form, shear + bulk under the table
        dict(name="event_fp32_81x77x41", kind="event", nx=81, ny=77, nz=41, dx=0.2, dz=0.2, steps=30, dt=0.01,
             physics="bulk", eos="table", precision="fp32", flux="per_cell", pl="isotropic", T0=0.4, b=9.0),
        # the boost-invariant conformal event that validation runs use: few cells, many steps, launch-bound
        dict(name="event_fp64_61x61", kind="event", nx=61, ny=61, nz=1, dx=0.2, dz=0.2, steps=50, dt=0.01,
             physics="shear", eos="conformal", precision="fp64", flux="per_cell", pl="isotropic", T0=0.6, b=7.0),
        # a wide boost-invariant event under the table
        dict(name="event_fp64_401x389", kind="event", nx=401, ny=389, nz=1, dx=0.05, dz=0.1, steps=40, dt=0.005,
             physics="bulk", eos="table", precision="fp64", flux="per_cell", pl="reference", T0=0.6, b=6.0),
        # faces evaluated once each, the option of programs that do not need the reference's fallbacks
        dict(name="event_fp64_shared_75x83x33", kind="event", nx=75, ny=83, nz=33, dx=0.15, dz=0.15, steps=30,
             dt=0.005, physics="bulk", eos="table", precision="fp64", flux="shared", pl="reference", T0=0.5, b=8.0),
        # event-by-event studies: a batch of 2+1D events of uneven size, in both forms
        dict(name="batch_fp64_2d", kind="batch", events=32, side_min=81, side_max=201, side_step=40, nz=1, dx=0.1,
             dz=0.1, steps=50, dt=0.01, physics="bulk", eos="table", precision="fp64", flux="per_cell",
             pl="isotropic", T0=0.6, b=12.0),
        dict(name="batch_fp32_2d", kind="batch", events=32, side_min=81, side_max=201, side_step=40, nz=1, dx=0.1,
             dz=0.1, steps=50, dt=0.01, physics="bulk", eos="table", precision="fp32", flux="per_cell",
             pl="isotropic", T0=0.6, b=12.0),
        # a few full events of a serving stream's size
        dict(name="batch_fp64_3d", kind="batch", events=3, side_min=81, side_max=97, side_step=8, nz=41, dx=0.2,
             dz=0.2, steps=20, dt=0.01, physics="bulk", eos="table", precision="fp64", flux="per_cell",
             pl="isotropic", T0=0.4, b=12.0),
        # a host program's time loop that hands its arrays over for one step
        dict(name="host_fp64_121x121x81", kind="host", nx=121, ny=121, nz=81, dx=0.1, dz=0.1, steps=1, dt=0.005,
             physics="bulk", eos="table", precision="fp64", flux="per_cell", pl="reference", T0=0.6, b=7.0),
        # the smallest call: one step on the caller's own device buffers
        dict(name="buffers_25x23x9", kind="buffers", nx=25, ny=23, nz=9, dx=0.3, dz=0.2, steps=1, dt=0.01,
             physics="bulk", eos="table", precision="fp64", flux="per_cell", pl="isotropic", T0=0.5, b=4.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["event", "event", "event", "event", "batch", "batch", "host", "buffers"])
    physics, eos = rng.choice([("bulk", "table")] * 4 + [("shear", "table"), ("shear", "conformal"),
                                                         ("ideal", "table"), ("ideal", "conformal")])
    c = dict(kind=kind, physics=physics, eos=eos, precision=rng.choice(["fp64", "fp64", "fp32"]), flux="per_cell",
             pl=rng.choice(["reference", "isotropic"]) if eos == "table" else "isotropic",
             T0=rng.choice([0.4, 0.5, 0.6]), b=round(rng.uniform(0.0, 10.0), 2))
    flat = rng.random() < 0.4  # boost-invariant
    if kind == "batch":
        c["side_min"] = _log_int(rng, 31, 101) if flat else _log_int(rng, 31, 71)
        c["side_step"] = rng.randint(3, 30)
        c["events"] = rng.randint(2, 24) if flat else rng.randint(2, 4)
        c["side_max"] = c["side_min"] + c["side_step"] * rng.randint(1, 3)
        c["nz"] = 1 if flat else rng.randint(5, 33)
    else:
        c["nx"], c["ny"] = (_log_int(rng, 31, 401) if flat else _log_int(rng, 21, 121) for _ in range(2))
        c["nz"] = 1 if flat else _log_int(rng, 5, 81)
    if kind == "buffers":  # the library's fixed scratch bounds these
        c["precision"] = "fp64"
        c["nx"], c["ny"] = min(c["nx"], 301 if flat else 45), min(c["ny"], 301 if flat else 45)
        c["nz"] = min(c["nz"], 25)
    elif c["precision"] == "fp64" and kind != "host" and rng.random() < 0.2:
        c["flux"] = "shared"
    c["steps"] = 1 if kind in ("host", "buffers") else _log_int(rng, 8, 40)
    c["dx"], c["dz"] = rng.choice([0.1, 0.15, 0.2]), rng.choice([0.1, 0.2])
    c["dt"] = round(c["dx"] * rng.choice([0.04, 0.05]), 6)
    return c


def _sides(case):
    """The lattices (nx, ny, nz) of a case, one per event."""
    if case["kind"] != "batch":
        return [(case["nx"], case["ny"], case["nz"])]
    sides = list(range(case["side_min"], case["side_max"] + 1, case["side_step"]))
    return [(sides[m % len(sides)], sides[(m * 3 + m // len(sides)) % len(sides)] if case["nz"] > 1
             else sides[m % len(sides)], case["nz"]) for m in range(case["events"])]


def work(case):
    """Per cell and step: the state in and out of both stages once (5 N_q + 32 values), and the scheme's
    floating-point operations, counted from its formulas: per face (one per axis) the limited reconstruction of
    both sides (22 N_q), the flux (6 N_q with its difference) and two inversions (60 each); per cell the sources
    and the regulator (about 1500 with shear, 700 without), the closure fits (2 x 10 terms, a product and a sum
    each), one inversion."""
    nq = NQ[case["physics"]]
    cells = sum(nx * ny * nz for nx, ny, nz in _sides(case))
    axes = 3 if case["nz"] > 1 else 2
    fits = {"ideal": 5, "shear": 5, "bulk": 13}[case["physics"]]
    per_stage = axes * (28 * nq + 120) + (700 if nq == 5 else 1500) + 40 * fits + 60
    width = 4 if case["precision"] == "fp32" else 8
    return {"bytes": float(cells * case["steps"] * (5 * nq + 32) * width),
            "flops": float(cells * case["steps"] * 2 * per_stage)}


# ----------------------------------------------------------------- inputs --
_table = None


def _eos_table():
    """A tabulated crossover EoS in the layout of include/vah.h, made here: c_s^2(T) = 1/3 - d / (1 + (T/Tc)^4),
    d ln s / d ln T = 1 / c_s^2, normalised to the conformal gas at high T; p by quadrature, e = T s - p."""
    global _table
    if _table is None:
        d, Tc = 1.0 / 3.0 - 0.15, 0.155 / HBARC
        a = 1.0 - 3.0 * d
        lnT = np.linspace(math.log(0.001 / HBARC), math.log(10.0 / HBARC), (1 << 19) + 1)

        def entropy(x):
            t4 = np.exp(4.0 * (x - math.log(Tc)))
            return 4.0 / 3.0 * EOS_FACTOR * np.exp(3.0 * x) * (t4 / (t4 + a)) ** (9.0 * d / (4.0 * a))

        T, s = np.exp(lnT), entropy(lnT)
        mid = 0.5 * (lnT[1:] + lnT[:-1])
        piece = (lnT[1] - lnT[0]) / 6.0 * (s[:-1] * T[:-1] + 4.0 * entropy(mid) * np.exp(mid) + s[1:] * T[1:])
        p = 3.0 * T[0] * s[0] / 23.0 + np.concatenate([[0.0], np.cumsum(piece)])
        lne = np.log(T * s - p)
        lo, hi = np.interp([math.log(0.005 / HBARC), math.log(5.0 / HBARC)], lnT, lne)
        nodes = np.linspace(lo, hi, TABLE_N)
        lnTn, pn = np.interp(nodes, lne, lnT), np.exp(np.interp(nodes, lne, np.log(p)))
        Tn = np.exp(lnTn)
        head = [TABLE_N, lo, (TABLE_N - 1) / (hi - lo), (hi - lo) / (TABLE_N - 1), math.exp(lo), hi, math.exp(hi), 0.0]
        _table = np.concatenate([head, pn, Tn, 1.0 / 3.0 - d / (1.0 + (Tn / Tc) ** 4)])
    return _table


def _peak(case):
    """Energy density at the peak temperature."""
    T = case["T0"] / HBARC
    if case["eos"] == "conformal":
        return EOS_FACTOR * T ** 4
    t = _eos_table()
    n = TABLE_N
    return float(np.exp(np.interp(math.log(T), np.log(t[8 + n:8 + 2 * n]), t[1] + t[3] * np.arange(n))))


def _energy_density(rng, nx, ny, nz, dx, dz, b, e_peak):
    """e(eta, y, x) of one collision of two Au nuclei."""
    r = np.linspace(0.0, 15.0, 3001)
    cdf = np.cumsum(r * r / (1.0 + np.exp((r - 6.38) / 0.535)))

    def nucleus(shift):
        rad = np.interp(rng.random(197), cdf / cdf[-1], r)
        ct, ph = 2.0 * rng.random(197) - 1.0, 2.0 * math.pi * rng.random(197)
        st = np.sqrt(1.0 - ct * ct)
        return np.stack([rad * st * np.cos(ph) + shift, rad * st * np.sin(ph)], 1)

    A, B = nucleus(0.5 * b), nucleus(-0.5 * b)
    hit = ((A[:, None] - B[None]) ** 2).sum(2) < 4.2 / math.pi
    part = np.concatenate([A[hit.any(1)], B[hit.any(0)]])
    if not len(part):
        part = np.zeros((1, 2))
    x, y = (np.arange(nx) - 0.5 * (nx - 1)) * dx, (np.arange(ny) - 0.5 * (ny - 1)) * dx
    gx = np.exp(-0.5 * ((x[None] - part[:, :1]) / 0.5) ** 2)
    gy = np.exp(-0.5 * ((y[None] - part[:, 1:]) / 0.5) ** 2)
    v = gy.T @ gx
    eta = np.abs((np.arange(nz) - 0.5 * (nz - 1)) * dz)
    f = np.exp(-0.5 * (np.maximum(eta - 1.5, 0.0) / 1.3) ** 2) if nz > 1 else np.ones(1)
    return np.ascontiguousarray(e_peak / v.max() * v[None] * f[:, None, None] + 1e-3)


def _inputs(case, seed):
    rng = np.random.default_rng([int(seed), 2024])
    out = []
    for nx, ny, nz in _sides(case):
        b = case["b"] if case["kind"] != "batch" else case["b"] * rng.random()
        out.append(_energy_density(rng, nx, ny, nz, case["dx"], case["dz"], b, _peak(case)))
    return out


T_INIT, ETA_S = 0.25, 0.16
FIELDS = {"ideal": list(range(5)) + list(range(16, 22)), "shear": list(range(15)) + list(range(16, 22)),
          "bulk": list(range(22))}
HOST_RESTART = 40  # a host loop starts its next event after this many steps


def _groups(case, rows):
    """The state from its field rows: the conserved block (T^{tau mu}, P_L, pi, Pi), e, p, u."""
    n = NQ[case["physics"]]
    return {"q": rows[:n], "e": rows[n], "p": rows[n + 1], "u": rows[n + 2:n + 6]}


def _pl_mode(case):
    return vah.VAH_PL_REFERENCE if case["pl"] == "reference" else vah.VAH_PL_ISOTROPIC


def _address(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def _pinned(*shape, dtype=torch.float64):
    return torch.empty(*shape, dtype=dtype, pin_memory=torch.cuda.is_available())


def prepare(case, seed):
    e = _inputs(case, seed)
    kind, n = case["kind"], len(FIELDS[case["physics"]])
    table = _eos_table() if case["eos"] == "table" else None
    opt = dict(physics=PHYSICS[case["physics"]], table=table, flux=FLUX[case["flux"]],
               eos=vah.VAH_EOS_TABLE if case["eos"] == "table" else vah.VAH_EOS_CONFORMAL,
               zeta=vah.VAH_ZETA_CROSSOVER if case["eos"] == "table" else vah.VAH_ZETA_REFERENCE)
    precision = vah.VAH_FP32 if case["precision"] == "fp32" else vah.VAH_FP64
    st = dict(case=case, e=e)
    if kind == "batch":
        st["batch"] = vah.Batch(capacity_bytes=40 << 30, precision=precision, **opt)
        st["sides"] = _sides(case)
        st["rows"] = _pinned(n, sum(x.size for x in e))
    else:
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        if kind in ("event", "host"):
            st["event"] = vah.Event(nx, ny, nz, case["dx"], case["dx"], case["dz"], ETA_S, t0=T_INIT,
                                    precision=precision, **opt)
        if kind == "event":
            st["rows"] = _pinned(n, e[0].size)
        if kind == "host":
            start = _start_arrays(case, torch.from_numpy(e[0]))
            st["start"] = start
            st["arrays"] = _pinned(*start.shape).copy_(start)
            ids = FIELDS[case["physics"]] + [22, 23, 24, 25]
            st["ptrs"] = [0] * vah.NUM_FIELDS
            for row, fid in enumerate(ids):
                st["ptrs"][fid] = st["arrays"][row].data_ptr()
            st["done"] = 0
        if kind == "buffers":
            st["stages"] = _stage_calls(case, e[0], table)
    if case["precision"] == "fp32" and "rows" in st:
        st["rows32"] = _pinned(*st["rows"].shape, dtype=torch.float32)
    return st


def _start_arrays(case, e):
    """The ghosted host arrays of a fresh event (conserved fields, e, p, u, previous u) at T_INIT, with u at rest
    and no viscous stress."""
    nq = NQ[case["physics"]]
    p = _pressure(case, e)
    pl = 0.0154483 * e if case["pl"] == "reference" else p
    rows = torch.zeros(nq + 10, *e.shape, dtype=torch.float64, device=e.device)
    rows[0], rows[4], rows[nq], rows[nq + 1], rows[nq + 2], rows[nq + 6] = e, pl, e, p, 1.0, 1.0
    return _ghosted(rows, 2, True).contiguous()


def _stage_calls(case, e, table):
    """The two stage calls of one step on device buffers: q0, e0, u0 -> stage 1 -> stage 2 -> the new state."""
    nq = NQ[case["physics"]]
    first = _start_arrays(case, torch.from_numpy(e)).cuda()
    mid, out = torch.zeros_like(first), torch.zeros_like(first)
    keep = dict(first=first, mid=mid, out=out)
    if table is not None:
        keep["table"] = torch.from_numpy(table).cuda()
    D = ctypes.c_void_p

    class Buffers(ctypes.Structure):
        _fields_ = [("q", D * 16), ("u", D * 4), ("u_prev", D * 4), ("e", D), ("p", D), ("q_avg", D * 16),
                    ("q_out", D * 16), ("u_out", D * 4), ("e_out", D), ("p_out", D)]

    def fill(src, prev, prev_row, avg, dst):
        b = Buffers()
        for m in range(nq):
            b.q[m], b.q_out[m] = src[m].data_ptr(), dst[m].data_ptr()
            if avg is not None:
                b.q_avg[m] = avg[m].data_ptr()
        b.e, b.p, b.e_out, b.p_out = (t.data_ptr() for t in (src[nq], src[nq + 1], dst[nq], dst[nq + 1]))
        for m in range(4):
            b.u[m], b.u_out[m] = src[nq + 2 + m].data_ptr(), dst[nq + 2 + m].data_ptr()
            b.u_prev[m] = prev[prev_row + m].data_ptr()
        return b

    L = vah.library()
    d = ctypes.c_double
    L.vah_stage_noalloc.argtypes = [ctypes.POINTER(vah.Lattice), d, ctypes.c_int, ctypes.c_int, ctypes.c_int, D,
                                    ctypes.c_int, d, d, D, D, D]
    keep["buffers"] = [fill(first, first, nq + 6, None, mid), fill(mid, first, nq + 2, first, out)]
    lat = vah.Lattice(case["nx"], case["ny"], case["nz"], case["dx"], case["dx"], case["dz"])
    tab = keep["table"].data_ptr() if table is not None else None
    torch.cuda.synchronize()

    def step():
        s = torch.cuda.current_stream().cuda_stream
        for k, b in enumerate(keep["buffers"]):
            vah.check(L.vah_stage_noalloc(ctypes.byref(lat), ETA_S, PHYSICS[case["physics"]],
                                          1 if table is not None else 0, 1 if table is not None else 0, tab, k + 1,
                                          T_INIT, case["dt"], ctypes.byref(b), s, None), "vah_stage_noalloc")

    keep["step"] = step
    keep["view"] = out[:nq + 6, 2:-2, 2:-2, 2:-2]
    return keep


def run(st):
    case = st["case"]
    kind, fields = case["kind"], FIELDS[case["physics"]]
    if kind == "buffers":
        st["stages"]["step"]()
        return _groups(case, st["stages"]["view"])
    if kind == "host":
        if st["done"] == HOST_RESTART:
            st["arrays"].copy_(st["start"])
            st["done"] = 0
        st["event"].step_host(T_INIT + st["done"] * case["dt"], case["dt"], st["ptrs"])
        st["done"] += 1
        return _groups(case, st["arrays"][:len(fields), 2:-2, 2:-2, 2:-2])
    rows = st["rows"]
    if kind == "event":
        ev = st["event"]
        ev.init_from_e(T_INIT, st["e"][0], _pl_mode(case))
        ev.run(T_INIT, case["dt"], case["steps"])
        for row, fid in enumerate(fields):
            vah.check(ev.L.vah_event_get_field(ev.ev, fid, _address(rows[row]), 0), "vah_event_get_field")
    else:
        b = st["batch"]
        slots = [b.add(nx, ny, nz, case["dx"], case["dx"], case["dz"], T_INIT, case["dt"], ETA_S, e, _pl_mode(case))
                 for (nx, ny, nz), e in zip(st["sides"], st["e"])]
        b.step(case["steps"])
        at = 0
        for slot, e in zip(slots, st["e"]):
            for row, fid in enumerate(fields):
                vah.check(b.L.vah_batch_get_field(b.b, slot, fid, _address(rows[row, at:]), 0), "vah_batch_get_field")
            at += e.size
        for slot in slots:
            b.remove(slot)
    if case["precision"] == "fp32":  # the form's own width
        rows = st["rows32"].copy_(rows)
    return _groups(case, rows)


# ------------------------------------------------------------------ exact --
# The scheme in torch, FP64, over whole lattices: (B, ny, nx) for boost-invariant events of one size (B of them),
# (nz, ny, nx) for a 3+1D event.
# numerator and denominator coefficients (constant term first) of the closures' rational fits in a = P_L / e
FITS = {
    "Rtilde": (
        [-6.674731906076046e-6, 0.004617789933500251, 0.7207562721999754, 9.097427250602184, -4.475814747302824,
         -36.37501529319408, 46.868405146729316, -15.833867583743228],
        [0.06856675185266, 2.9181587012768597, 11.951184087839218, -29.708257843442173, -2.618233802059826,
         34.646239784689065, -19.62596366454439, 2.374808442453899],
    ),
    "Rhat": (
        [0.0024792827625583747, 1.943027171680747, 53.46970495217282, 19.989171951866325, -347.1285593126723,
         412.2647882672885, -140.53693383827797],
        [0.5061402347582388, 29.466067530916984, 126.07947638942892, -334.420268508072, 86.57706367583984,
         183.53625188578846, -91.68259808111912],
    ),
    "Rbar0": (
        [0.015267955823446243, 7.725572805021035, 421.0063884634789, 3422.877939650926, -5785.670846299543,
         -12261.66452089229, 31491.409484673808, -22737.05146992673, 5441.373392185447],
        [0.05470696094814806, 14.505878005231883, 522.6643024173569, 2731.7776413939037, -6161.1991042880445,
         -3989.4375208972588, 15008.260526258282, -10243.036679405379, 2116.74060159494],
    ),
    "Rgamma": (
        [0.0001373796340585521, -0.6149634004722385, 3.1968875683514253, 246.35973783799196, -764.319750320186,
         834.160165071214, -371.64955466673234, 52.87411921963021],
        [-1.673322188488071, 13.343782941396997, 561.7566534476223, -1790.2296622275915, 1896.4688704912812,
         -658.7933063369629, -85.96181900698849, 65.09739194472589],
    ),
    "Rbar0P": (
        [2.473173363908116e-10, -4.899839370307281e-6, -0.004301975027942015, -0.14858206981041563,
         6.249255189587875, -92.79641927240235, 807.175057749925, -4760.015905266286, 20324.533122685436,
         -64758.869552496515, 155055.91462124084, -275435.45350226434, 350689.68825705117, -299725.38986957155,
         151477.08809203724, -33196.47417939176],
        [0.00008222793468208523, 0.03411917870833943, 0.23871740573818725, -23.50912574236691,
         417.4953123877312, -4234.215775452717, 29824.022790048104, -157419.8447785501, 641300.6529027821,
         -2.0248032895288002e6, 4.895969276094396e6, -8.84162305829353e6, 1.1445063656613324e7,
         -9.918442713390596e6, 5.065882388219598e6, -1.1181016364928822e6],
    ),
    "g0m2040DividedBym2ConstantTerm": (
        [0.0002022034619596147, -0.3465776971894224, -0.46483928190644463, 305.8182449301262,
         -3094.0393881108607, 13530.068145958274, -33008.96608710712, 47814.11155495329, -40754.13233671886,
         18877.099618956072, -3669.180338013278],
        [0.3231726678495768, 6.510257837715722, -66.42749605402405, 278.2072846508577, -659.8881404723605,
         1009.6856692105162, -1129.2454150937733, 1136.3819011323233, -1029.3638914685152, 600.4581631072344,
         -146.6399433638468],
    ),
    "g0m2040DividedBym2Zm2Term": (
        [-5.428668780471906e-6, 0.07087180484499124, -3.6056344041371626, -75.98232257237731, 314.3389560219402,
         -4860.077726215435, 28903.651438438494, -74655.13722955724, 95355.62148623986, -59409.22212071206,
         14430.23620485441],
        [0.06525900311126431, 1.7911514139670908, -1.0324279865217276, 81.69891535142081, -259.5916250456495,
         -59.79985417459323, 2029.823700195329, -4622.384249181224, 4479.931023062334, -1935.0883554632262,
         284.5874952982027],
    ),
    "g0m2040DividedBym2LogZTerm": (
        [1.5260366926367532e-7, -0.00024895619154304205, -0.0027342593291142404, 0.20899592202076162,
         -2.1908540237701564, 10.836996467643049, -31.053876569731955, 55.16397490084364, -61.60172864783581,
         42.08494163892432, -16.08135726710075, 2.635895081202281],
        [0.0000605632612588605, 0.0012923594925415354, -0.016304038454467058, 0.07975759323101335,
         -0.21819092742589902, 0.37685396820303946, -0.45029351728017364, 0.44970998105242493,
         -0.44680890883509927, 0.3691002339464134, -0.18379144108413883, 0.038614228316574885],
    ),
    "g0m2020ConstantTerm": (
        [-0.000011732877574172216, 0.0008995982417255349, 0.7361757170685882, 8.855369493730423,
         -76.00475510029524, 261.7208147369771, -479.7229720410445, 487.6088140168412, -260.7802309619955,
         57.58861537142237],
        [-0.0001445869624012341, 0.03556951252765837, 3.2344009306364274, 12.514996006390815,
         -118.07971915906703, 347.32729764112844, -483.55235351080324, 310.7815908976544, -67.06626623263872,
         -5.19154598317511],
    ),
    "g0m2020Z2Term": (
        [-0.02907781069921067, -13.745970067614193, -325.2706635847172, 2604.8287335227815, -4049.1372422838062,
         -16667.365141623744, 83158.20010908133, -154605.3533428809, 147412.71289551136, -71512.66891762966,
         13997.84367889844],
        [0.9697656616566325, 117.19185209632286, 842.3723825380051, -5926.237511293323, 14247.062719381864,
         -16353.128301113404, 21213.272784815457, -46076.07167476786, 59110.92666130391, -34796.81744513102,
         7621.0452633237755],
    ),
    "g0m2020Z2LogZTerm": (
        [-0.0005534368375549849, -0.3080130050685187, -11.136413628061584, 34.63107256159966, 367.6376955018988,
         -2567.818354775122, 7178.293271719852, -10678.12443252271, 8758.211709132715, -3711.7083581405914,
         630.3245252759478],
        [0.009248889228618452, 1.4181948328169438, 21.503144137961534, -62.705284754794086, -83.17143447631213,
         693.6443740085989, -1134.2586687505138, 513.1520937342799, 331.751797652403, -376.7067817672707,
         95.39051233960058],
    ),
    "G_G1": (
        [0.000034723242182175396, 0.012572522745974798, 0.427982420164622, 1.3191165093454609,
         -5.616153984227332, 4.28680523098434, 1.5082210795675917, -2.6464367629253513, 0.707946904809862],
        [0.00017101953273167538, 0.030287072809487548, 0.5997230938576861, 0.3789662678043767,
         -5.429830325143101, 7.101821088278835, -1.968210179097073, -1.3532147373075232, 0.6402914643622666],
    ),
}


def _ghosted(a, n, along_eta):
    """`a` (..., z, y, x) with n zero-gradient ghost layers along x, y (and eta)."""
    for dim in (-1, -2) + ((-3,) if along_eta else ()):
        size = a.shape[dim]
        at = torch.arange(-n, size + n, device=a.device).clamp(0, size - 1)
        a = a.index_select(dim % a.dim(), at)
    return a


def _table_at(e):
    """(p, T, c_s^2) of the tabulated EoS: linear in ln e between nodes, power laws outside."""
    t = torch.from_numpy(_eos_table()).to(e.device)
    n = TABLE_N
    P, T, C = t[8:8 + n], t[8 + n:8 + 2 * n], t[8 + 2 * n:]
    x = torch.log(e.clamp_min(1e-300))
    f = (x - t[1]) * t[2]
    i = f.clamp(0, n - 2).long()
    w = f - i

    def lin(a):
        return a[i] + w * (a[i + 1] - a[i])

    low, high, neg = f <= 0, f >= n - 1, ~(e > 0)
    p = torch.where(high, e * (P[-1] / t[6]), torch.where(low | neg, e * (P[0] / t[4]), lin(P)))
    Tv = torch.where(high, T[-1] * torch.exp(0.25 * (x - t[5])), torch.where(low, T[0] * torch.exp(3 / 23 * (x - t[1])), lin(T)))
    c = torch.where(high, C[-1], torch.where(low | neg, C[0], lin(C)))
    return p, torch.where(neg, torch.zeros_like(Tv), Tv), c


def _pressure(case, e):
    return e / 3.0 if case["eos"] == "conformal" else _table_at(e)[0]


def _fit(name, a):
    num, den = FITS[name]

    def poly(c):
        v = torch.full_like(a, c[-1])
        for x in c[-2::-1]:
            v = v * a + x
        return v

    return poly(num) / poly(den)


def _setup(nq, t, q):
    """The guess-independent part of the inversion of conserved values q (N_q first)."""
    z = torch.zeros_like(q[0])
    pi = q[5:9] if nq >= 15 else (z, z, z, z)
    bulk = q[15] if nq == 16 else z
    pl = q[4]
    m0, m1, m2, m3 = q[0] - pi[0], q[1] - pi[1], q[2] - pi[2], q[3] - pi[3]
    d = m0 + pl
    F = m3 / torch.where(d == 0, torch.full_like(d, 1e-16), d)
    Ft2 = (t * F) ** 2
    x = torch.sqrt(torch.abs(1 - Ft2))
    mbt = torch.sqrt(m1 * m1 + m2 * m2)
    mbt = torch.where(mbt == 0, torch.full_like(mbt, 1e-16), mbt)
    bL, b, c0 = x * x * m0 - Ft2 * pl, x * x + Ft2, m0 - t * t * F * m3
    return dict(m1=m1, m2=m2, F=F, x=x, mbt=mbt, bT=x * mbt, bL=bL, b=b, c0=c0, pl=pl, bulk=bulk)


def _newton(s, guess):
    """Newton's iteration on u_T to 1e-7: (u_T, converged)."""
    w = guess.clone()
    ok, going = torch.zeros_like(w, dtype=torch.bool), torch.ones_like(w, dtype=torch.bool)
    for _ in range(200):
        r = 1 / torch.sqrt(1 + w * w)
        v = w * r
        e = s["c0"] - v * s["x"] * s["mbt"]
        g = s["bL"] + s["b"] * (0.5 * (e - s["pl"]) + 1.5 * s["bulk"])
        r3 = r * r * r
        fp = r3 * g - 0.5 * v * s["b"] * s["bT"] * r3
        fp = torch.where(fp == 0, torch.full_like(fp, 1e-16), fp)
        nxt = w - (v * g - s["bT"]) / fp
        fine = (e >= 0) & (nxt >= 0) & (nxt <= 9.0072e15)
        near = (nxt - w).abs() <= 1e-7 * nxt.abs()
        w = torch.where(going & fine, nxt, w)
        ok |= going & fine & near
        going &= fine & ~near
        if not bool(going.any()):
            break
    return w, ok


def _minmod(x, y, z):
    l, r, c = 1.1 * (y - x), 1.1 * (z - y), 0.5 * (z - x)
    m = torch.minimum(torch.minimum(l.abs(), r.abs()), c.abs())
    neg = l < 0
    return torch.where(neg == (r < 0), torch.where(neg, -m, m), torch.zeros_like(m))


def _axis_flux(nq, t, q, e, ut, axis):
    """H(-1/2) - H(+1/2) of every cell along one axis: q, e, u_T with two ghost layers along it, each face
    evaluated as the cell on either side of it does."""
    dim = {0: -1, 1: -2, 2: -3}[axis]
    n = q.shape[dim] - 4

    def cut(a, at, m):
        return a.narrow(dim, at, m)

    slope = _minmod(cut(q, 0, n + 2), cut(q, 1, n + 2), cut(q, 2, n + 2))  # of cells 1 .. n + 2
    qL = cut(q, 1, n + 1) + 0.5 * cut(slope, 0, n + 1)
    qR = cut(q, 2, n + 1) - 0.5 * cut(slope, 1, n + 1)
    states = [(_setup(nq, t, s), s) for s in (qR, qL)]
    H = []
    for at in (1, 2):  # the left cell's guess, the right cell's
        guess = cut(ut, at, n + 1)
        vel = []
        for s, _ in states:
            w, ok = _newton(s, guess)
            v = s["F"] if axis == 2 else w * (s["m1"] if axis == 0 else s["m2"]) * s["x"] / (torch.sqrt(1 + w * w) * s["mbt"])
            vel.append(torch.where(ok, v, torch.zeros_like(v)))
        a = torch.maximum(vel[0].abs(), vel[1].abs())
        H.append(0.5 * ((vel[0] - a) * qR + (vel[1] + a) * qL))
    return cut(H[1], 0, n) - cut(H[0], 1, n)


def _sources(case, nq, t, dt, q, e, p, u, up, grad):
    """The local sources S (SourceTerms of the scheme, W off) as rows."""
    shear, bulk = nq >= 15, nq == 16
    z = torch.zeros_like(e)
    ttt, ttx, tty, ttn, pl = q[0:5]
    pitt, pitx, pity, pitn, pixx, pixy, pixn, piyy, piyn, pinn = q[5:15] if shear else (z,) * 10
    Pi = q[15] if bulk else z
    ut, ux, uy, un = u
    (dxut, dxux, dxuy, dxun), (dyut, dyux, dyuy, dyun), (dnut, dnux, dnuy, dnun) = (g["u"] for g in grad)
    (dxe, dye, dne), (dxp, dyp, dnp), (dxpl, dypl, dnpl) = ([g[k] for g in grad] for k in ("e", "p", "pl"))
    vx, vy, vn = ux / ut, uy / ut, un / ut
    dkvk = (dxux - vx * dxut + dyuy - vy * dyut + dnun - vn * dnut) / ut
    t2 = t * t
    dtut, dtux, dtuy, dtun = (ut - up[0]) / dt, (ux - up[1]) / dt, (uy - up[2]) / dt, (un - up[3]) / dt

    def along(a, b, c, d):
        return ut * a + ux * b + uy * c + un * d

    dut, dux = along(dtut, dxut, dyut, dnut), along(dtux, dxux, dyux, dnux)
    duy, dun = along(dtuy, dxuy, dyuy, dnuy), along(dtun, dxun, dyun, dnun)
    Dut, Dux, Duy, Dun = dut + t * un * un, -dux, -duy, -t2 * (dun + 2 * ut * un / t)
    theta = ut / t + dtut + dxux + dyuy + dnun
    th = theta / 3
    stt = -t * ut * un * un + (dtut - ut * dut) + (ut * ut - 1) * th
    stx = -t * un * un * ux / 2 + (dtux - dxut) / 2 - (ux * dut + ut * dux) / 2 + ut * ux * th
    sty = -t * un * un * uy / 2 + (dtuy - dyut) / 2 - (uy * dut + ut * duy) / 2 + ut * uy * th
    stn = -un * (2 * ut * ut + t2 * un * un) / (2 * t) + (dtun - dnut / t2) / 2 - (un * dut + ut * dun) / 2 + ut * un * th
    sxx = -(dxux + ux * dux) + (1 + ux * ux) * th
    sxy = -(dxuy + dyux) / 2 - (uy * dux + ux * duy) / 2 + ux * uy * th
    sxn = -ut * ux * un / t - (dxun + dnux / t2) / 2 - (un * dux + ux * dun) / 2 + ux * un * th
    syy = -(dyuy + uy * duy) + (1 + uy * uy) * th
    syn = -ut * uy * un / t - (dyun + dnuy / t2) / 2 - (un * duy + uy * dun) / 2 + uy * un * th
    snn = -ut * (1 + 2 * t2 * un * un) / t ** 3 - dnun / t2 - un * dun + (1 / t2 + un * un) * th
    F = 1 + ux * ux + uy * uy
    sF = torch.sqrt(F)
    uTdx, uTdy, uTdn = ux * dxux + uy * dxuy, ux * dyux + uy * dyuy, ux * dnux + uy * dnuy
    uTd = ut * (ux * dtux + uy * dtuy) + ux * uTdx + uy * uTdy + un * uTdn
    z0, z3 = t * un / sF, ut / t / sF
    dz0 = (ut * un + t * dun - t * un / F * uTd) / sF
    dz3 = (-ut * ut / t2 + dut / t - ut / t / F * uTd) / sF
    Dz0, Dz3 = dz0 + t * un * z3, -t2 * (dz3 + (ut * z3 + un * z0) / t)
    A = z0 * z0 * stt - 2 * t2 * z0 * z3 * stn + t2 * t2 * z3 * z3 * snn
    B0, B1, B2, B3 = (z0 * a - t2 * z3 * b for a, b in ((stt, stn), (stx, sxn), (sty, syn), (stn, snn)))
    thT = 2 * th + A
    zDzu = theta - thT
    sttT = stt + 2 * z0 * B0 + z0 * z0 * A - (1 - ut * ut + z0 * z0) * A / 2
    stxT, styT = stx + z0 * B1 + ut * ux * A / 2, sty + z0 * B2 + ut * uy * A / 2
    stnT = stn + z0 * B3 + z3 * B0 + z0 * z3 * A - (-ut * un + z0 * z3) * A / 2
    sxxT, sxyT, syyT = sxx + (1 + ux * ux) * A / 2, sxy + ux * uy * A / 2, syy + (1 + uy * uy) * A / 2
    sxnT, synT = sxn + z3 * B1 + ux * un * A / 2, syn + z3 * B2 + uy * un * A / 2
    snnT = snn + 2 * z3 * B3 + z3 * z3 * A - (-1 / t2 - un * un + z3 * z3) * A / 2

    e = torch.where(e == 0, torch.full_like(e, 1e-7), e)
    if case["eos"] == "conformal":
        T, cs2 = (e / EOS_FACTOR) ** 0.25, z
    else:
        _, T, cs2 = _table_at(e)
    a = pl / e
    Rtilde, Rbar0, Rgamma, Rbar0P = (_fit(k, a) for k in ("Rtilde", "Rbar0", "Rgamma", "Rbar0P"))
    e3p = e - 3 * p
    ptHat = (e - pl - Rbar0 * e3p) / 2
    pt = ptHat + 1.5 * Pi
    DP = pl - pt
    Ltt, Ltn, Lnn = DP * t2 * un * un / F, DP * ut * un / F, DP * ut * ut / F / t2
    tnn = (e + pt) * un * un + pt / t2 + Lnn + pinn

    def grads(de, dp, dpl):
        dpt = (de - dpl - Rbar0 * (de - 3 * dp) - e3p * Rbar0P * (dpl - a * de) / e) / 2
        return dpt, dpl - dpt

    dxpt, dxDP = grads(dxe, dxp, dxpl)
    dypt, dyDP = grads(dye, dyp, dypl)
    dnpt, dnDP = grads(dne, dnp, dnpl)

    def dL(kind, dDP, dut_, dun_, uTdi):
        if kind == "tt":
            return t2 * (2 * DP * dun_ * un / F + dDP * un * un / F - 2 * DP * uTdi * un * un / F ** 2)
        if kind == "tn":
            return DP * dut_ * un / F + DP * dun_ * ut / F + dDP * un * ut / F - 2 * DP * uTdi * un * ut / F ** 2
        return (2 * DP * dut_ * ut / F + dDP * ut * ut / F - 2 * DP * uTdi * ut * ut / F ** 2) / t2

    ax = ((dxDP, dxut, dxun, uTdx), (dyDP, dyut, dyun, uTdy), (dnDP, dnut, dnun, uTdn))
    dxLtt, dyLtt, dnLtt = (dL("tt", *k) for k in ax)
    dxLtn, dyLtn, dnLtn = (dL("tn", *k) for k in ax)
    dnLnn = dL("nn", *ax[2])
    zzz, zzT = Rtilde * e - 3 * pl, (Rtilde * e + pl) / 2
    dpipi = (3 + Rgamma) / 2
    tpipi, lpipi, tauinv = 4 * dpipi / 3, Rgamma - 1, 0.2 * T / ETA_S
    psT = (pitt * sttT - 2 * pitx * stxT - 2 * pity * styT + pixx * sxxT + 2 * pixy * sxyT + piyy * syyT
           - 2 * t2 * (pitn * stnT - pixn * sxnT - piyn * synT) + t2 * t2 * pinn * snnT)
    S = torch.zeros_like(q)
    dPL = -(pl - p) * tauinv + zzz * zDzu - zzT * thT - Rgamma * psT
    if bulk:
        third = 1 / 3 - cs2
        m2 = 36 * torch.where(third == 0, torch.full_like(third, 1e-16), third)
        zl = -2 * (1 + 0.02536 * m2)
        g40 = ((_fit("g0m2040DividedBym2LogZTerm", a) * zl + _fit("g0m2040DividedBym2Zm2Term", a)) / m2
               + _fit("g0m2040DividedBym2ConstantTerm", a))
        g20c = _fit("g0m2020ConstantTerm", a)
        g20 = g20c + _fit("g0m2020Z2LogZTerm", a) * zl + _fit("g0m2020Z2Term", a) * m2
        dPL = dPL - 3 * g40 * Pi * zDzu - (g20 + g40) * Pi * thT
        Rhat = _fit("Rhat", a)
        x = (T - 0.155 / HBARC) / (0.050 / HBARC)  # the crossover zeta/s: 0.05 at 155 MeV, half-width 50 MeV
        tauPiinv = 15 * third * third * T / (0.05 / (1 + x * x))
        dPi = (-((1 - Rbar0) * e3p / 3 + Pi) * tauPiinv - (Rhat - Rbar0) * e3p / 3 * zDzu + (Rbar0 + Rhat) * e3p / 6 * thT
               - (1 - g20c) * Pi * zDzu - (1 + g20c) / 2 * Pi * thT - 3 * _fit("G_G1", a) / 5 * cs2 * psT)
        S[15] = dPi / ut + Pi * dkvk
    S[4] = dPL / ut + dkvk * pl
    S[0] = (-(ttt / t + t * tnn) + dkvk * (Ltt + pitt - pt) - vx * dxpt - vy * dypt - vn * dnpt + vx * dxLtt + vy * dyLtt
            + vn * dnLtt - dnLtn)
    S[1] = -ttx / t - dxpt + dkvk * pitx
    S[2] = -tty / t - dypt + dkvk * pity
    S[3] = -3 * ttn / t - dnpt / t2 + dkvk * (Ltn + pitn) + vx * dxLtn + vy * dyLtn + 2 * vn * dnLtn - dnLnn
    if shear:
        U, D, Z, DZ = (ut, ux, uy, un), (Dut, Dux, Duy, Dun), (z0, z, z, z3), (Dz0, z, z, Dz3)
        pi = ((pitt, pitx, pity, pitn), (pitx, pixx, pixy, pixn), (pity, pixy, piyy, piyn), (pitn, pixn, piyn, pinn))
        sg = ((sttT, stxT, styT, stnT), (stxT, sxxT, sxyT, sxnT), (styT, sxyT, syyT, synT), (stnT, sxnT, synT, snnT))
        g = (1.0, -1.0, -1.0, -t2)
        delta = {(0, 0): 1.0, (1, 1): -1.0, (2, 2): -1.0, (3, 3): -1.0 / t2}
        two_eta = ((3 - Rtilde) * e - 2 * pl) / 4
        c2 = dpipi * thT + lpipi * zDzu
        # the connection terms of d_tau pi along the flow
        conn = {(0, 0): 2 * un * t * pitn, (0, 1): un * t * pixn, (0, 2): un * t * piyn,
                (0, 3): un * t * pinn + (ut * pitn + un * pitt) / t, (1, 3): (ut * pixn + un * pitx) / t,
                (2, 3): (ut * piyn + un * pity) / t, (3, 3): 2 * (ut * pinn + un * pitn) / t}
        row = 5
        for m in range(4):
            for k in range(m, 4):
                I1 = sum((pi[m][l] * U[k] + pi[k][l] * U[m]) * D[l] for l in range(4))
                # the z-parts as the scheme has them: pi^{t..} Dz0 and pi^{n..} Dz3; its t x and t y components
                # take the second one's first factor from u
                zm, zk = Z[m], Z[k]
                if (m, k) in ((0, 1), (0, 2)):
                    I1 = I1 - ((pi[k][0] * zm) * Dz0 + (pitn * U[k] + pi[k][3] * zm) * Dz3)
                else:
                    I1 = I1 - ((pi[m][0] * zk + pi[k][0] * zm) * Dz0 + (pi[m][3] * zk + pi[k][3] * zm) * Dz3)
                I4 = sum(g[l] * (pi[m][l] * sg[k][l] + pi[k][l] * sg[m][l]) for l in range(4)) / 2
                I4 = I4 - (delta.get((m, k), 0.0) - U[m] * U[k] + zm * zk) * psT / 2
                d = two_eta * sg[m][k] - pi[m][k] * tauinv - (I1 - c2 * pi[m][k] + tpipi * I4)
                if (m, k) in conn:
                    d = d - conn[(m, k)]
                S[row] = d / ut + pi[m][k] * dkvk
                row += 1
    return S


def _regulate(nq, t, e, p, q, u):
    low = e < 0
    e, p = torch.where(low, torch.full_like(e, 1e-7), e), torch.where(low, torch.full_like(p, 1e-7), p)
    q[4] = torch.where(q[4] < 0, torch.full_like(e, 1e-7), q[4])
    if nq == 5:
        return e, p, q
    pl, t2 = q[4], t * t
    ptHat = (e - pl - _fit("Rbar0", pl / e) * (e - 3 * p)) / 2
    tt, tx, ty, tn, xx, xy, xn, yy, yn, nn = q[5:15]
    ut, ux, uy, un = u
    sF = torch.sqrt(1 + ux * ux + uy * uy)
    z0, z3 = t * un / sF, ut / t / sF
    pipi = (tt * tt - 2 * tx * tx - 2 * ty * ty + xx * xx + 2 * xy * xy + yy * yy - 2 * t2 * (tn * tn - xn * xn - yn * yn)
            + nn * nn * t2 * t2)
    s = torch.sqrt(pipi.abs())
    rho = s / torch.sqrt((e * e + pl * pl + 2 * ptHat * ptHat).abs())
    num = torch.stack([tt - xx - yy - nn * t2, -tn * t2 * un + tt * ut - tx * ux - ty * uy,
                       -xn * t2 * un + tx * ut - xx * ux - xy * uy, -yn * t2 * un + ty * ut - xy * ux - yy * uy,
                       -nn * t2 * un + tn * ut - xn * ux - yn * uy, z0 * tt - t2 * z3 * tn, z0 * tx - t2 * z3 * xn,
                       z0 * ty - t2 * z3 * yn, z0 * tn - t2 * z3 * nn]) / s
    rho = torch.maximum(rho, torch.nan_to_num(num, nan=-math.inf, posinf=math.inf, neginf=-math.inf).amax(0))
    fac = torch.where(rho < 1e-7, torch.ones_like(rho), torch.tanh(rho) / rho)
    q[5:15] = q[5:15] * fac
    return e, p, q


def _stage(case, nq, t, t_inv, dt, along_eta, q, e, p, u, up, guess, avg):
    """One RK stage: conserved q, e, p, u in (up: the stage before's u), the same out."""
    g2 = _ghosted(torch.cat([q, e[None], p[None], u]), 2, along_eta)
    h = (case["dx"], case["dx"], case["dz"])
    axes = 3 if along_eta else 2

    def inner(a, skip=None):
        """The interior along all axes but `skip` (which keeps its ghosts)."""
        for dim, axis in ((-1, 0), (-2, 1), (-3, 2)):
            if axis != skip and (axis < 2 or along_eta):
                a = a.narrow(dim, 2, a.shape[dim] - 4)
        return a

    grad, flux, axis_src = [], torch.zeros_like(q), torch.zeros_like(q[:4])
    for axis in range(3):
        if axis >= axes:
            z = torch.zeros_like(e)
            grad.append(dict(u=(z, z, z, z), e=z, p=z, pl=z))
            continue
        a = inner(g2, axis)
        dim = {0: -1, 1: -2, 2: -3}[axis]
        n = a.shape[dim] - 4
        d = (a.narrow(dim, 3, n) - a.narrow(dim, 1, n)) / h[axis] / 2
        grad.append(dict(u=d[nq + 2:nq + 6], e=d[nq], p=d[nq + 1], pl=d[4]))
        uT = torch.sqrt(a[nq + 3] ** 2 + a[nq + 4] ** 2)
        flux += dt / h[axis] * _axis_flux(nq, t, a[:nq], a[nq], uT, axis)
        if nq >= 15:
            v = u[1 + axis] / u[0]
            rows = {0: (6, 9, 10, 11), 1: (7, 10, 12, 13), 2: (8, 11, 13, 14)}[axis]
            for k in range(4):
                axis_src[k] += d[5 + k] * v - d[rows[k]]
            if nq == 16:
                axis_src[0] -= v * 1.5 * d[15]
                axis_src[1 + axis] -= 1.5 * d[15] / (t * t if axis == 2 else 1.0)
    new = q + dt * _sources(case, nq, t, dt, q, e, p, u, up, grad) + flux
    new[:4] += dt * axis_src
    if avg is not None:
        new = (new + avg) / 2
    s = _setup(nq, t_inv, new)
    w, ok = _newton(s, torch.sqrt(guess[1] ** 2 + guess[2] ** 2))
    C = torch.sqrt(1 + w * w)
    one, zero = torch.ones_like(w), torch.zeros_like(w)
    e2 = torch.where(ok, s["c0"] - w / C * s["x"] * s["mbt"], 0.999 * e)
    u2 = torch.stack([torch.where(ok, C / s["x"], one), torch.where(ok, w * s["m1"] / s["mbt"], zero),
                      torch.where(ok, w * s["m2"] / s["mbt"], zero), torch.where(ok, s["F"] * C / s["x"], zero)])
    p2 = _pressure(case, e2)
    e2, p2, new = _regulate(nq, t_inv, e2, p2, new, u2)
    return new, e2, p2, u2


def _simulate(case, e, steps):
    """`steps` RK2 steps from the energy densities e (z or event, y, x): the state's rows."""
    nq, along_eta = NQ[case["physics"]], case["nz"] > 1
    p = _pressure(case, e)
    q = torch.zeros(nq, *e.shape, dtype=torch.float64, device=e.device)
    q[0], q[4] = e, 0.0154483 * e if case["pl"] == "reference" else p
    u = torch.zeros(4, *e.shape, dtype=torch.float64, device=e.device)
    u[0] = 1.0
    up, dt = u, case["dt"]
    for k in range(steps):
        t = T_INIT + k * dt
        q1, e1, p1, u1 = _stage(case, nq, t, t + dt, dt, along_eta, q, e, p, u, up, u, None)
        q2, e2, p2, u2 = _stage(case, nq, t + dt, t + dt, dt, along_eta, q1, e1, p1, u1, u, u, q)
        q, e, p, u, up = q2, e2, p2, u2, u
    return torch.cat([q, e[None], p[None], u])


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    fields = [torch.from_numpy(x).to(dev) for x in _inputs(case, seed)]
    if case["kind"] != "batch":
        rows = _simulate(case, fields[0], case["steps"])
        return _groups(case, rows if case["kind"] in ("host", "buffers") else rows.flatten(1))
    if case["nz"] > 1:
        return _groups(case, torch.cat([_simulate(case, e, case["steps"]).flatten(1) for e in fields], 1))
    parts = [None] * len(fields)
    for shape in {e.shape for e in fields}:  # events of one size at once
        same = [k for k, e in enumerate(fields) if e.shape == shape]
        rows = _simulate(case, torch.cat([fields[k] for k in same]), case["steps"])
        for at, k in enumerate(same):
            parts[k] = rows[:, at].flatten(1)
    return _groups(case, torch.cat(parts, 1))
