"""What is timed: the calls that a user of this framework makes, over the sizes they come in.

A case is a dict of plain values. Flashes (calibration): one through the drop-in
``transport`` call, an uneven served batch through ``run``, a full stream through
``launch`` on resident buffers, and a broadband batch. Showers: the stages of the
route through their own entry points (order 0, the coarse and the fine order 1,
the order >=2 source compile and contraction), then one shower and a served batch
through ``ShowerTransport``. Sizes are those of the tests and the benchmark: 48 and
384 OMs, 500-50000 elements per shower (log-uniform, 0.15 m of charged track per
element), flash batches of 1-256 and streams of 4096.

Tables, transports and routes are made once per process and kept, as a serving
program keeps them; inputs are made from the seed. Showers start at least 6 m away
from every OM (closer ones take the rare near-field clamp).
"""
import functools
import math
from pathlib import Path

import numpy as np
import torch

from lighthit_b200.flash import BroadbandFlashTransport, FlashTable, FlashTransport
from lighthit_b200.ge2 import AxialSources
from lighthit_b200.model import IsotropicFlash, KernelConfig, synthetic_detector
from lighthit_b200.order0 import ElementBatch, order0
from lighthit_b200.order1 import grouped_widening, pencils
from lighthit_b200.shower import ShowerTables, ShowerTransport

TABLES = Path(__file__).resolve().parent.parent / "lighthit_b200" / "tables"
C_M_PER_NS = 0.299792458
FLASH_TABLES = {411.27: "flash_411.27nm_2-250m.npz", 450.0: "flash_450nm_2-250m.npz",
                488.73: "flash_488.73nm_2-250m.npz"}
SOURCE_ROWS = 200  # rows of a kept source buffer: at most 5 x 37 slices of a 7.2 m shower
FLASH_PAIR_BYTES = 65 * 3 * 8 + 3 * 160 * 4 + 3 * 8 + 8 + 1  # outputs of one (flash, OM)
OMS = {"c0": 48, "c2": 384, "c3": 384}


def listed():
    return [
        # one calibration flash, read back as a response: latency
        dict(name="flash-one", kind="flash", call="transport", flashes=1, mode="split-bf16"),
        # an uneven batch of a flash server
        dict(name="flash-few", kind="flash", call="run", flashes=137, mode="split-bf16"),
        # the calibration stream on resident buffers: the largest flash call
        dict(name="flash-stream", kind="flash", call="launch", flashes=4096, mode="split-bf16"),
        # flashes with a spectral shape: three wavelength nodes and their sum
        dict(name="flash-broadband", kind="flash", call="broadband", flashes=501,
             mode="split-bf16"),
        # direct light of one ordinary shower on the small array
        dict(name="order0-one", kind="order0", tables="c0", showers=1, low=2000, high=2000),
        # direct light of a served batch, with the error estimate
        dict(name="order0-batch", kind="order0", tables="c2", showers=8, low=500, high=50000),
        # the coarse order-1 charge of every OM of the large array
        dict(name="order1-screen", kind="order1", tables="c2", elements=20011, oms=384,
             coarse=True),
        # order 1 at full resolution at the OMs around a median shower
        dict(name="order1-fine", kind="order1", tables="c2", elements=6637, oms=64,
             coarse=False),
        # the order >=2 sources of a median shower
        dict(name="sources", kind="sources", tables="c2", elements=6637),
        # order >=2 spectra of a served batch's active OMs
        dict(name="spectra", kind="spectra", tables="c2", showers=8, elements=2003, oms=48,
             mode="split-bf16"),
        # one shower on the small array, start to response: latency
        dict(name="shower-one", kind="shower", tables="c0", showers=1, low=2000, high=2000),
        # a served batch on the large array, host elements to responses
        dict(name="shower-batch", kind="shower", tables="c2", showers=8, low=500, high=50000),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["flash", "flash", "order0", "order1", "order1", "sources", "spectra",
                       "shower"])
    if kind == "flash":
        call = rng.choice(["transport", "run", "launch", "broadband"])
        top = {"transport": 1, "run": 256, "launch": 4000, "broadband": 500}[call]
        mode = "split-bf16" if call == "broadband" else rng.choice(["split-bf16", "bf16", "fp32"])
        return dict(kind=kind, call=call, flashes=_log_uniform(rng, 1, top), mode=mode)
    tables = rng.choice(["c0", "c2"])
    if kind in ("order0", "shower"):
        showers = rng.randint(1, 8)
        low = _log_uniform(rng, 500, 5000)
        return dict(kind=kind, tables=tables, showers=showers, low=low,
                    high=low if showers == 1 else _log_uniform(rng, low, 40000))
    elements = _log_uniform(rng, 500, 50000)
    if kind == "order1":
        coarse = rng.random() < 0.5
        most = OMS[tables] if coarse else min(OMS[tables], 96)
        return dict(kind=kind, tables=tables, elements=elements, oms=rng.randint(5, most),
                    coarse=coarse)
    tables = rng.choice(["c0", "c2", "c3"])
    if kind == "sources":
        return dict(kind=kind, tables=tables, elements=elements)
    return dict(kind=kind, tables=tables, showers=rng.randint(1, 3 if tables == "c3" else 8),
                elements=_log_uniform(rng, 500, 5000), oms=rng.randint(3, 48),
                mode=rng.choice(["split-bf16", "split-bf16", "bf16", "fp32"]))


# ---------------------------------------------------------------- what a program keeps

@functools.lru_cache(maxsize=None)
def _tables(name):
    return ShowerTables.synthetic(name)


@functools.lru_cache(maxsize=None)
def _route(name):
    return ShowerTransport(_tables(name))


def _flash_config():
    return KernelConfig(omega_per_ns=np.linspace(0, 1.2, 65),
                        readout_omega_per_ns=np.linspace(0, 1.2, 321),
                        relative_time_edges_ns=np.arange(-60.0, 745.0, 5.0),
                        radial_range_m=(2.0, 250.0), threshold_pe=0.01)


@functools.lru_cache(maxsize=None)
def _flash_route(mode):
    return FlashTransport(synthetic_detector(), _flash_config(),
                          FlashTable.load(TABLES / FLASH_TABLES[450.0]), mode=mode)


@functools.lru_cache(maxsize=None)
def _broadband_route():
    tables = [FlashTable.load(TABLES / name) for name in FLASH_TABLES.values()]
    nodes = [t.medium.wavelength_nm for t in tables]
    return BroadbandFlashTransport(synthetic_detector(), _flash_config(), tables, nodes,
                                   FLASH_NODE_WEIGHTS)


FLASH_NODE_WEIGHTS = [27.77777777777778, 44.44444444444444, 27.77777777777778]  # nm


def _flash_shape(wavelength_nm):
    return np.exp(-((np.asarray(wavelength_nm, float) - 455.0) / 30.0) ** 2)


# ---------------------------------------------------------------- inputs from the seed

def _oms(clusters):
    """OM centres of the synthetic array: 8 strings of 6 modules per cluster."""
    azimuth = np.arange(8) * 2 * np.pi / 8
    strings = np.column_stack((25.0 * np.cos(azimuth), 25.0 * np.sin(azimuth), np.zeros(8)))
    heights = (np.arange(6) - 2.5) * 15.0
    return np.array([[180.0 * c + x, y, h] for c in range(clusters) for x, y, _ in strings
                     for h in heights])


def _flash_inputs(case, seed):
    """Positions in a 60 m x 300 m cylinder at least 2.5 m from every OM, photons, times."""
    rng = np.random.default_rng(seed)
    oms, n = _oms(1), case["flashes"]
    got = np.zeros((0, 3))
    while len(got) < n:
        r, phi = 60.0 * np.sqrt(rng.uniform(size=n)), rng.uniform(0, 2 * np.pi, n)
        p = np.column_stack((r * np.cos(phi), r * np.sin(phi), rng.uniform(-150, 150, n)))
        p = p + oms.mean(axis=0)
        far = np.linalg.norm(p[:, None] - oms[None], axis=2).min(axis=1) > 2.5
        got = np.concatenate((got, p[far]))
    return got[:n], 10.0 ** rng.uniform(9.0, 10.0, n), rng.uniform(0.0, 50.0, n)


def _shower(rng, elements, centre, oms, radius, height):
    """One Gaussian shower: ``elements`` chords of a 1.2 m long, 0.08 m wide profile,
    at a random pose in a cylinder around ``centre``, at least 6 m from every OM."""
    while True:
        r, phi = radius * math.sqrt(rng.uniform()), rng.uniform(0, 2 * math.pi)
        vertex = centre + np.array([r * math.cos(phi), r * math.sin(phi),
                                    rng.uniform(-height / 2, height / 2)])
        if np.linalg.norm(oms - vertex, axis=1).min() > 6.0:
            break
    axis = rng.normal(size=3)
    axis /= np.linalg.norm(axis)
    side = np.cross(axis, [0.0, 0.0, 1.0] if abs(axis[2]) < 0.9 else [1.0, 0.0, 0.0])
    side /= np.linalg.norm(side)
    basis = np.stack((side, np.cross(axis, side), axis))
    sigma, beta = 1.2, 0.999
    z = np.linspace(-3 * sigma, 3 * sigma, elements)
    share = np.exp(-0.5 * (z / sigma) ** 2)
    share /= share.sum()
    start = np.column_stack((rng.normal(scale=0.08, size=(elements, 2)), z))
    unit = np.column_stack((rng.normal(scale=0.025, size=(elements, 2)), np.ones(elements)))
    unit /= np.linalg.norm(unit, axis=1)[:, None]
    length = np.full(elements, max(0.01, 6 * sigma / elements))
    c0 = 2 * np.pi * 7.2973525693e-3 * 1e9 * 0.15 * elements * share
    t0 = (z - z[0]) / (beta * C_M_PER_NS)
    return dict(start_m=start @ basis + vertex, direction=unit @ basis, length_m=length,
                coefficient0=c0, coefficient2=-c0 / beta ** 2, beta=np.full(elements, beta),
                start_ns=t0, end_ns=t0 + length / (beta * C_M_PER_NS))


def _showers(case, seed):
    """The case's showers (their element counts spread evenly in the logarithm)."""
    rng = np.random.default_rng(seed)
    oms = _oms(OMS[case["tables"]] // 48)
    if case["kind"] in ("order0", "shower"):
        sizes = np.round(np.geomspace(case["low"], case["high"], case["showers"])).astype(int)
    else:
        sizes = [case["elements"]] * case.get("showers", 1)
    # the stream's cylinder for batches, the array's own volume for single stages
    radius, height = (40.0, 90.0) if case["tables"] == "c0" else (200.0, 600.0)
    if case["kind"] not in ("order0", "shower"):
        radius, height = min(radius, 100.0), 90.0
    return [_shower(rng, int(n), oms.mean(axis=0), oms, radius, height) for n in sizes]


def _clock(positions, element, group_index):
    """Per-OM clock: earliest element start plus the fastest flight."""
    first = int(np.argmin(element["start_ns"]))
    distance = np.linalg.norm(positions - element["start_m"][first], axis=1)
    return element["start_ns"][first] + distance * group_index / C_M_PER_NS


def _nearest(positions, element, count):
    distance = np.linalg.norm(positions - element["start_m"].mean(axis=0), axis=1)
    return np.sort(np.argsort(distance, kind="stable")[:count])


# ---------------------------------------------------------------- prepare and run

def prepare(case, seed):
    kind = case["kind"]
    if kind == "flash":
        pos, photons, times = _flash_inputs(case, seed)
        if case["call"] == "broadband":
            return dict(case=case, route=_broadband_route(), inputs=(pos, photons, times))
        route = _flash_route(case["mode"])
        if case["call"] == "transport":
            return dict(case=case, route=route, flash=IsotropicFlash.monochromatic(
                pos[0], float(photons[0]), 450.0, time_ns=float(times[0])))
        if case["call"] == "run":
            return dict(case=case, route=route, inputs=(pos, photons, times))
        return dict(case=case, route=route, buffers=route.allocate(len(pos)),
                    inputs=[torch.tensor(v, device=route.device) for v in (pos, photons, times)])
    tables = _tables(case["tables"])
    showers = _showers(case, seed)
    state = dict(case=case, tables=tables, showers=showers)
    if kind == "shower":
        return dict(state, route=_route(case["tables"]))
    fastest = float(np.min(tables.group))
    state["clock"] = np.stack([_clock(tables.positions, el, fastest) for el in showers])
    state["work"] = [_nearest(tables.positions, el, case.get("oms", 0)) for el in showers]
    if kind == "order0":
        state["batch"] = ElementBatch(showers, tables.device)
    elif kind == "order1":
        el = showers[0]
        cone = float(np.sum(tables.prompt["s0w"] * tables.phase) / np.sum(tables.prompt["s0w"]))
        state["resident"] = {k: torch.tensor(v, device=tables.device) for k, v in el.items()}
        state["cone"] = 1.0 / (state["resident"]["beta"] * cone)
    elif kind == "sources":
        state["buffers"] = [torch.zeros((len(tables.fold_bands), SOURCE_ROWS) + tail, dtype=dtype,
                                        device=tables.device)
                            for tail, dtype in (((3,), torch.float64),
                                                ((tables.source.nch, len(tables.omega)),
                                                 torch.complex64))]
    elif kind == "spectra":  # the compiled sources of every shower, as the route holds them
        state["items"] = []
        for el, oms in zip(showers, state["work"]):
            points, channels, counts, reference, frame = tables.source.compile(el)
            n = int(counts[0])
            centre, axis, first, second = (np.asarray(v, float) for v in frame)
            local = points[0, :n].cpu().numpy()
            world = (centre + local[:, :1] * axis + local[:, 1:2] * first
                     + local[:, 2:3] * second)
            source = AxialSources(world, channels[:, :n], np.full(len(counts), reference),
                                  (centre, first, second, axis), tables.source_degree,
                                  tables.azimuthal_degree)
            state["items"].append((source, tables.positions[oms], tables.looks[oms],
                                   tables.areas[oms], tables.radial))
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "flash":
        route = state["route"]
        if case["call"] == "transport":
            r = route.transport(state["flash"])
            return dict(spectrum=r.spectrum_pe, components=r.components_pe,
                        charge=r.charge_components_pe, origin=r.time_origin_ns, active=r.active)
        if case["call"] == "run":
            out = route.run(*state["inputs"])
        elif case["call"] == "broadband":
            out = route.run(*state["inputs"], _flash_shape)
        else:
            out = route.launch(*state["inputs"], state["buffers"])
        return {k: out[k] for k in ("spectrum", "components", "charge", "origin", "active")}
    tables = state["tables"]
    if kind == "order0":
        out = order0(tables.order0, state["batch"], state["clock"], tables.edges, estimate=True)
        return {k: out[k] for k in ("charge", "charge_check", "bins")}
    if kind == "order1":
        t = tables.order1_screen if case["coarse"] else tables.order1
        table = pencils(t, state["showers"][0], state["cone"], device_elements=state["resident"])
        charge, bins = grouped_widening(t, table, state["work"][0], state["clock"][0])
        return dict(charge=charge, bins=bins)
    if kind == "sources":
        points, channels, counts, reference, _ = tables.source.compile(state["showers"][0])
        n = int(counts[0])
        for buffer, values in zip(state["buffers"], (points, channels)):
            buffer[:, :n] = values[:, :n]
            buffer[:, n:] = 0
        return dict(zip(("points", "channels"), state["buffers"]), reference=reference)
    if kind == "spectra":
        return tables.ge2.apply_batch(state["items"], mode=case["mode"])
    if case["showers"] == 1:
        responses = [state["route"](state["showers"][0])]
    else:
        responses = state["route"].batch(state["showers"])
    return [dict(charge=r.charge_components_pe, bins=r.components_pe, spectrum=r.spectrum_ge2_pe,
                 clock=r.time_origin_ns, active=r.active) for r in responses]


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    """Inputs read once, outputs written once; the operations are those that every
    element, ring node or (OM, point) pair needs whatever the geometry is (how many
    pairs a shower lights is known only after the call)."""
    kind = case["kind"]
    if kind == "flash":
        pairs = case["flashes"] * 48
        return dict(bytes=pairs * FLASH_PAIR_BYTES + 40 * case["flashes"],
                    flops=2.0 * pairs * 2 * 130 * 160)
    n_om = OMS[case["tables"]]
    if kind in ("order0", "shower"):
        elements = float(np.round(np.geomspace(case["low"], case["high"],
                                               case["showers"])).sum())
    else:
        elements = float(case["elements"] * case.get("showers", 1))
    slices, nch = 33, 133 if case["tables"] == "c3" else 39
    channels = 5 * slices * nch * 3 * 65 * 8.0  # bytes of one shower's source channels
    if kind == "order0":  # the candidate test of every (element, OM)
        return dict(bytes=96 * elements + case["showers"] * n_om * 162 * 8.0,
                    flops=40 * elements * n_om)
    if kind == "order1":  # every ring node's moments
        return dict(bytes=96 * elements + case["oms"] * 161 * 8.0,
                    flops=100 * elements * (24 if case["coarse"] else 192))
    if kind == "sources":  # each element's links x moments x channels per band
        return dict(bytes=96 * elements + channels, flops=2 * elements * 8 * 5 * nch * 3)
    if kind == "spectra":  # the complex channel product of every (OM, point, channel, frequency)
        pairs = case["showers"] * case["oms"] * 5.0 * slices
        return dict(bytes=case["showers"] * (channels + case["oms"] * 65 * 16),
                    flops=8 * pairs * nch * 3 * 65)
    return dict(bytes=96 * elements + case["showers"] * n_om * (160 * 3 * 8 + 65 * 16.0),
                flops=elements * (40 * n_om + 100 * 192))


# ---------------------------------------------------------------- the same in 64 bits

def exact(case, seed):
    """Flashes and the order >=2 spectra (from the elements on, so with the sources) in
    float64 NumPy / torch. The orders 0 and 1 and the whole route integrate tens of
    millions of nodes per shower, minutes in plain array code: None. The sources alone:
    None, as whether an empty first slice is listed hangs on the last bit of the first
    element's coordinate."""
    if case["kind"] == "flash":
        return _exact_flash(case, seed)
    if case["kind"] == "spectra":
        return _exact_spectra(case, seed)
    return None


def _spline(x, y):
    """Not-a-knot cubic coefficients (interval, 4, ...) in powers 3..0 of x - x_i."""
    n, h = len(x), np.diff(x)
    flat = y.reshape(n, -1)
    a = np.zeros((n, n))
    rhs = np.zeros((n, flat.shape[1]), flat.dtype)
    secant = np.diff(flat, axis=0) / h[:, None]
    for i in range(1, n - 1):  # second derivatives at the knots
        a[i, i - 1:i + 2] = h[i - 1], 2 * (h[i - 1] + h[i]), h[i]
        rhs[i] = 6 * (secant[i] - secant[i - 1])
    a[0, :3] = -h[1], h[0] + h[1], -h[0]  # third derivative continuous at both ends
    a[-1, -3:] = -h[-1], h[-1] + h[-2], -h[-2]
    m = np.linalg.solve(a, rhs)
    c = np.stack(((m[1:] - m[:-1]) / (6 * h[:, None]), m[:-1] / 2,
                  secant - h[:, None] * (2 * m[:-1] + m[1:]) / 6, flat[:-1]), axis=1)
    return c.reshape((n - 1, 4) + y.shape[1:])


def _at(c, x, values):
    """A spline of ``_spline`` at ``values``: (value, ...)."""
    j = np.clip(np.searchsorted(x, values, side="right") - 1, 0, len(x) - 2)
    t = (values - x[j]).reshape((-1,) + (1,) * (c.ndim - 2))
    return ((c[j, 0] * t + c[j, 1]) * t + c[j, 2]) * t + c[j, 3]


def _readout(omega, fine, edges):
    """Complex (bin, frequency) operator: refinement to ``fine``, exact bin integrals."""
    step = np.diff(fine)
    w = np.r_[step[0] / 2, (step[:-1] + step[1:]) / 2, step[-1] / 2]
    width, centre = np.diff(edges), (edges[:-1] + edges[1:]) / 2
    kernel = (width[:, None] * np.sinc(width[:, None] * fine / (2 * np.pi))
              * np.exp(-1j * centre[:, None] * fine) * (w / np.pi))
    return kernel @ _at(_spline(omega, np.eye(len(omega))), omega, fine)


def _exact_flash(case, seed):
    pos, photons, times = _flash_inputs(case, seed)
    oms, n = _oms(1), len(pos)
    edges = np.arange(-60.0, 745.0, 5.0)
    displacement = pos[:, None] - oms[None]
    radius = np.linalg.norm(displacement, axis=2).ravel()
    cosine = -(displacement[:, :, 2].ravel() / radius)  # the OMs look down
    legendre = np.stack((np.ones_like(cosine), cosine, 1.5 * cosine ** 2 - 0.5), axis=1)
    acceptance = .45 + .45 * cosine + .10 * cosine * cosine
    alpha = 4 * np.pi * np.array([.45 + .10 / 3, .45 / 3, .10 * 2 / 3 / 5])
    nodes = [450.0] if case["call"] != "broadband" else list(FLASH_TABLES)
    tables = [dict(np.load(TABLES / FLASH_TABLES[w])) for w in nodes]
    if case["call"] == "broadband":
        share = FLASH_NODE_WEIGHTS * _flash_shape([float(t["wavelength_nm"]) for t in tables])
        share = share / share.sum()
    else:
        share = np.ones(1)
    clock = times.repeat(48) + radius / (C_M_PER_NS / min(float(t["group_index"])
                                                          for t in tables))
    inside = (radius >= 2.0) & (radius <= 250.0)
    omega, total, late, direct = None, 0.0, 0.0, 0.0
    for table, part in zip(tables, share):
        omega, grid = table["omega_per_ns"], table["radii_m"]
        mu_a, speed = float(table["absorption_per_m"]), C_M_PER_NS / float(table["group_index"])
        mu_t = mu_a + float(table["scattering_per_m"])
        weight = .20 * np.exp(-0.5 * ((float(table["wavelength_nm"]) - 450.0) / 90.0) ** 2)
        scale = part * photons.repeat(48) * np.pi * .2 ** 2 * weight

        def amplitude(r):
            return np.exp(-mu_a * r) / (4 * np.pi * r ** 2)

        moments = table["moments"][:, :, :3] / amplitude(grid)[None, :, None, None]
        if str(table["radial_phase"]) == "flight":
            moments = moments * np.exp(-1j * np.outer(omega, grid) / speed)[:, :, None, None]
        c = _spline(np.log(grid), moments.transpose(1, 0, 2, 3))
        spectrum = np.zeros((len(radius), len(omega), 3), complex)
        for lo in range(0, len(radius), 8192):
            k = slice(lo, lo + 8192)
            value = _at(c, np.log(grid), np.log(radius[k]))  # (pair, omega, degree, order)
            value = np.einsum("pwlo,pl->pwo", value, legendre[k] * alpha / (4 * np.pi))
            flight = np.exp(1j * np.outer(radius[k], omega) / speed)
            spectrum[k, :, 1:] = value * (inside[k] * scale[k] * amplitude(radius[k]))[:, None, None]
            spectrum[k, :, 1:] *= flight[:, :, None]
            first = scale[k] * acceptance[k] * np.exp(-mu_t * radius[k])
            first = first / (4 * np.pi * radius[k] ** 2)
            spectrum[k, :, 0] = first[:, None] * flight * np.exp(
                1j * np.outer(np.where(inside[k], 0.0, times.repeat(48)[k]), omega))
        total = total + spectrum
        q0 = scale * acceptance * np.exp(-mu_t * radius) / (4 * np.pi * radius ** 2)
        slot = np.searchsorted(edges, times.repeat(48) + radius / speed - clock, "right") - 1
        bins0 = np.zeros((len(radius), len(edges) - 1))
        ok = (slot >= 0) & (slot < bins0.shape[1])
        bins0[ok, slot[ok]] = q0[ok]
        direct = direct + bins0
    relative = total[:, :, 1:] * np.exp(-1j * np.outer(clock, omega))[:, :, None]
    operator = _readout(omega, np.linspace(0, 1.2, 321), edges)
    late = np.einsum("bw,pwo->pob", operator, relative, optimize=True).real
    components = np.concatenate((direct[:, None], late), axis=1).reshape(n, 48, 3, -1)
    spectrum = total.reshape(n, 48, len(omega), 3)
    out = dict(spectrum=spectrum, components=components, charge=spectrum[:, :, 0].real.copy(),
               origin=clock.reshape(n, 48), active=None)
    if case["call"] == "transport":  # one flash: (frequency, OM, order), (OM, bin, order)
        out = {k: None if v is None else v[0] for k, v in out.items()}
        out["spectrum"] = out["spectrum"].transpose(1, 0, 2)
        out["components"] = out["components"].transpose(0, 2, 1)
    return out


def _layout(degree, top):
    kept = [(ell, m) for ell in range(degree + 1) for m in range(-min(ell, top), min(ell, top) + 1)]
    return kept


def _real_harmonics(v, kept):
    """Real orthonormal harmonics of unit vectors ``v`` for the (l, m) in ``kept``."""
    mu = v[:, 2]
    sine = np.hypot(v[:, 0], v[:, 1])
    phi = np.arctan2(v[:, 1], v[:, 0])
    degree, top = max(l for l, _ in kept), max(m for _, m in kept)
    p = {}
    for m in range(top + 1):
        seed = math.sqrt((2 * m + 1) / (4 * math.pi))
        for k in range(1, m + 1):
            seed *= math.sqrt((2 * k - 1) / (2 * k))
        p[m, m] = seed * sine ** m
        for ell in range(m + 1, degree + 1):
            lower = p.get((ell - 2, m), 0.0)
            p[ell, m] = (math.sqrt((4 * ell * ell - 1) / (ell * ell - m * m)) * (
                mu * p[ell - 1, m] - (math.sqrt(((ell - 1) ** 2 - m * m) / (4 * (ell - 1) ** 2 - 1))
                                      if ell > m + 1 else 0.0) * lower))
    out = np.empty((len(v), len(kept)))
    for k, (ell, m) in enumerate(kept):
        turn = 1.0 if m == 0 else math.sqrt(2) * (np.cos(m * phi) if m > 0 else np.sin(-m * phi))
        out[:, k] = p[ell, abs(m)] * turn
    return out


def _frame(el):
    share = el["coefficient0"] / el["coefficient0"].sum()
    middle = el["start_m"] + 0.5 * el["length_m"][:, None] * el["direction"]
    centre = share @ middle
    off = middle - centre
    values, vectors = np.linalg.eigh((off * share[:, None]).T @ off)
    axis = vectors[:, np.argmax(values)]
    axis = axis / np.linalg.norm(axis)
    if share @ (el["direction"] @ axis) < 0:
        axis = -axis
    first = np.cross(axis, [1.0, 0.0, 0.0] if abs(axis[2]) > 0.9 else [0.0, 0.0, 1.0])
    first /= np.linalg.norm(first)
    return centre, axis, first, np.cross(axis, first)


@functools.lru_cache(maxsize=None)
def _constants(name):
    return dict(np.load(TABLES / f"route_{name}.npz"))


def _exact_sources(name, el):
    """Axial slices of 0.25 m (cubic weights), a 0.02 ns linear time lattice, five-point
    transverse stencils of 0.2 m for slices wider than 0.03 m."""
    r = _constants(name)
    device = "cuda" if torch.cuda.is_available() else "cpu"
    degree, omega = int(r["source_degree"]), r["omega_per_ns"]
    kept = _layout(degree, int(r["azimuthal_degree"]))
    centre, axis, first, second = frame = _frame(el)
    cell, dt, h = 0.25, 0.02, 0.2
    order = 1 if el["length_m"].max() <= cell / 10 else 2
    nodes, weights = np.polynomial.legendre.leggauss(order)
    off = el["start_m"] - centre
    at = {f: off + (f * el["length_m"])[:, None] * el["direction"] for f in [0.5, *(nodes + 1) / 2]}
    z0 = float((at[0.5] @ axis).min()) - 2 * cell
    reference = float(el["start_ns"].min())
    turned = _real_harmonics(np.stack([el["direction"] @ v for v in (first, second, axis)], 1), kept)
    slot, value, moment = [], [], []
    for f, w in zip((nodes + 1) / 2, weights / 2):
        p = at[f]
        x, y, z = p @ first, p @ second, (p @ axis - z0) / cell
        t = (el["start_ns"] + f * (el["end_ns"] - el["start_ns"]) - reference) / dt
        zb, tb = np.floor(z), np.floor(t)
        u, v = z - zb, t - tb
        axial = (-u * (u - 1) * (u - 2) / 6, (u + 1) * (u - 1) * (u - 2) / 2,
                 -(u + 1) * u * (u - 2) / 2, (u + 1) * u * (u - 1) / 6)
        # linear interpolation of the phase between ticks
        phase = ((1 - v)[:, None] * np.exp(1j * np.outer(tb * dt, omega))
                 + v[:, None] * np.exp(1j * np.outer((tb + 1) * dt, omega)))
        m = np.stack((np.ones_like(x), x, y, x * x, y * y), 1) * w
        for j in range(4):
            slot.append(zb.astype(int) + j - 1)
            value.append(phase * axial[j][:, None])
            moment.append(m)
    slot = np.concatenate(slot)
    used, row = np.unique(slot, return_inverse=True)
    row_d = torch.as_tensor(row, device=device)
    value = torch.as_tensor(np.concatenate(value), device=device)
    moment = np.concatenate(moment)
    element = np.tile(np.arange(len(el["length_m"])), len(slot) // len(el["length_m"]))
    points, channels = [], []
    for band in r["fold_bands"]:
        lam, n = float(r["wavelength_nm"][band]), float(r["fold_phase"][band])
        photons = el["coefficient0"] / lam ** 2 + el["coefficient2"] / (lam * n) ** 2
        cone = 1.0 / (el["beta"] * n)
        legendre = [np.ones_like(cone), cone]
        for ell in range(2, degree + 1):
            legendre.append(((2 * ell - 1) * cone * legendre[-1]
                             - (ell - 1) * legendre[-2]) / ell)
        angular = turned * np.stack([legendre[ell] for ell, _ in kept], 1)
        angular = torch.as_tensor(angular[element], device=device)
        factor = torch.as_tensor(moment * photons[element][:, None], device=device)
        field = torch.zeros((len(used), 5, len(kept), len(omega)), dtype=torch.complex128,
                            device=device)
        for s in range(len(used)):
            k = torch.nonzero(row_d == s).ravel()
            left = (factor[k][:, :, None] * angular[k][:, None, :]).reshape(len(k), -1)
            field[s] = (left.T.to(torch.complex128) @ value[k]).reshape(field.shape[1:])
        field = field.cpu().numpy()
        mass = np.zeros((len(used), 5))
        axial_sum = value[:, 0].real.cpu().numpy()  # zero frequency: the phase is 1
        for m in range(5):
            mass[:, m] = np.bincount(row, weights=axial_sum * moment[:, m] * photons[element],
                                     minlength=len(used))
        safe = np.where(mass[:, 0] != 0, mass[:, 0], 1.0)
        wide = np.sqrt(np.abs(mass[:, 3] + mass[:, 4]) / np.abs(safe)) > 0.03
        z = z0 + used * cell
        on_axis = np.where(wide[:, None], 0.0, mass[:, 1:3] / safe[:, None])
        where = [np.column_stack((z, on_axis))]
        m0, mx, my, mxx, myy = (field[:, m] for m in range(5))
        parts = [np.where(wide[:, None, None], m0 - (mxx + myy) / h ** 2, m0)]
        for (dx, dy), second_m, first_m in (((h, 0), mxx, mx), ((-h, 0), mxx, -mx),
                                            ((0, h), myy, my), ((0, -h), myy, -my)):
            where.append(np.column_stack((z, np.full(len(z), dx), np.full(len(z), dy)))[wide])
            parts.append((0.5 * (second_m / h ** 2 + first_m / h))[wide])
        points.append(np.concatenate(where))
        channels.append(np.concatenate(parts) * float(r["fold_scale"][band]))
    return np.stack(points), np.stack(channels), reference, frame


def _small_d(top_out, top_in, degree, cosine):
    """Wigner ``d^l_(m' m)``, m' in 0..top_in, m in -top_out..top_out, by the explicit sum:
    ``{(l, m, m'): (pair,)}``."""
    half_c, half_s = np.sqrt((1 + cosine) / 2), np.sqrt((1 - cosine) / 2)
    out = {}
    for ell in range(degree + 1):
        for mp in range(min(ell, top_in) + 1):
            for m in range(-min(ell, top_out), min(ell, top_out) + 1):
                total = 0.0
                lead = 0.5 * sum(math.lgamma(v + 1) for v in (ell + mp, ell - mp, ell + m, ell - m))
                for k in range(max(0, m - mp), min(ell + m, ell - mp) + 1):
                    size = math.exp(lead - sum(math.lgamma(v + 1) for v in (
                        ell + m - k, k, mp - m + k, ell - mp - k)))
                    total = total + (-1) ** (mp - m + k) * size * half_c ** (
                        2 * ell + m - mp - 2 * k) * half_s ** (mp - m + 2 * k)
                out[ell, m, mp] = total
    return out


def _exact_spectra(case, seed):
    name = case["tables"]
    r = _constants(name)
    fold = dict(np.load(TABLES / {"c0": "ge2_fold_48om_2-150m.npz",
                                  "c2": "ge2_fold_384om_2-450m.npz",
                                  "c3": "ge2_fold_384om_1-300m.npz"}[name]))
    return [_exact_apply(r, fold, el, *_exact_sources(name, el),
                         _nearest(r["positions_m"], el, case["oms"])) for el in _showers(case, seed)]


def _exact_apply(r, fold, el, points, channels, reference, frame, oms):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    centre, axis, first, second = frame
    basis = np.stack((first, second, axis))
    local = points[0][:, [1, 2, 0]]  # (x, y, z) in the frame, shared by the bands
    receivers, looks = (r["positions_m"][oms] - centre) @ basis.T, r["looks"][oms] @ basis.T
    omega, degree = r["omega_per_ns"], int(fold["degree"])
    top, out_top = min(int(r["azimuthal_degree"]), degree), int(fold["acceptance_degree"])
    alpha, low_high = r["alpha"], r["radial_range_m"]
    coefficients = torch.as_tensor(fold["coefficients"], device=device).to(torch.complex128)
    field = torch.as_tensor(channels, device=device)
    kept = _layout(int(r["source_degree"]), int(r["azimuthal_degree"]))
    inner = _layout(out_top, out_top)
    result = np.zeros((len(oms), len(omega)), complex)
    for i in range(len(oms)):
        d = receivers[i] - local
        radius = np.linalg.norm(d, axis=1)
        sel = np.flatnonzero((radius >= low_high[0]) & (radius <= low_high[1]))
        if not len(sel):
            continue
        d, radius = d[sel], radius[sel]
        cosine = np.clip(d[:, 2] / radius, -1, 1)
        phi = np.arctan2(d[:, 1], d[:, 0])
        sine = np.hypot(d[:, 0], d[:, 1]) / radius
        cp, sp = np.cos(phi), np.sin(phi)
        lx, ly, lz = looks[i]
        turned = np.stack((cosine * cp * lx + cosine * sp * ly - sine * lz, -sp * lx + cp * ly,
                           sine * cp * lx + sine * sp * ly + cosine * lz), 1)
        detector = _real_harmonics(turned / np.linalg.norm(turned, axis=1)[:, None], inner)
        small = _small_d(out_top, top, degree, cosine)
        j = np.clip(np.searchsorted(fold["log_r"], np.log(radius), "right") - 1, 0,
                    len(fold["log_r"]) - 2)
        t = torch.as_tensor(np.log(radius) - fold["log_r"][j], device=device)
        powers = torch.stack((t ** 3, t ** 2, t, torch.ones_like(t)), 1)
        response = torch.zeros((field.shape[0], len(sel), len(omega)), dtype=torch.complex128,
                               device=device)
        for ell in range(degree + 1):
            near, reach = min(ell, top), min(ell, out_top)
            # rotation of the source's (l, m) onto the ray: rows m', columns m
            turn = np.zeros((len(sel), 2 * out_top + 1, 2 * near + 1))
            root = math.sqrt(2)
            turn[:, out_top, near] = small[ell, 0, 0]
            for m in range(1, near + 1):
                base = root * (-1) ** m * small[ell, 0, m]
                turn[:, out_top, near + m] = base * np.cos(m * phi)
                turn[:, out_top, near - m] = base * np.sin(m * phi)
            for p in range(1, reach + 1):
                turn[:, out_top + p, near] = root * (-1) ** p * small[ell, p, 0]
                for m in range(1, near + 1):
                    cross, straight = (-1) ** p * small[ell, p, m], small[ell, -p, m]
                    even = (-1) ** m * (cross + straight)
                    odd = (-1) ** m * (cross - straight)
                    turn[:, out_top + p, near + m] = even * np.cos(m * phi)
                    turn[:, out_top + p, near - m] = even * np.sin(m * phi)
                    turn[:, out_top - p, near + m] = -odd * np.sin(m * phi)
                    turn[:, out_top - p, near - m] = odd * np.cos(m * phi)
            rows = [k for k, (l, _) in enumerate(kept) if l == ell and abs(kept[k][1]) <= near]
            look = np.zeros((len(sel), len(fold["pair_mu"]), 2 * near + 1))
            for q, (lam, mu) in enumerate(zip(fold["pair_lambda"], fold["pair_mu"])):
                if mu > reach:
                    continue
                for m in {int(mu), -int(mu)}:
                    weight = alpha[lam] * detector[:, inner.index((int(lam), m))]
                    look[:, q] += weight[:, None] * turn[:, out_top + m]
            mix = torch.as_tensor(look, device=device).to(torch.complex128)
            rotated = torch.einsum("pqc,bpcw->bpqw", mix, field[:, sel][:, :, rows])
            radial = torch.einsum("bpqkw,pk->bpqw", coefficients[:, j, ell],
                                  powers.to(torch.complex128))
            response += (rotated * radial).sum(2)
        scale = (r["areas_m2"][oms[i]] * np.exp(-np.outer(fold["absorption"], radius))
                 / (4 * np.pi * radius ** 2))
        phase = np.ones((len(scale), len(sel), len(omega)), complex)
        if str(fold["phase"]) == "flight":
            phase = np.exp(1j * omega * (radius[None, :, None] / fold["speed"][:, None, None]))
        factor = torch.as_tensor(scale[:, :, None] * phase, device=device)
        result[i] = (response * factor).sum((0, 1)).cpu().numpy()
    return result * np.exp(1j * omega * reference)
