"""Calls on a stream of the caller's (``-m gpu``): each uploads and clears on the current
stream, so its launches have to come after that, and its status read after them."""
import numpy as np
import pytest

from conftest import GOLDEN, TABLES

pytestmark = pytest.mark.gpu
KEYS = ("start_m", "direction", "length_m", "coefficient0", "coefficient2", "beta", "start_ns",
        "end_ns")


def contraction():
    from lighthit_b200.ge2 import AxialSources, Ge2Table
    from test_ge2 import fixture, points
    g, t, frame = fixture()
    table = Ge2Table(t, g["alpha"], source_degree=8, azimuthal_degree=2)
    table.tc_packed()
    rng = np.random.default_rng(21)
    pts = points(g, frame, "zero")
    shape = (3, len(pts), 39, 65)
    ch = (rng.normal(size=shape) + 1j * rng.normal(size=shape)).astype(np.complex64)
    src = AxialSources(pts, ch, np.zeros(3), (frame["centre"], frame["first"], frame["second"],
                                              frame["axis"]), 8, 2)
    item = (src, g["om_positions_m"], g["om_looks"], g["om_area_m2"], g["radial_window_m"])
    return lambda mode: lambda stream: table.apply_batch([item], mode=mode, stream=stream)


def direct_light():
    from lighthit_b200.order0 import order0
    from test_order0_gpu import fixture, optics_of
    g, el = fixture()
    optics = optics_of(g, 2)

    def call(stream):
        out = order0(optics, [el], g["origins_ns"][None], g["edges_ns"], stream=stream)
        return out["charge"], out["bins"]
    return call


def scattered_light():
    from lighthit_b200.order1 import grouped, pencils
    from test_order1_gpu import fixture, tables_of
    g = fixture()
    tables = tables_of(g)
    source = np.load(GOLDEN / "order0_c0.npz")
    el = {k: source[k][::7] for k in KEYS}
    cone = 1.0 / (1.35 * el["beta"])
    work = np.arange(0, len(g["positions_m"]), 5)

    def call(stream):
        table = pencils(tables, el, cone, stream=stream)
        return grouped(tables, table, work, g["origins_ns"], stream=stream)
    return call


def sources():
    from lighthit_b200.source import SourceCompiler
    g = np.load(GOLDEN / "source_c0.npz")
    source = np.load(GOLDEN / "order0_c0.npz")
    el = {k: source[k] for k in KEYS}
    bands = g["bands"]
    comp = SourceCompiler(g["wavelengths_nm"][bands], g["phase_index"], g["scale"][bands],
                          int(g["source_degree"]), int(g["azimuthal_degree"]), g["omega_per_ns"])
    frame = (g["frame_centre_m"], g["frame_axis"], g["frame_first"], g["frame_second"])

    def call(stream):
        points, channels, counts, _, _ = comp.compile(el, frame, stream=stream)
        n = int(counts[0])
        return points[:, :n], channels[:, :n]
    return call


@pytest.mark.parametrize("make, tolerance", [
    (lambda: contraction()("split-bf16"), 0.0), (lambda: contraction()("fp32"), 0.0),
    (direct_light, 1e-12), (scattered_light, 1e-9), (sources, 1e-6)],
    ids=["tensor-cores", "cuda-cores", "order0", "order1", "sources"])
def test_a_given_stream_waits_for_the_uploads(make, tolerance):
    """The current stream is held busy while a call uploads on it and launches on another
    stream: the results are those of the current stream (float64 atomics in any order:
    1e-12 of the largest for order 0, 1e-9 for order 1 whose groups' order differs, 1e-6
    for complex64 sources)."""
    import torch
    call = make()
    expected = [t.clone() for t in call(None)]
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for _ in range(2):
        torch.cuda._sleep(20_000_000)  # 10 ms of the current stream
        got = call(side)
        side.synchronize()
        for a, b in zip(expected, got):
            scale = float(a.abs().max())
            assert scale > 0
            assert float((a - b).abs().max()) <= tolerance * scale
