"""Order >=2 contraction: oracle pinned to the reference, device kernel vs oracle."""
import numpy as np
import pytest

from conftest import GOLDEN, TABLES
from oracle.ge2 import apply_folded as oracle_apply

# Device >=2 spectra: float32 contraction, float64 geometry. Error relative to
# the largest |value| of the spectrum (>=2 charges can be slightly negative).
GE2_TOL = 2e-5


def fixture():
    g = np.load(GOLDEN / "shower_c0.npz")
    t = dict(np.load(TABLES / "ge2_fold_48om_2-150m.npz"))
    frame = dict(centre=g["frame_centre_m"], first=g["frame_first"], second=g["frame_second"],
                 axis=g["frame_axis"])
    return g, t, frame


def points(g, frame, tag):
    z, tr = g[f"{tag}_z_m"], g[f"{tag}_transverse_m"]
    return (frame["centre"][None] + z[:, None] * frame["axis"][None]
            + tr[:, 0:1] * frame["first"][None] + tr[:, 1:2] * frame["second"][None])


def oracle_sources(g, frame, tag, channels=None):
    return dict(points_m=points(g, frame, tag),
                channels=g[f"{tag}_channels"] if channels is None else channels,
                reference_ns=g[f"{tag}_reference_ns"], frame=frame,
                degree=int(g["source_degree"]), azimuthal_degree=int(g["azimuthal_degree"]))


def test_oracle_matches_reference_full_frequency_subset():
    g, t, frame = fixture()
    out = oracle_apply(t, oracle_sources(g, frame, "sub"), g["om_positions_m"], g["om_looks"],
                       g["alpha"], g["om_area_m2"], g["radial_window_m"])
    assert np.abs(out - g["spec_sub"]).max() <= 1e-12 * np.abs(g["spec_sub"]).max()


@pytest.mark.gpu
@pytest.mark.parametrize("tag", ["zero", "sub"])
def test_device_apply_matches_reference(tag):
    from lighthit_b200.ge2 import AxialSources, Ge2Table
    g, t, frame = fixture()
    table = Ge2Table(t, g["alpha"], source_degree=int(g["source_degree"]),
                     azimuthal_degree=int(g["azimuthal_degree"]))
    src = AxialSources(points(g, frame, tag), g[f"{tag}_channels"], g[f"{tag}_reference_ns"],
                       (frame["centre"], frame["first"], frame["second"], frame["axis"]),
                       int(g["source_degree"]), int(g["azimuthal_degree"]))
    out = table.apply(src, g["om_positions_m"], g["om_looks"], g["om_area_m2"],
                      g["radial_window_m"], zero_frequency=(tag == "zero"))
    ref = g[f"spec_{tag}"]
    assert out.shape == ref.shape
    assert np.abs(out - ref).max() <= GE2_TOL * np.abs(ref).max()


@pytest.mark.gpu
def test_device_apply_all_points_random_channels_vs_oracle():
    """Every basis point at all 65 frequencies (seeded channels), vs the oracle."""
    from lighthit_b200.ge2 import AxialSources, Ge2Table
    g, t, frame = fixture()
    rng = np.random.default_rng(8)
    P = int(g["n_points"])
    zero_pts = points(g, frame, "zero")
    ch = (rng.normal(size=(3, P, 39, 65)) + 1j * rng.normal(size=(3, P, 39, 65))).astype(np.complex64)
    ch *= np.abs(g["zero_channels"][:, :, :, :1])  # keep the sources' magnitude profile
    oms = np.arange(0, 48, 4)
    src_o = dict(points_m=zero_pts, channels=ch, reference_ns=np.array([0.0, 0.3, -0.2]),
                 frame=frame, degree=int(g["source_degree"]),
                 azimuthal_degree=int(g["azimuthal_degree"]))
    ref = oracle_apply(t, src_o, g["om_positions_m"][oms], g["om_looks"][oms], g["alpha"],
                       g["om_area_m2"][oms], g["radial_window_m"])
    table = Ge2Table(t, g["alpha"], source_degree=8, azimuthal_degree=2)
    src = AxialSources(zero_pts, ch, src_o["reference_ns"],
                       (frame["centre"], frame["first"], frame["second"], frame["axis"]), 8, 2)
    out = table.apply(src, g["om_positions_m"][oms], g["om_looks"][oms], g["om_area_m2"][oms],
                      g["radial_window_m"])
    assert np.abs(out - ref).max() <= GE2_TOL * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("zero_frequency", [True, False])
def test_batched_problems_equal_alone(zero_frequency):
    """Problems of one batched launch (different OM subsets, sources, frames,
    one without points) equal each problem applied alone, bit for bit: the
    point chunks are summed in the same fixed order either way."""
    from lighthit_b200.ge2 import AxialSources, Ge2Table
    g, t, frame = fixture()
    table = Ge2Table(t, g["alpha"], source_degree=8, azimuthal_degree=2)
    rng = np.random.default_rng(17)
    pts = points(g, frame, "zero")
    P = len(pts)
    basis = (frame["centre"], frame["first"], frame["second"], frame["axis"])
    items = []
    for k, oms in enumerate([np.arange(48), np.arange(3, 40, 5), np.array([7])]):
        ch = (rng.normal(size=(3, P, 39, 65)) + 1j * rng.normal(size=(3, P, 39, 65))).astype(
            np.complex64) * np.abs(g["zero_channels"][:, :, :, :1])
        shifted = tuple(np.asarray(v) + (0.3 * k * frame["axis"] if i == 0 else 0)
                        for i, v in enumerate(basis))
        src = AxialSources(pts + 0.3 * k * frame["axis"], ch, np.array([0.0, 0.1 * k, 0.0]),
                           shifted, 8, 2)
        items.append((src, g["om_positions_m"][oms], g["om_looks"][oms], g["om_area_m2"][oms],
                      g["radial_window_m"]))
    empty = AxialSources(np.zeros((0, 3)), np.zeros((3, 0, 39, 65), np.complex64),
                         np.zeros(3), basis, 8, 2)
    items.append((empty,) + items[1][1:])
    together = [r.cpu().numpy() for r in table.apply_batch(items, zero_frequency=zero_frequency)]
    for it, got in zip(items, together):
        alone = table.apply_device(*it, zero_frequency=zero_frequency).cpu().numpy()
        assert got.shape == alone.shape
        assert np.array_equal(got, alone)
    assert not np.any(together[-1])
    assert np.any(together[0])


# Tensor-core contraction: BF16 operands with float32 accumulation. Split-BF16
# carries 24 significant bits per operand (hi + mid + lo, six products), as the
# float32 contraction; a single BF16 product 8 bits. Error relative to the
# largest |value|.
TC_TOL = {"split-bf16": GE2_TOL, "bf16": 2e-2}


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["split-bf16", "bf16"])
def test_tensor_core_apply_vs_oracle(mode):
    """Every basis point at all 65 frequencies (seeded channels) through the
    tcgen05 contraction, against the float64 oracle and the float32 CUDA-core
    contraction."""
    from lighthit_b200.ge2 import AxialSources, Ge2Table
    g, t, frame = fixture()
    rng = np.random.default_rng(9)
    P = int(g["n_points"])
    pts = points(g, frame, "zero")
    ch = (rng.normal(size=(3, P, 39, 65)) + 1j * rng.normal(size=(3, P, 39, 65))).astype(np.complex64)
    ch *= np.abs(g["zero_channels"][:, :, :, :1])
    oms = np.arange(48)
    refs = np.array([0.0, 0.2, -0.1])
    src_o = dict(points_m=pts, channels=ch, reference_ns=refs, frame=frame,
                 degree=int(g["source_degree"]), azimuthal_degree=int(g["azimuthal_degree"]))
    ref = oracle_apply(t, src_o, g["om_positions_m"], g["om_looks"], g["alpha"],
                       g["om_area_m2"], g["radial_window_m"])
    table = Ge2Table(t, g["alpha"], source_degree=8, azimuthal_degree=2)
    assert table.tc_packed() is not None
    src = AxialSources(pts, ch, refs, (frame["centre"], frame["first"], frame["second"],
                                       frame["axis"]), 8, 2)
    item = (src, g["om_positions_m"][oms], g["om_looks"][oms], g["om_area_m2"][oms],
            g["radial_window_m"])
    out = table.apply_batch([item], mode=mode)[0].cpu().numpy().T
    assert int(table.status.item()) == 0
    fp32 = table.apply_batch([item], mode="fp32")[0].cpu().numpy().T
    scale = np.abs(ref).max()
    err, err32 = np.abs(out - ref).max() / scale, np.abs(fp32 - ref).max() / scale
    print(f"\n{mode}: max error {err:.2e} of the largest value (fp32 CUDA cores {err32:.2e})")
    assert err <= TC_TOL[mode]


@pytest.mark.gpu
def test_tensor_core_batched_problems_equal_alone():
    """The tensor-core path computes every (OM, point) pair on its own and sums
    the points in a fixed order: a problem's spectrum is the same bit for bit
    alone and in a batch (other OMs, sources, frames, an empty problem)."""
    from lighthit_b200.ge2 import AxialSources, Ge2Table
    g, t, frame = fixture()
    table = Ge2Table(t, g["alpha"], source_degree=8, azimuthal_degree=2)
    rng = np.random.default_rng(18)
    pts = points(g, frame, "zero")
    P = len(pts)
    basis = (frame["centre"], frame["first"], frame["second"], frame["axis"])
    items = []
    for k, oms in enumerate([np.arange(48), np.arange(3, 40, 5), np.array([7])]):
        ch = (rng.normal(size=(3, P, 39, 65)) + 1j * rng.normal(size=(3, P, 39, 65))).astype(
            np.complex64) * np.abs(g["zero_channels"][:, :, :, :1])
        shifted = tuple(np.asarray(v) + (0.3 * k * frame["axis"] if i == 0 else 0)
                        for i, v in enumerate(basis))
        src = AxialSources(pts + 0.3 * k * frame["axis"], ch, np.array([0.0, 0.1 * k, 0.0]),
                           shifted, 8, 2)
        items.append((src, g["om_positions_m"][oms], g["om_looks"][oms], g["om_area_m2"][oms],
                      g["radial_window_m"]))
    empty = AxialSources(np.zeros((0, 3)), np.zeros((3, 0, 39, 65), np.complex64),
                         np.zeros(3), basis, 8, 2)
    items.append((empty,) + items[1][1:])
    together = [r.cpu().numpy() for r in table.apply_batch(items, mode="split-bf16")]
    assert int(table.status.item()) == 0
    for it, got in zip(items, together):
        alone = table.apply_batch([it], mode="split-bf16")[0].cpu().numpy()
        assert np.array_equal(got, alone)
    assert not np.any(together[-1])
    assert np.any(together[0])


@pytest.mark.gpu
@pytest.mark.parametrize("n_points", [1, 15, 16, 17, 48, 49, 140])
def test_tensor_core_tile_edges(n_points):
    """Work items at the edges of a group (16 pairs) and of a tile (48), with few
    pairs per interval and with many, and problems whose channel rows have other
    strides (more frequencies stored than read): against the float64 oracle."""
    from lighthit_b200.ge2 import AxialSources, Ge2Table
    g, t, frame = fixture()
    table = Ge2Table(t, g["alpha"], source_degree=8, azimuthal_degree=2)
    rng = np.random.default_rng(n_points)
    pts = points(g, frame, "zero")[:n_points]
    P = len(pts)
    basis = (frame["centre"], frame["first"], frame["second"], frame["axis"])
    oms = np.array([3, 20, 41])
    items, expected = [], []
    for stored in (65, 70, 65, 66):
        ch = (rng.normal(size=(3, P, 39, stored))
              + 1j * rng.normal(size=(3, P, 39, stored))).astype(np.complex64)
        for some in (oms[:1], oms):
            src = AxialSources(pts, ch, np.zeros(3), basis, 8, 2)
            items.append((src, g["om_positions_m"][some], g["om_looks"][some],
                          g["om_area_m2"][some], g["radial_window_m"]))
            expected.append(oracle_apply(
                t, dict(points_m=pts, channels=ch[..., :65], reference_ns=np.zeros(3),
                        frame=frame, degree=8, azimuthal_degree=2), g["om_positions_m"][some],
                g["om_looks"][some], g["alpha"], g["om_area_m2"][some], g["radial_window_m"],
                fast=True))
    out = table.apply_batch(items, mode="split-bf16")
    assert int(table.status.item()) == 0
    for got, ref in zip(out, expected):
        assert np.abs(got.cpu().numpy().T - ref).max() <= GE2_TOL * np.abs(ref).max()


def folded_of(n_bands, n_intervals, n_omega, *, degree=1, seed=5):
    """Seeded folded kernels of one (lambda, mu) pair over 2-150 m."""
    rng = np.random.default_rng(seed)
    shape = (n_bands, n_intervals, degree + 1, 1, 4, n_omega)
    return dict(coefficients=rng.normal(size=shape) + 1j * rng.normal(size=shape),
                log_r=np.linspace(np.log(2.0), np.log(150.0), n_intervals + 1),
                omega=np.linspace(0.0, 0.5, n_omega), absorption=np.full(n_bands, 0.02),
                speed=np.full(n_bands, 0.218), degree=degree, acceptance_degree=0,
                pair_lambda=np.array([0]), pair_mu=np.array([0]), phase="flight")


def test_tensor_core_shapes_by_their_shared_memory():
    """The pairs' channel pointers of every band, and the starts of every interval, lie
    in shared memory: tables with more take the CUDA cores, others the tensor cores
    (16 pairs per group up to azimuthal degree 2, 8 above)."""
    import ctypes
    from lighthit_b200 import _lib

    def packed(n_bands, n_intervals=47, n_omega=1, max_m=2):
        one = ctypes.c_void_p(16)  # only its presence is looked at
        return int(_lib.load().lh_ge2_tc_pack_bytes(_lib.Ge2Table(
            n_bands, n_intervals, 8, 2, max_m, 6, 39, n_omega, one, one, one, one, one, one, one,
            one, one, one, 2, 1)))

    for n_bands, max_m, takes in ((1, 2, True), (60, 2, True), (61, 2, False), (256, 2, False),
                                  (61, 4, True), (121, 4, True), (122, 4, False)):
        assert (packed(n_bands, max_m=max_m) > 0) == takes, (n_bands, max_m)
    for n_intervals, takes in ((6000, True), (6200, True), (29000, True), (29100, False)):
        assert (packed(3, n_intervals, 65) > 0) == takes, n_intervals


@pytest.mark.gpu
@pytest.mark.parametrize("n_bands, n_intervals", [(60, 7), (64, 7), (2, 6200)])
def test_many_bands_and_many_intervals_match_the_oracle(n_bands, n_intervals):
    """Tables on both sides of the shared-memory limit of the channel pointers, and
    one whose interval starts pass 48 KB: split-BF16 applies against the float64
    oracle, on whichever cores they take."""
    from lighthit_b200.ge2 import AxialSources, Ge2Table
    g, _, frame = fixture()
    t = folded_of(n_bands, n_intervals, 4 if n_bands > 2 else 3)
    W = len(t["omega"])
    table = Ge2Table(t, [1.0], source_degree=1, azimuthal_degree=1)
    assert (table.tc_packed() is not None) == (n_bands != 64)
    rng = np.random.default_rng(n_bands)
    pts = points(g, frame, "zero")[:20]
    ch = (rng.normal(size=(n_bands, 20, 4, W))
          + 1j * rng.normal(size=(n_bands, 20, 4, W))).astype(np.complex64)
    src = AxialSources(pts, ch, np.zeros(n_bands),
                       (frame["centre"], frame["first"], frame["second"], frame["axis"]), 1, 1)
    oms = np.arange(0, 48, 5)
    out = table.apply_batch([(src, g["om_positions_m"][oms], g["om_looks"][oms],
                              g["om_area_m2"][oms], g["radial_window_m"])], mode="split-bf16")[0]
    assert table.status is None or int(table.status.item()) == 0
    ref = oracle_apply(t, dict(points_m=pts, channels=ch, reference_ns=np.zeros(n_bands),
                               frame=frame, degree=1, azimuthal_degree=1),
                       g["om_positions_m"][oms], g["om_looks"][oms], [1.0], g["om_area_m2"][oms],
                       g["radial_window_m"], fast=True)
    assert np.abs(out.cpu().numpy().T - ref).max() <= GE2_TOL * np.abs(ref).max()


@pytest.mark.gpu
def test_channel_rows_beyond_32_bit_offsets():
    """Channels cut from a buffer whose rows lie so far apart that a point's block passes
    4 GB: its last row is read at its own offset, not at that modulo 2^32."""
    import torch
    from lighthit_b200.ge2 import AxialSources, Ge2Table
    g, _, frame = fixture()
    t = folded_of(1, 7, 3)
    table = Ge2Table(t, [1.0], source_degree=1, azimuthal_degree=1)
    rng = np.random.default_rng(3)
    values = (rng.normal(size=(1, 1, 4, 3)) + 1j * rng.normal(size=(1, 1, 4, 3))).astype(np.complex64)
    stored = torch.empty((1, 1, 4, 180_000_000), dtype=torch.complex64, device=table.device)
    stored[..., :3] = torch.from_numpy(values).to(table.device)
    basis = (frame["centre"], frame["first"], frame["second"], frame["axis"])
    pts = points(g, frame, "zero")[:1]
    item = (AxialSources(pts, stored, np.zeros(1), basis, 1, 1), g["om_positions_m"][:1],
            g["om_looks"][:1], g["om_area_m2"][:1], g["radial_window_m"])
    out = table.apply_batch([item], mode="split-bf16")[0].cpu().numpy().T
    assert table.tc_packed() is not None and int(table.status.item()) == 0
    ref = oracle_apply(t, dict(points_m=pts, channels=values, reference_ns=np.zeros(1),
                               frame=frame, degree=1, azimuthal_degree=1), g["om_positions_m"][:1],
                       g["om_looks"][:1], [1.0], g["om_area_m2"][:1], g["radial_window_m"],
                       fast=True)
    assert np.abs(out - ref).max() <= GE2_TOL * np.abs(ref).max()


@pytest.mark.parametrize("kind", ["host", "host slice", "contiguous", "point slice"])
@pytest.mark.parametrize("shifted", [False, True])
def test_zero_frequency_problems_copy_one_column(kind, shifted):
    """What a zero-frequency problem takes of its channels: the first frequency alone
    wherever they have to be copied (host arrays, a slice of a larger buffer, bands
    aligned to one reference), the caller's own tensor where it is contiguous."""
    import torch
    from lighthit_b200.ge2 import AxialSources, Ge2Table
    g, t, frame = fixture()
    table = Ge2Table(t, g["alpha"], source_degree=8, azimuthal_degree=2, device="cpu")
    rng = np.random.default_rng(12)
    full = (rng.normal(size=(3, 9, 39, 65)) + 1j * rng.normal(size=(3, 9, 39, 65))).astype(
        np.complex64)
    kept = full if kind in ("host", "contiguous") else full[:, :5]
    channels = kept if kind.startswith("host") else torch.from_numpy(full)[:, :kept.shape[1]]
    refs = np.array([0.0, 0.2, 0.1]) if shifted else np.zeros(3)
    src = AxialSources(points(g, frame, "zero")[:kept.shape[1]], channels, refs,
                       (frame["centre"], frame["first"], frame["second"], frame["axis"]), 8, 2)
    q = table._prepare(src, g["om_positions_m"], g["om_looks"], g["om_area_m2"],
                       g["radial_window_m"], True)
    got = q["ch"] if isinstance(q["ch"], np.ndarray) else q["ch"].numpy()
    if kind == "contiguous" and not shifted:
        assert q["ch"].data_ptr() == channels.data_ptr()
    else:
        assert got.shape[3] == 1 and got.flags.c_contiguous
    assert q["W"] == 1
    # at the first frequency (zero) the bands' alignment is the identity
    assert np.array_equal(got[..., 0], kept[..., 0])


@pytest.mark.gpu
@pytest.mark.parametrize("group, fill, groups", [(16, 100, 2), (16, 160, 3), (8, 50, 2), (8, 110, 3)])
def test_tensor_core_tiles_of_several_groups(group, fill, groups):
    """Launches of enough pairs make tiles of two and of three groups (16 pairs each, or 8
    above azimuthal degree 2): intervals that hold every remainder of such tiles, in one
    problem of a batch whose other problem fills the launch. Against the float64 oracle,
    and bit for bit against the same problem alone, whose tiles are one group."""
    from lighthit_b200.ge2 import AxialSources, Ge2Table
    g, t, frame = fixture()
    if group == 16:
        degree, azimuthal, alpha = 8, 2, g["alpha"]
    else:
        degree, azimuthal, alpha = 4, 4, [1.0]
        t = folded_of(3, 20, 65, degree=degree)
    table = Ge2Table(t, alpha, source_degree=degree, azimuthal_degree=azimuthal)
    rng = np.random.default_rng(group + fill)
    basis = (frame["centre"], frame["first"], frame["second"], frame["axis"])
    log_r, om = np.asarray(t["log_r"], float), g["om_positions_m"][7]

    def sources(intervals):
        step = log_r[1] - log_r[0]
        r = np.exp(log_r[intervals] + step * rng.uniform(0.1, 0.9, len(intervals)))
        u = rng.normal(size=(len(intervals), 3))
        pts = om + r[:, None] * u / np.linalg.norm(u, axis=1)[:, None]
        shape = (3, len(pts), table.nch, 65)
        ch = (rng.normal(size=shape) + 1j * rng.normal(size=shape)).astype(np.complex64)
        return AxialSources(pts, ch, np.zeros(3), basis, degree, azimuthal)

    full = 3 * group  # pairs of a tile of three groups
    counts = [1, group - 1, group, group + 1, 2 * group, 2 * group + 1, full - 1, full, full + 1]
    window = (float(np.exp(log_r[0])), float(np.exp(log_r[-1])))
    edges = sources(np.repeat(np.arange(3, 3 + len(counts)), counts))
    filler = sources(np.full(fill, 15))
    one, many = np.array([7]), np.full(48, 7)  # 48 OMs at one place: 48 x fill pairs
    # a tile takes as many groups as leave every SM two work items (tile, half)
    pairs = sum(counts) + 48 * fill
    assert 148 * groups * group <= pairs and (groups == 3 or pairs < 148 * full)
    items = [(s, g["om_positions_m"][k], g["om_looks"][k], g["om_area_m2"][k], window)
             for s, k in ((edges, one), (filler, many))]
    out = [r.cpu().numpy() for r in table.apply_batch(items, mode="split-bf16")]
    assert table.tc_packed() is not None and int(table.status.item()) == 0
    alone = table.apply_batch(items[:1], mode="split-bf16")[0].cpu().numpy()
    assert np.array_equal(out[0], alone)
    for got, (s, pos, looks, area, _) in zip(out, items):
        ref = oracle_apply(t, dict(points_m=s.points_m, channels=s.channels,
                                   reference_ns=np.zeros(3), frame=frame, degree=degree,
                                   azimuthal_degree=azimuthal), pos, looks, alpha, area, window,
                           fast=True)
        assert np.abs(got.T - ref).max() <= GE2_TOL * np.abs(ref).max()
