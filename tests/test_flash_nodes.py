"""Photons of a broadband flash at the wavelength nodes (CPU).

``flash_node_photons`` restates ``_flash_nodes`` (``transport.py:1049-1059``):
``photons * weight * shape / (weight . shape)``. The node wavelengths and
weights are the reference kernel's (``tests/golden/flash_broadband_c1.npz``).
"""
import numpy as np
import pytest

from conftest import GOLDEN


def test_node_photons_split_the_flash_by_weight_and_shape():
    from lighthit_b200.flash import flash_node_photons
    g = np.load(GOLDEN / "flash_broadband_c1.npz")
    nodes, weights = g["node_wavelength_nm"], g["node_weight_nm"]
    centre, width = float(g["shape_centre_nm"]), float(g["shape_width_nm"])

    def shape(wavelength):
        return np.exp(-((np.asarray(wavelength, float) - centre) / width) ** 2)

    photons = g["flash_photons"]
    got = flash_node_photons(nodes, weights, photons, shape)
    assert got.shape == (len(nodes), len(photons))
    assert np.allclose(got.sum(axis=0), photons, rtol=1e-14)  # the nodes share the photons
    w = weights * shape(nodes)
    assert np.allclose(got[:, 0], photons[0] * w / w.sum(), rtol=1e-15)
    with pytest.raises(ValueError):
        flash_node_photons(nodes, weights, photons, lambda x: np.zeros_like(x))
    with pytest.raises(ValueError):
        flash_node_photons(nodes, weights, photons, lambda x: -np.ones_like(x))


def test_response_of_outputs_kept_on_the_host():
    """A batch's outputs moved to host memory give the flash's response, in arrays of
    their own."""
    import torch
    from lighthit_b200.flash import FlashTransport
    from lighthit_b200.model import synthetic_detector
    g = np.load(GOLDEN / "flash_c1.npz")
    ft = FlashTransport.__new__(FlashTransport)  # no device: only what a response reads
    ft.detector, ft.wavelength_nm, ft.mode = synthetic_detector(), 450.0, "fp32"
    ft.config = type("Config", (), dict(omega_per_ns=g["omega_per_ns"],
                                        relative_time_edges_ns=g["edges_ns"],
                                        radial_range_m=(2.0, 250.0)))()
    D, W, B = len(ft.detector), len(g["omega_per_ns"]), len(g["edges_ns"]) - 1
    rng = np.random.default_rng(4)
    out = dict(spectrum=torch.from_numpy((rng.normal(size=(2, D, W, 3)) + 1j).astype(np.complex64)),
               components=torch.from_numpy(rng.normal(size=(2, D, 3, B)).astype(np.float32)),
               charge=torch.from_numpy(rng.normal(size=(2, D, 3))),
               origin=torch.from_numpy(rng.normal(size=(2, D))),
               active=torch.from_numpy(rng.integers(0, 2, (2, D)).astype(np.uint8)))
    r = ft.response(out, 1)
    assert np.array_equal(r.spectrum_pe, out["spectrum"][1].numpy().transpose(1, 0, 2))
    assert np.array_equal(r.components_pe, out["components"][1].numpy().transpose(0, 2, 1))
    assert np.array_equal(r.charge_components_pe, out["charge"][1].numpy())
    assert np.array_equal(r.time_origin_ns, out["origin"][1].numpy())
    assert np.array_equal(r.active, out["active"][1].numpy().astype(bool))
    r.charge_components_pe[:] = 0
    r.time_origin_ns[:] = 0
    assert np.all(out["charge"][1].numpy() != 0) and np.all(out["origin"][1].numpy() != 0)
