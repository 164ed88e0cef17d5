"""The envelope grid's node responses at every row length of the register transform, with an odd
number of nodes (the last pair is half empty), one or two field components and one or two Raman
kernels, against the oracle."""

import dataclasses

import numpy as np
import pytest

from oracle import source as S
from solprop_b200 import _lib, grin
from tests._cases import rel


def _record(n_to, form, grid=3):
    rec, _ = grin.grin_record(n_to=n_to, grid=grid, seed=n_to)
    if form == "trace":
        return dataclasses.replace(rec, raman_tensor_weights=np.array([[1.0, 0.0]]))
    if form == "kerr":
        return dataclasses.replace(rec, raman_enabled=False, raman_undamped=None, raman_rates=[],
                                   raman_tensor_weights=None)
    if form == "scalar":
        return dataclasses.replace(
            rec, n_modes=15, n_pol_transform=1, phi_terms=rec.phi_terms[:, ::2], prefactor_terms=rec.prefactor_terms[:, ::2],
            synthesis=np.ascontiguousarray(rec.synthesis[::2, ::2]),
            projection=np.ascontiguousarray(rec.projection[::2, ::2]),
            projection_coarse=np.ascontiguousarray(rec.projection[::2, ::2]), raman_tensor_weights=None,
            field0=rec.field0[::2])
    return rec


# FP64 rows differ from the oracle by the transforms' rounding, a few 1e-16 log2 n; the mixed form
# by the FP32 transforms' and products' (the bounds of test_envelope_modal.py)
@pytest.mark.gpu
@pytest.mark.parametrize("precision, bound", [("fp64", 1e-13), ("mixed", 2e-6)])
@pytest.mark.parametrize("form", ["tensor", "trace", "scalar", "kerr"])
@pytest.mark.parametrize("n_to", [512, 1024, 2048, 4096, 8192, 16384])
def test_source_matches_oracle(n_to, form, precision, bound):
    rec = _record(n_to, form)
    rng = np.random.default_rng(n_to)
    lab = rec.launch_field()
    lab = (lab + 0.1 * np.exp(2j * np.pi * rng.uniform(size=(rec.n_modes, 1, 1))) * lab[:1]) * rec.active_mask
    ws = _lib.Workspace(_lib.Problem(rec), 0, precision)
    assert rel(ws.source(lab, 0.0), S.lab_source(rec, lab, 0.0)) < bound


# up to 148 nodes take a CTA each (above), more take one for two
@pytest.mark.gpu
@pytest.mark.parametrize("precision, bound", [("fp64", 1e-13), ("mixed", 2e-6)])
@pytest.mark.parametrize("form", ["tensor", "trace", "scalar"])
@pytest.mark.parametrize("n_to, grid", [(512, 12), (512, 13), (1024, 13), (2048, 13), (4096, 13), (8192, 13), (16384, 13)])
def test_many_nodes(n_to, grid, form, precision, bound):
    rec = _record(n_to, form, grid)
    lab = rec.launch_field()
    ws = _lib.Workspace(_lib.Problem(rec), 0, precision)
    assert rel(ws.source(lab, 0.0), S.lab_source(rec, lab, 0.0)) < bound


# Raman alone on a field whose cube overflows FP32 (above 7e12): no cubic is formed
@pytest.mark.gpu
@pytest.mark.parametrize("form", ["tensor", "trace", "scalar"])
@pytest.mark.parametrize("n_to", [512, 16384])
def test_strong_field_without_kerr(n_to, form):
    rec = dataclasses.replace(_record(n_to, form), kerr_enabled=False)
    lab = rec.launch_field()
    peak = np.abs(rec.synthesis @ np.fft.ifft(lab.reshape(rec.n_modes, -1), axis=-1)).max()
    lab = lab * (2e13 / peak)
    ws = _lib.Workspace(_lib.Problem(rec), 0, "mixed")
    assert rel(ws.source(lab, 0.0), S.lab_source(rec, lab, 0.0)) < 2e-6


# Two drives share a complex row: neighbouring nodes' traces, and one node's difference and
# coherence.  A mode of its own on each, fields 1e4 apart (drives 1e8), a continuous wave beside a
# pulse, or nothing at all beside one: the error of every mode's source against its own norm
@pytest.mark.gpu
@pytest.mark.parametrize("precision, bound", [("fp64", 1e-13), ("mixed", 2e-6)])
@pytest.mark.parametrize("form, rows", [("scalar", (2, 3)), ("trace", (4, 6)), ("tensor", (4, 6)), ("tensor", (4, 5))])
@pytest.mark.parametrize("first", ["pulse", "continuous", "none"])
@pytest.mark.parametrize("n_to", [512, 4096, 8192, 16384])
def test_uneven_drives_of_one_row(n_to, first, form, rows, precision, bound):
    rec = _record(n_to, form, 3 if rows == (4, 5) else 13)
    synthesis, projection = np.zeros((rec.synthesis.shape[0], 2)), np.zeros((2, rec.synthesis.shape[0]))
    for mode, row in enumerate(rows):
        synthesis[row, mode], projection[mode, row] = abs(rec.synthesis).max(), abs(rec.projection).max()
    rec = dataclasses.replace(
        rec, n_modes=2, phi_terms=rec.phi_terms[:, :2], prefactor_terms=rec.prefactor_terms[:, :2], synthesis=synthesis,
        projection=projection, projection_coarse=projection, kerr_enabled=False, absorber_scheme="none",
        temporal_absorber_fine=None, field0=rec.field0[:2])
    lab = rec.launch_field()
    lab[1] = 1e-4 * lab[0]
    if first == "continuous":
        peak = abs(lab[0]).argmax()
        lab[0], lab[0].flat[peak] = 0.0, abs(lab[0]).sum()
    elif first == "none":
        lab[0] = 0.0
    ws = _lib.Workspace(_lib.Problem(rec), 0, precision)
    got, want = ws.source(lab, 0.0), S.lab_source(rec, lab, 0.0)
    for mode in range(2):
        assert np.linalg.norm(got[mode] - want[mode]) <= bound * np.linalg.norm(want[mode]), mode


# the products: mode counts about the projections' 32- and 64-wide tiles and the synthesis's 16-
# and 64-wide K slices, rows of nodes that fill neither a tile nor a K slice
@pytest.mark.gpu
@pytest.mark.parametrize("precision, bound", [("fp64", 1e-13), ("mixed", 2e-6)])
@pytest.mark.parametrize("modes", [2, 32, 33, 64, 65, 130])
def test_products_at_mode_counts(modes, precision, bound):
    rec, _ = grin.grin_record(n_to=512, grid=13, seed=modes)
    idx = np.arange(modes) % rec.n_modes
    weight = np.random.default_rng(modes).uniform(0.5, 1.0, modes) * np.sqrt(30 / max(modes, 30))
    rec = dataclasses.replace(
        rec, n_modes=modes, phi_terms=rec.phi_terms[:, idx], prefactor_terms=rec.prefactor_terms[:, idx],
        synthesis=np.ascontiguousarray(rec.synthesis[:, idx] * weight),
        projection=np.ascontiguousarray(rec.projection[idx] * weight[:, None]),
        projection_coarse=np.ascontiguousarray(rec.projection[idx] * weight[:, None]), field0=rec.field0[idx])
    lab = rec.launch_field()
    ws = _lib.Workspace(_lib.Problem(rec), 0, precision)
    assert rel(ws.source(lab, 0.0), S.lab_source(rec, lab, 0.0)) < bound


# one mode on one node: the cluster kernel's row lengths, with and without the Raman halves
@pytest.mark.gpu
@pytest.mark.parametrize("raman", [True, False])
@pytest.mark.parametrize("n_to", [512, 1024, 2048, 4096])
def test_single_mode_source(n_to, raman):
    rec = _record(n_to, "scalar" if raman else "kerr")
    rec = dataclasses.replace(
        rec, n_modes=1, n_nodes=1, n_pol_transform=1, phi_terms=rec.phi_terms[:, :1],
        prefactor_terms=rec.prefactor_terms[:, :1], synthesis=np.array([[3e6]]), projection=np.array([[1 / 3e6]]),
        projection_coarse=np.array([[1 / 3e6]]), absorber_scheme="none", temporal_absorber_fine=None,
        field0=rec.field0[:1])
    lab = rec.launch_field()
    ws = _lib.Workspace(_lib.Problem(rec), 0)
    assert rel(ws.source(lab, 0.0), S.lab_source(rec, lab, 0.0)) < 1e-13
