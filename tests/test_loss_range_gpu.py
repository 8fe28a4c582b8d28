"""The loss in FP64 from a tile's columns on: residuals whose squares fit in float32,
but not the sum over a tile."""
import numpy as np
import pytest
import torch

from problems import engine_atoms, engine_geometry, make_atoms, make_geometry

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("psf", [False, True])
@pytest.mark.parametrize("kind,form", [("2d", 1), ("2p5d", 1), ("2p5d", 2)])
def test_loss_of_large_residuals(eng, cuda_ready, kind, form, psf):
    lib = __import__("importlib").import_module("2018_dictionary_tomography_gb300._lib")
    g = make_geometry(kind, 3, 70)
    atoms = engine_atoms(*make_atoms(2 if kind == "2d" else 3, 40, 7))
    geom = engine_geometry(g)
    # half a square is 8e36, a column of 32 cells 2.6e38, two columns beyond float32
    data = torch.full(geom.shape, 4e18, device="cuda")
    saved = lib.load().gr_get_tuning(3)
    lib.check(lib.load().gr_set_tuning(3, form), "gr_set_tuning")
    try:
        fw = eng.fit_forward(atoms, geom, data, "l2", psf=psf)
    finally:
        lib.check(lib.load().gr_set_tuning(3, saved), "gr_set_tuning")
    want = 0.5 * (fw["alpha"].double() ** 2).sum().item()
    assert abs(float(fw["loss"]) - want) < 1e-7 * want


@pytest.mark.parametrize("kind,D,psf,line", [("2d", (32, None), False, 5120), ("2d", (32, None), True, 5120),
                                             ("2p5d", (16, 32), True, 5120),
                                             ("2p5d", (16, 32), False, 12288)])
@pytest.mark.parametrize("more", [0, 1])
def test_loss_on_both_sides_of_the_fused_line(eng, cuda_ready, kind, D, psf, line, more):
    """A tile an angle: the most items that the projection's last block sums, and one more."""
    g = make_geometry(kind, line + more, *D)
    atoms = engine_atoms(*make_atoms(2 if kind == "2d" else 3, 3, 5))
    geom = engine_geometry(g)
    data = torch.rand(geom.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    fw = eng.fit_forward(atoms, geom, data, "l2", psf=psf)
    want = 0.5 * (fw["alpha"].double() ** 2).sum().item()
    assert abs(float(fw["loss"]) - want) < 1e-6 * want
