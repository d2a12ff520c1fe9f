"""The grid-wide resident PCG of the mixed path (k_mx_pcg_grid) against the
kernels it replaces there (the gathering cluster kernel, and past 20,000
vertices the element-scatter kernel), forced by CLOSIM_MX_RESIDENT=0.

Every vertex and element does the same FP32 operations in the same order; only
the FP64 dot products are summed in another order, which moves an FP32 alpha or
beta by an ulp when their ratio lies within 1e-16 of a rounding boundary, about
once in 1e8 iterations. So one step at the reference budget agrees to 1e-9 of
the positions' size, and a converged step to what gradTol leaves. Also which
kernel a solver says it runs."""
import numpy as np
import pytest

import closim_b200 as cb
from closim_b200 import configs

pytestmark = pytest.mark.gpu


def one_step(monkeypatch, resident, cfg, mode, **opts):
    if resident:
        monkeypatch.delenv("CLOSIM_MX_RESIDENT", raising=False)
    else:
        monkeypatch.setenv("CLOSIM_MX_RESIDENT", "0")
    s = cb.CudaSolver("mixed", **{**cfg["options"], **opts})
    sc = configs.make_scene(cfg)
    s.initialize(sc)
    s.setGraphMode(False)
    s.setNewtonMode(mode, 3e-4)
    s.step(cfg["h"])
    info, st = s.launchInfo(), s.lastStats
    s.close()
    return sc.positions.copy(), st, info


@pytest.mark.parametrize("nx,ny,precond,mode", [
    (65, 64, "mas2", "exact"),           # just past the cluster's lists in this mode
    (99, 84, "schwarz", "reference"),
    (1050, 3, "schwarz", "exact"),       # a ribbon: many vertices of the halo per owned one
    (79, 71, "jacobi", "reference"),
    (150, 140, "schwarz", "reference"),  # past 20,000 vertices
    (255, 252, "schwarz", "reference"),  # near the most shared memory takes
])
def test_grid_pcg_matches_the_kernels_it_replaces(monkeypatch, nx, ny, precond, mode):
    cfg = configs.floor_drape(nx=nx, ny=ny, w=0.0127 * nx, hgt=0.0127 * ny, height=0.002, precond=precond)
    cfg["v"] = np.tile([0.3, -0.1, 0.1], cfg["x"].size // 3)
    cfg["fixed_pins"] = [0, nx]
    opts = dict(newtonIters=30, pcgMaxIters=2000, gradTol=1e-9) if mode == "exact" else {}
    x1, st1, info = one_step(monkeypatch, True, cfg, mode, **opts)
    x0, st0, old = one_step(monkeypatch, False, cfg, mode, **opts)
    assert info["pcgKernel"] == "k_mx_pcg_grid"
    assert old["pcgKernel"] == ("k_mx_pcg_cluster" if (nx + 1) * (ny + 1) <= 20000 else "k_mx_pcg")
    assert st1.contact["floorPairs"] > 0
    assert st1.newtonItersUsed == st0.newtonItersUsed and st1.pcgIters == st0.pcgIters
    assert np.max(np.abs(x1 - x0)) <= 1e-9 * np.max(np.abs(x0))


@pytest.mark.parametrize("mode", ["reference", "exact"])
def test_grid_pcg_with_many_contacts_per_vertex(monkeypatch, mode):
    """A sheet sliding over the pole of a finely divided sphere, where 64 edges
    meet: vertices with more than four contact records, which a warp sums. That
    there are some follows from the counts: the records (one per vertex-triangle
    pair at the least, two per edge-edge pair) outnumber four for every vertex
    within reach of the sphere. (A converged exact step lifts the sheet off again, so
    that one stops after two Newton iterations.)"""
    cell = 0.003
    cfg = configs.sphere_drape(nx=84, ny=79, w=84 * cell, hgt=79 * cell, radius=0.1, drop=0.1004, segments=64, rings=32)
    cfg["contact"]["dHatM"] = 1e-3
    cfg["v"][0::3] = 0.2
    cfg["v"][1::3] = -0.05
    opts = dict(newtonIters=2, pcgMaxIters=2000, gradTol=1e-9) if mode == "exact" else {}
    x1, st1, info = one_step(monkeypatch, True, cfg, mode, **opts)
    x0, st0, old = one_step(monkeypatch, False, cfg, mode, **opts)
    assert info["pcgKernel"] == "k_mx_pcg_grid" and old["pcgKernel"] == "k_mx_pcg_cluster"
    far = np.linalg.norm(cfg["x"].reshape(-1, 3) - np.asarray(cfg["sphere"]["centre"]), axis=1) - 0.1
    near = int(np.count_nonzero(far < 1e-3 + 3 * cell))
    assert st1.contact["vtPairs"] + 2 * st1.contact["eePairs"] > 4 * near > 0
    assert st1.newtonItersUsed == st0.newtonItersUsed and st1.pcgIters == st0.pcgIters
    assert np.max(np.abs(x1 - x0)) <= 1e-9 * np.max(np.abs(x0))


@pytest.mark.parametrize("precision,nx,ny,precond,mode,kernel", [
    ("mixed", 63, 63, "schwarz", "exact", "k_mx_pcg_cluster"),
    ("mixed", 69, 69, "schwarz", "reference", "k_mx_pcg_cluster"),  # the lists fit one cluster without the hinges,
    ("mixed", 69, 69, "schwarz", "exact", "k_mx_pcg_grid"),         # with them they do not
    ("mixed", 69, 69, "jacobi", "reference", "k_mx_pcg_grid"),      # the resident cluster kernel has no Jacobi
    ("mixed", 39, 39, "jacobi", "reference", "k_mx_pcg_cluster"),
    ("mixed", 150, 140, "schwarz", "reference", "k_mx_pcg_grid"),
    ("mixed", 150, 140, "schwarz", "exact", "k_adj_pcg"),
    ("fp64", 20, 20, "schwarz", "reference", "k_pcg64"),
    ("fp64", 20, 20, "schwarz", "exact", "k_adj_pcg"),
])
def test_launch_info_names_the_kernel(precision, nx, ny, precond, mode, kernel):
    cfg = configs.floor_drape(nx=nx, ny=ny, w=0.0127 * nx, hgt=0.0127 * ny, precond=precond)
    s = cb.CudaSolver(precision, **cfg["options"])
    s.initialize(configs.make_scene(cfg))
    s.setNewtonMode(mode, 3e-4)
    info = s.launchInfo()
    s.close()
    assert info["pcgKernel"] == kernel
    if precision == "mixed" and kernel != "k_adj_pcg":
        assert (info["pcgClusterCtas"] > 0) == (kernel == "k_mx_pcg_cluster")
