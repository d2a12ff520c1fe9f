"""Per-CTA element lists of the one-cluster PCG's resident phase A, and the
batched solver's choice between clusters and lone blocks (host logic).

The builder (closim_b200/csrc/cluster_plan.cpp) is compiled for the host with
a checker of its invariants (tests/plancheck): the owned vertex ranges cover
the mesh; every owned vertex's triangle and hinge incidences appear in the
membrane and hinge CSRs' order and point at list slots whose halo-local ids
map back to the right global vertices; every listed element touches an owned
vertex; shared-memory regions are 16-byte aligned; every vertex's dofs are
pushed to the phase-B slot of the warp that owns its Schwarz domain. Meshes: the floor drape's
64 x 64 grid (which must fit in a CTA's shared memory at 16 CTAs), the strip,
an irregular annulus and a UV sphere.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from closim_b200 import configs
from tests.test_gpu_garment import annulus

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "plancheck", "libplancheck.so")
SMEM_LIMIT = 227 * 1024 - 4096  # the kernel's dynamic shared-memory budget per CTA


@pytest.fixture(scope="module")
def lib():
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "plancheck")], check=True)
    L = ctypes.CDLL(LIB)
    L.pc_check.restype = ctypes.c_int
    return L


def check(L, mesh, nrank):
    idx = np.ascontiguousarray(mesh.indices, dtype=np.uint32)
    hin = np.ascontiguousarray(np.asarray(mesh.hinges, dtype=np.int32).reshape(-1))
    n = len(mesh.restPositions) // 3
    info = np.zeros(7, dtype=np.int64)
    rest = np.ascontiguousarray(mesh.restPositions, dtype=np.float32)
    rc = L.pc_check(n, len(idx) // 3, len(hin) // 4, idx.ctypes.data_as(ctypes.c_void_p),
                    hin.ctypes.data_as(ctypes.c_void_p), rest.ctypes.data_as(ctypes.c_void_p), nrank,
                    info.ctypes.data_as(ctypes.c_void_p))
    return rc, info


def scene_mesh(cfg):
    return configs.make_scene(cfg).mesh


def test_plan_invariants_floor_drape(lib):
    rc, info = check(lib, scene_mesh(configs.floor_drape()), 16)
    assert rc == 0, rc
    print(f"64x64 at 16 CTAs: shared memory {info[0]} B (reference mode), {info[1]} B (exact-Newton mode)")
    assert info[1] <= SMEM_LIMIT, info


@pytest.mark.parametrize("nrank", [8, 1])
def test_plan_refused_when_a_warp_would_own_more_than_three_domains(lib, nrank):
    # 513 Schwarz domains need at least 171 warps (3 domains each): 16 per CTA
    rc, _ = check(lib, scene_mesh(configs.floor_drape()), nrank)
    assert rc == 1, rc


def test_plan_invariants_strip_and_sphere(lib):
    for cfg in (configs.strip_pull(), configs.sphere_drape(nx=31, ny=31)):
        rc, _ = check(lib, scene_mesh(cfg), 16)
        assert rc == 0, (cfg["name"], rc)


def test_plan_invariants_irregular_mesh(lib):
    from closim_b200.garment import AssembledGarment
    from closim_b200.solver import preprocess
    pos, uv, idx = annulus()
    mesh = preprocess(pos.astype(np.float32), uv.astype(np.float32), idx.astype(np.uint32), 0.15)
    for nrank in (16, 4, 3):
        rc, _ = check(lib, mesh, nrank)
        assert rc == 0, (nrank, rc)


def test_plan_more_ctas_than_vertices(lib):
    # a 3 x 3 sheet over 16 CTAs: most CTAs own nothing
    cfg = configs.floor_drape(nx=2, ny=2, w=0.1, hgt=0.1, steps=2)
    rc, info = check(lib, scene_mesh(cfg), 16)
    assert rc == 0, rc


@pytest.mark.parametrize("nx,ny,nrank,fits", [
    (63, 63, 16, True), (99, 84, 16, True), (134, 108, 16, False),  # one cluster (its domains aside)
    (134, 108, 148, True), (255, 255, 148, True), (419, 419, 148, False), (1050, 3, 100, True),
])
def test_counted_bound_of_the_lists(lib, nx, ny, nrank, fits):
    """The bound that spares building lists which cannot fit is one: never above
    what the built lists need, and above the limit where they are far from fitting."""
    mesh = scene_mesh(configs.floor_drape(nx=nx, ny=ny, w=0.0127 * nx, hgt=0.0127 * ny))
    idx = np.ascontiguousarray(mesh.indices, dtype=np.uint32)
    hin = np.ascontiguousarray(np.asarray(mesh.hinges, dtype=np.int32).reshape(-1))
    info = np.zeros(4, dtype=np.int64)
    rc = lib.pc_least(len(mesh.restPositions) // 3, len(idx) // 3, len(hin) // 4, idx.ctypes.data_as(ctypes.c_void_p),
                      hin.ctypes.data_as(ctypes.c_void_p), nrank, info.ctypes.data_as(ctypes.c_void_p))
    assert rc == 0
    assert 0 < info[0] <= info[1] and 0 < info[2] <= info[3] and info[0] <= info[2]
    assert (info[0] <= SMEM_LIMIT) == fits, info


@pytest.mark.parametrize("sides,sizes", [
    ([64] * 9, (4, 1, 1)), ([64] * 37, (4, 1, 1)), ([64] * 74, (4, 1, 1)), ([64] * 148, (1, 1, 1)),
    ([64] * 296, (1, 1, 1)), ([80] * 74, (4, 1, 1)), ([80] * 148, (1, 1, 1)), ([55] * 37, (4, 1, 1)),
    ([55] * 74, (1, 1, 1)), ([55] * 111, (1, 1, 1)), ([55] * 148, (1, 1, 1)), ([45] * 74, (1, 2, 1)),
    ([45] * 111, (1, 1, 1)), ([45] * 148, (1, 1, 1)), ([38] * 400, (1, 1, 1)),
    ([16 + i % 113 for i in range(0, 113, 2)], (4, 1, 1)), ([16 + i * 7 % 113 for i in range(512)], (1, 1, 1)),
])
def test_batch_route(lib, sides, sizes):
    """Clusters or lone blocks as the measured times (batch_plan.hpp) say, on a
    device of 148 SMs that holds 33 clusters of four and 74 of two; lone blocks
    where no cluster fits."""
    verts = np.array([s * s for s in sides], np.int32)
    out = np.zeros(3, np.int32)
    p = ctypes.c_void_p
    lib.pc_batch_route(verts.ctypes.data_as(p), len(verts), 148, 33, 74, out.ctypes.data_as(p))
    assert tuple(out) == sizes
    lib.pc_batch_route(verts.ctypes.data_as(p), len(verts), 148, 0, 0, out.ctypes.data_as(p))
    assert tuple(out) == (1, 1, 1)
