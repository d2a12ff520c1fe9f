"""The pieces of the FP64 solve that must round as the reference does: the
parallel left-to-right sum (closim_b200/csrc/ordered_sum.cuh) equals the
sequential loop bit for bit: its chunk maps on the CPU, the block-wide sum on a
GPU, on sums that cross many binades, cancel, tie, vanish or overflow; the division
by a shared divisor (div_rn.cuh) equals the IEEE quotient; the solve itself
(pcg64.cu) equals the oracle's at the edges of its launch shapes."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PTR = np.ctypeslib.ndpointer(np.float64, flags="C_CONTIGUOUS")


@pytest.fixture(scope="module")
def hc():
    subprocess.run(["make", "-s", "-C", os.path.join(HERE, "hostcheck")], check=True)
    L = C.CDLL(os.path.join(HERE, "hostcheck", "libhostcheck.so"))
    L.hc_ordered_maps.restype = C.c_double
    L.hc_ordered_maps.argtypes = [PTR, C.c_int, C.c_double, C.POINTER(C.c_int)]
    L.hc_gpu_ordered_sum.argtypes = [PTR, C.c_int, C.c_int, PTR]
    L.hc_div_rn.argtypes = [PTR, PTR, C.c_int, PTR]
    L.hc_pcg64_smem.restype = C.c_int64
    return L


def sequential(t):
    return np.cumsum(np.concatenate([[0.0], t]))[-1]  # numpy's cumulative sum adds left to right


def arrays(n):
    rng = np.random.default_rng(n)
    half = np.ldexp(rng.integers(1, 64, n).astype(np.float64), -53)
    yield "positive", rng.random(n)
    yield "signed", rng.normal(size=n)
    yield "drifting", rng.normal(size=n) + 0.05
    yield "negative", -np.exp(rng.normal(0.0, 12.0, n))
    yield "ties", np.where(np.arange(n) == 0, 1.0, half)  # half-ulp steps of a sum near 1
    yield "ties signed", np.where(np.arange(n) == 0, 1.5, half * rng.choice([-1.0, 1.0], n))
    yield "at a power of two", np.where(np.arange(n) == 0, 2.0, rng.normal(0.0, 1e-14, n))
    yield "zeros", np.zeros(n)
    yield "mostly zeros", np.where(rng.random(n) < 0.01, rng.normal(size=n), 0.0)
    yield "leading zeros", np.where(np.arange(n) < n // 2, 0.0, rng.random(n))
    yield "cancelling", np.where(np.arange(n) % 2 == 0, 1.0, -1.0) * (1 + rng.random(n) * 1e-9)
    yield "tiny", rng.random(n) * 1e-310
    yield "wide", rng.normal(size=n) * np.exp(rng.uniform(-80.0, 80.0, n))
    bad = rng.random(n)
    if n:
        bad[n // 2] = np.inf
    yield "infinite", bad
    bad = bad.copy()
    if n:
        bad[n // 3] = np.nan
    yield "nan", bad


def same_bits(a, b):
    return (np.isnan(a) and np.isnan(b)) or np.float64(a).tobytes() == np.float64(b).tobytes()


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1000, 12288])
def test_chunk_maps(hc, n):
    for name, t in arrays(n):
        for rel in (0.0, 1e-15, 3e-13):
            k = C.c_int(0)
            got = hc.hc_ordered_maps(np.ascontiguousarray(t), n, rel, C.byref(k))
            assert same_bits(got, sequential(t)), (name, rel)
            if n >= 1000 and name == "positive":
                assert k.value >= (n // 4) * 0.99  # the maps carry the sum, not the fallback


def test_division(hc):
    rng = np.random.default_rng(7)
    n = 400000
    a, b = rng.normal(size=n), rng.normal(size=n)
    a *= np.exp2(rng.integers(-40, 40, n))
    b[: n // 4] = rng.integers(1, 1 << 12, n // 4)  # short divisors: exact and half-way quotients
    a[: n // 4] = b[: n // 4] * (rng.integers(1, 1 << 40, n // 4) + 0.5)
    b[n // 4: n // 2] = np.nextafter(2.0, 0.0) * np.exp2(rng.integers(-3, 4, n // 4))  # all-ones significands
    a[-6:] = [0.0, 1.0, np.inf, np.nan, 1e-300, 1e300]
    b[-5] = 1e-200
    out = np.zeros(n)
    with np.errstate(all="ignore"):
        want = a / b
    hc.hc_div_rn(a, b, n, out)
    said = ~np.isnan(out)  # the range it answers for
    assert said[:-6].all() and said[-6] and not said[-5:].any()
    assert np.array_equal(out[said], want[said])


@pytest.mark.parametrize("n,parts", [
    (1, 7), (4096, 7), (4097, 7), (120000, 7), (150000, 5), (6000000, 5), (6710000, 5), (6800000, 4),
    (7000000, 4), (30000000, 4),
])
def test_solve_fits_shared_memory_at_any_size(hc, n, parts):
    """The launch never asks for more than a CTA may take (227 KB less the kernel's
    static 22 KB): what does not fit stays in global memory."""
    kept = C.c_int(0)
    assert 0 < hc.hc_pcg64_smem(n, C.byref(kept)) <= (227 - 22) * 1024
    assert kept.value == parts


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,precond", [
    (1, 1, "schwarz"), (2, 1, "jacobi"), (7, 9, "mas2"), (10, 12, "jacobi"),   # one CTA
    (15, 15, "jacobi"), (15, 15, "mas2"), (42, 5, "jacobi"), (42, 5, "schwarz"),  # the last alone, the first cluster
    (63, 63, "schwarz"), (64, 63, "schwarz"), (64, 63, "jacobi"),              # the last cluster, the first grid
    (255, 70, "mas2"), (300, 299, "jacobi"),                                   # element results in memory
    (500, 399, "jacobi"),                                                      # vectors in memory too
])
def test_solve_at_launch_edges(nx, ny, precond):
    import closim_b200 as cb
    from closim_b200 import configs
    from tests.helpers import oracle_scene, oracle_step_kwargs
    cfg = configs.strip_pull(nx=nx, ny=ny, w=0.025 * nx, hgt=0.025 * ny)
    cfg["v"] = np.random.default_rng(3).normal(0.0, 0.01, cfg["x"].size)
    cfg["options"] = dict(newtonIters=2, pcgMaxIters=5, gradTol=1e-6, lineSearchIters=4, precond=precond)
    pins = configs.pins_at(cfg, 0)
    sc = configs.make_scene(cfg)
    s = cb.CudaSolver("fp64", **cfg["options"])
    s.initialize(sc)
    s.step(cfg["h"])
    osc = oracle_scene(cfg)
    osc.set_pins(pins)
    st = osc.step(cfg["h"], **oracle_step_kwargs(cfg))
    assert s.lastStats.pcgIters == st["pcgIters"]
    assert np.array_equal(sc.positions, osc.positions)
    assert np.array_equal(sc.velocities, osc.velocities)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [0, 1, 127, 128, 129, 1024, 1025, 3968, 3969, 12288, 196608, 200001])
def test_block_sum(hc, n):
    for name, t in arrays(n):
        out = np.zeros(1)
        for brief in range(2 if n <= 1024 else 1):  # short sums: by stages, and by one thread
            assert hc.hc_gpu_ordered_sum(np.ascontiguousarray(t), n, brief, out) == 0
            assert same_bits(out[0], sequential(t)), (name, brief)
