"""Which wave lookups take the short form (hydro_device.cuh): every point whose
texel indices lie in the grid, whatever the grid's size."""
import os
import subprocess

import numpy as np
import pytest

from stonefish_gb300 import abi, scenarios

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "stonefish_gb300", "csrc")

PROGRAM = """
#include <cstdio>
#include "hydro_device.cuh"
int main()
{
    long wrong = 0;
    for (uint32_t N : {2u, 3u, 7u, 100u, 384u, 600u, 1000u, 1024u, 65536u}) {
        const uint32_t at[] = {0u, N / 3u, N / 2u, N - 1u, N, N + 1u, 0xFFFFFFFFu};
        for (uint32_t a : at) for (uint32_t b : at) for (uint32_t c : at) for (uint32_t d : at)
            wrong += sfh::texels_in_grid(a, b, c, d, N) != (a < N && b < N && c < N && d < N);
    }
    std::printf("%ld\\n", wrong);
    return 0;
}
"""


def test_indices_of_any_grid_size_are_recognised(tmp_path):
    src, exe = tmp_path / "texels.cu", tmp_path / "texels"
    src.write_text(PROGRAM)
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    r = subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I", CSRC,
                        "-I", abi.INCLUDE_DIR, str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout.strip() == "0"


def _points(rng, gs, N, count):
    """x coordinates in units of the grid: inside, just beside the wrap and the
    texel borders, beyond 2^21 grids, negative, and not finite."""
    u = rng.uniform(-3.0, 3.0, count)
    edge = rng.integers(-2, 3, count) + rng.choice([0.5 / N, -0.5 / N, 0.0, 1.0 - 0.5 / N], count)
    x = np.where(rng.uniform(size=count) < 0.5, u, edge).astype(np.float32) * np.float32(gs)
    for _ in range(3):
        step = rng.uniform(size=count) < 0.4
        x = np.where(step, np.nextafter(x, np.float32(rng.choice([-1e9, 1e9]))), x).astype(np.float32)
    far = rng.uniform(size=count)
    x = np.where(far < 0.03, x * np.float32(3e7), np.where(far < 0.05, x + np.float32(2.0 ** 21 * gs), x))
    return x.astype(np.float32)


@pytest.mark.gpu
@pytest.mark.parametrize("N,layers", [(2, 1), (3, 1), (100, 1), (384, 2), (600, 1), (1000, 2), (1024, 2)])
def test_lookups_match_oracle_on_any_grid(oracle, built_library, N, layers):
    """Depths (one point at a time) bit for bit, and fluid positions, whose
    corners are looked up in pairs; the short and the general form meet in
    both."""
    from stonefish_gb300.hydro import HydroContext
    rng = np.random.default_rng(N)
    waves = {"data": rng.normal(size=(N, N, layers)).astype(np.float32),
             "layers": [(l, 0.1 * N / (1 + 2 * l)) for l in range(layers)]}
    waves["layers"] = [(c, float(np.float32(g))) for c, g in waves["layers"]]
    gs = waves["layers"][0][1]
    ocean = scenarios.flat_ocean()
    ocean.waves = 1
    pts = np.stack([_points(rng, gs, N, 4000), _points(rng, gs, N, 4000), rng.uniform(-2, 2, 4000)], 1).astype(np.float32)
    pts[:6, 0] = [np.nan, np.inf, -np.inf, 3e38, -3e38, 1e-44]
    pts[6:9, 1] = [np.nan, np.inf, -3e38]
    h = HydroContext(0)
    try:
        h.set_wave_grid(waves)
        got = h.depth(ocean, pts)
        with np.errstate(all="ignore"):
            ref = np.array([oracle.depth(ocean, waves, *map(float, p)) for p in pts], dtype=np.float32)
        assert np.array_equal(got, ref, equal_nan=True)
        lo = pts[9:1009].astype(np.float64)
        lo[:, 2] *= 0.5
        hi = lo + rng.uniform(0.0, 0.3, lo.shape)
        want = [oracle.fluid_position(ocean, a, b, waves) for a, b in zip(lo, hi)]
        assert _positions(h, ocean, lo, hi).tolist() == [w == abi.INSIDE for w in want]
        assert len(set(want)) == 3
    finally:
        h.close()


def _positions(h, ocean, lo, hi):
    """INSIDE states (hydro_nn_gate_inside rejects them)."""
    import ctypes as C

    import torch
    from stonefish_gb300 import surrogate as S
    b = S.sample_states(np.random.default_rng(0), len(lo))
    b["aabb_min"], b["aabb_max"] = lo, hi
    d_b = torch.from_numpy(b.view(np.uint8).copy()).cuda()
    mask = torch.ones(len(lo), dtype=torch.uint8, device="cuda")
    h._ck(h.lib.hydro_nn_gate_inside(h.ctx, S._ptr(d_b), len(lo), C.byref(ocean), S._ptr(mask), None))
    torch.cuda.synchronize()
    return mask.cpu().numpy() == 0


@pytest.mark.gpu
def test_grid_of_one_texel(oracle, built_library):
    """One texel of two channels: both fractions round up to one beside the
    wrap, and the index wraps back to the texel."""
    from stonefish_gb300.hydro import HydroContext
    waves = {"data": np.array([[[0.75, -0.5]]], dtype=np.float32), "layers": [(0, 4.0), (1, 8.0)]}
    ocean = scenarios.flat_ocean()
    ocean.waves = 1
    u = np.concatenate([[0.5], np.nextafter(np.float32(0.5), np.float32([0, 1])), [-0.5, 0.0, 3.25, 1e9]]).astype(np.float32)
    x, y = np.meshgrid(np.concatenate([u * 4, u * 8]), np.concatenate([u * 4, u * 8]))
    pts = np.stack([x.ravel(), y.ravel(), np.ones(x.size)], 1).astype(np.float32)
    h = HydroContext(0)
    try:
        h.set_wave_grid(waves)
        ref = np.array([oracle.depth(ocean, waves, *map(float, p)) for p in pts], dtype=np.float32)
        assert np.array_equal(h.depth(ocean, pts), ref)
    finally:
        h.close()
