"""The FP32 volume scatter over the range of its cotangents, on rays that share no voxel, so that a
gradient is each ray's own sums and repeats bit for bit."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from dpt_b200.geometry import BatchedGeometry, ParallelGeometry
from dpt_b200.phantoms import centred_grid
from dpt_b200.plan import plan_rays
from dpt_b200.projection import ProjectionSpec, ProjectionWorkspace
from oracle import oracle as O
from scenes import cone_scene, poses_for

pytestmark = pytest.mark.gpu
SAMPLES = 97


def apart():
    """One view of 4 x 8 rays (one warp) about four voxels apart."""
    grid, geometry, values = cone_scene(shape=(40, 44, 48), spacing=(1.0, 1.0, 1.0), views=1, detector=(4, 8),
                                        pitch=(8.0, 8.0))
    poses = poses_for(1, seed=3)
    ws = ProjectionWorkspace(plan_rays(grid, geometry), ProjectionSpec(SAMPLES, precision="float32",
                             sampling_precision="float32"), "cuda:0")
    return ws, values, poses


def gradient(ws, values, poses, seeds, pose=None):
    field = torch.tensor(values, dtype=torch.float32, device="cuda:0")
    cot = torch.tensor(seeds, dtype=torch.float32, device="cuda:0").reshape(ws.plan.image_shape)
    volume, _ = ws.vjp(field, torch.tensor(poses, device="cuda:0"), cot, volume=True, pose=pose)
    return volume.double().cpu().numpy().reshape(-1)


@pytest.mark.parametrize("pose", [None, "matrix"])
def test_gradient_scales_exactly_with_a_power_of_two(pose):
    """Seeds of 1e-3 and 2^10, 2^40 and 2^80 times that take the same sums: every rounding scales."""
    ws, values, poses = apart()
    seeds = np.random.default_rng(8).uniform(0.5e-3, 1e-3, ws.plan.rays).astype(np.float32)
    expected = gradient(ws, values, poses, seeds, pose)
    assert np.count_nonzero(expected) > 1000
    for power in (10, 40, 80):
        np.testing.assert_array_equal(gradient(ws, values, poses, seeds * np.float32(2.0**power), pose),
                                      expected * 2.0**power)


def test_seeds_of_every_size_in_one_warp_match_the_oracle():
    """2e-6 of each size's own norm, the bar of the other parity tests, where no other size reaches."""
    ws, values, poses = apart()
    sizes = (1e-3, 1.0, 100.0, 1e27, 1e30)  # below, at and above one; beyond the loop without tests
    rng = np.random.default_rng(9)
    order = rng.permutation(np.arange(ws.plan.rays) % len(sizes))
    seeds = (rng.uniform(0.5, 1.0, ws.plan.rays) * np.take(sizes, order)).astype(np.float32)
    actual = gradient(ws, values, poses, seeds)
    parts = [O.vjp(ws.plan, values, poses, np.where(order == k, seeds, np.float32(0)), samples=SAMPLES,
                   flags=O.VJP_VOLUME, arith=O.ARITH_F32)[0] for k in range(len(sizes))]
    touched = sum((part != 0).astype(int) for part in parts)
    for part in parts:
        own = (part != 0) & (touched == 1)
        assert own.sum() > 100
        assert np.linalg.norm(actual[own] / part.max() - part[own] / part.max()) <= 2e-6 * np.linalg.norm(part[own] / part.max())
    assert not actual[touched == 0].any()


@pytest.mark.parametrize("sampling", ["float32", "float64"])
def test_a_rays_increments_do_not_depend_on_its_warp(sampling):
    """A warp with a ray along a face marches every sample in one clamped loop, without one margin
    samples and interior pairs apart: both form the same sums, bit for bit."""
    grid = centred_grid((40, 44, 48), (1.0, 1.0, 1.0))
    # along x; the last column 0.27 beyond the outer voxel centres, inside the half-cell support
    panel = ParallelGeometry((40.0, 21.77 - 7 * 5.93, -12.31), (1.0, 0.0, 0.0), 80.0, (0.0, 1.0, 0.0), (0.0, 0.0, 1.0),
                             (5.93, 7.07), (4, 8))
    precision = "float64" if sampling == "float64" else "float32"
    ws = ProjectionWorkspace(plan_rays(grid, BatchedGeometry((panel,))),
                             ProjectionSpec(SAMPLES, precision=precision, sampling_precision=sampling), "cuda:0")
    dtype = torch.float64 if precision == "float64" else torch.float32
    field = torch.rand(grid.shape, device="cuda:0")
    pose = torch.tensor([[1.0, 0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0]], dtype=torch.float64, device="cuda:0")
    seeds = torch.linspace(0.3, 1.7, 32, dtype=dtype, device="cuda:0").reshape(ws.plan.image_shape)
    together, _ = ws.vjp(field, pose, seeds, volume=True, pose=None)
    apart = torch.zeros_like(together)
    for ray in range(32):
        one = torch.zeros_like(seeds)
        one.view(-1)[ray] = seeds.view(-1)[ray]
        alone, _ = ws.vjp(field, pose, one, volume=True, pose=None)
        # 48 voxels along x by two in z and, off the face, two in y, of no other ray
        assert not bool(((alone != 0) & (apart != 0)).any())
        assert int((alone != 0).sum()) == (96 if ray % 8 == 7 else 192)
        apart += alone
    torch.testing.assert_close(together, apart, rtol=0, atol=0)
