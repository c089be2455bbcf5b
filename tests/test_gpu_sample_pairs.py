"""The interior sample loops (pairs of FP32 samples, predicated corner reloads and run flushes) and
the compensated cell walk where they can go wrong: axes of one and two samples (no interior), one, two and three interior
samples, power-of-two and odd extents, one sample per ray and many per cell.

Images are bit for bit the oracle's; volume gradients agree to FP32 summation order, the bar of
the other parity tests (2e-6 relative L2), pose gradients to FP64 reduction order (1e-9)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from dpt_b200 import _native as N
from dpt_b200.plan import plan_rays
from dpt_b200.projection import ProjectionSpec, ProjectionWorkspace
from oracle import oracle as O
from scenes import cone_scene, poses_for

pytestmark = pytest.mark.gpu

ARITH = {"float32": O.ARITH_F32, "float64": O.ARITH_F64, "compensated": O.ARITH_F32C}


@pytest.mark.parametrize("sampling", ["float32", "float64", "compensated"])
@pytest.mark.parametrize("samples", [1, 2, 64, 257])
@pytest.mark.parametrize("shape", [(2, 2, 2), (1, 9, 3), (3, 1, 8), (16, 32, 64), (5, 21, 33)])
def test_interior_loops_match_the_oracle(shape, samples, sampling):
    grid, geometry, values = cone_scene(shape=shape, spacing=(0.9, 1.0, 1.1), views=3, detector=(11, 13),
                                        pitch=(3.0, 3.0))
    poses = poses_for(3, seed=21)
    precision, image_dtype = ("float64", O.F64) if sampling == "float64" else ("float32", O.F32)
    ws = ProjectionWorkspace(plan_rays(grid, geometry), ProjectionSpec(samples, precision=precision,
                             sampling_precision=sampling), "cuda:0")
    field = torch.tensor(values.astype(np.float32), device="cuda:0")
    pose = torch.tensor(poses, device="cuda:0")
    image = ws.forward(field, pose).cpu().numpy().reshape(-1)
    expected, _ = O.forward(ws.plan, values, poses, samples=samples, arith=ARITH[sampling], image_dtype=image_dtype)
    np.testing.assert_array_equal(image, expected)
    assert np.abs(expected).sum() > 0
    seed = np.random.default_rng(5).uniform(-1.0, 1.0, ws.plan.rays).astype(image.dtype)
    cot = torch.tensor(seed, device="cuda:0").reshape(ws.plan.image_shape)
    e_volume, e_pose, _ = O.vjp(ws.plan, values, poses, seed, samples=samples, flags=O.VJP_VOLUME | O.VJP_POSE12,
                                arith=ARITH[sampling], image_dtype=image_dtype)
    norm = np.linalg.norm(e_volume)
    for moments, want_pose in ((False, False), (False, True), (True, True)):
        ws.forward(field, pose, moments=moments)
        volume, pose_grad = ws.vjp(field, pose, cot, volume=True, pose="matrix" if want_pose else None)
        assert np.linalg.norm(volume.cpu().numpy().reshape(-1) - e_volume) <= 2e-6 * norm
        if want_pose:
            np.testing.assert_allclose(pose_grad.cpu().numpy(), e_pose, rtol=1e-9, atol=1e-12)


@pytest.mark.parametrize("offset", [0, 16, 32])
@pytest.mark.parametrize("sampling", ["float32", "compensated"])
def test_field_copies_at_every_alignment_the_abi_accepts(sampling, offset):
    """A copy that starts on a 16-byte but not a 32-byte boundary takes the narrower stores: the
    forward that reads it equals the workspace's own bit for bit."""
    grid, geometry, values = cone_scene(shape=(5, 7, 37))
    poses = poses_for(len(geometry.views), seed=22)
    ws = ProjectionWorkspace(plan_rays(grid, geometry), ProjectionSpec(50, sampling_precision=sampling), "cuda:0")
    field = torch.tensor(values.astype(np.float32), device="cuda:0")
    pose = torch.tensor(poses, device="cuda:0")
    expected = ws.forward(field, pose)
    lib = N.library()
    size = lib.dpt_b200_packed_bytes(ws.problem)
    buffer = torch.zeros(size + 64, dtype=torch.uint8, device="cuda:0")
    copy = buffer.data_ptr() + offset  # the allocator aligns to at least 32 bytes
    stream = torch.cuda.current_stream().cuda_stream
    image = torch.empty_like(expected)
    N.check(lib.dpt_b200_prepare_field(ws.problem, field.data_ptr(), copy, pose.data_ptr(), ws.status.data_ptr(),
                                       stream), "prepare_field")
    N.check(lib.dpt_b200_forward(ws.problem, ws.rays(pose), copy, image.data_ptr(), ws.status.data_ptr(), stream),
            "forward")
    torch.testing.assert_close(image, expected, rtol=0, atol=0)
    assert int(buffer[:offset].sum()) == 0 and int(buffer[offset + size:].sum()) == 0
