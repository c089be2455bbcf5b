"""State kept between calls, where no GPU is needed to show it sound: what every later call may read
is complete when it is stored, and is ordered after the stream that wrote it."""

from __future__ import annotations

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from dpt_b200.geometry import RigidTransform
from dpt_b200.torch import Projector
from scenes import cone_scene

ANCHORS = [None, RigidTransform(translation_mm=(1.0, -2.0, 3.0))]


class DeviceInputs(TorchDispatchMode):
    """Names of the operators that read a device tensor: kernels, ordered by their stream alone."""

    def __init__(self, device: str) -> None:
        super().__init__()
        self.device = device
        self.names: list[str] = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        name = func.overloadpacket.__name__
        if name not in ("lift_fresh", "detach") and any(
                isinstance(a, torch.Tensor) and a.device.type == self.device for a in args):
            self.names.append(name)
        return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("anchor", ANCHORS)
def test_poses_of_a_fixed_anchor_are_uploaded_whole(anchor):
    grid, geometry, _ = cone_scene(views=3)
    projector = Projector(grid=grid, geometry=geometry, samples_per_ray=4, anchor=anchor)
    field = torch.empty(grid.shape, device="meta")
    with DeviceInputs("meta") as kernels:
        poses = projector._packed_poses(field, None, None)
    assert tuple(poses.shape) == (3, 12) and poses.is_contiguous()
    assert kernels.names == []
    assert projector._packed_poses(field, None, None) is poses
    rows = projector._fixed_anchor.on(torch.device("cpu"), 3)
    assert rows.tolist() == [list((anchor or RigidTransform()).packed())] * 3


def test_poses_first_used_in_inference_mode_can_be_saved_for_backward():
    grid, geometry, _ = cone_scene(views=2)
    projector = Projector(grid=grid, geometry=geometry, samples_per_ray=4)
    field = torch.empty(grid.shape)
    with torch.inference_mode():
        projector._packed_poses(field, None, None)
        projector._packed_poses(field, torch.zeros(6, dtype=torch.float64), None)
    assert not projector._packed_poses(field, None, None).is_inference()
    assert not projector._anchor_on(field.device).is_inference()
