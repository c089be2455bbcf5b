"""State kept between calls, and the operators' registration, where no GPU is needed to show them
sound: what a later call may read is complete when it is stored, and is ordered after the stream that
wrote it; a gradient that does not exist is an error."""

from __future__ import annotations

import contextlib
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from dpt_b200._device import StatusWord
from dpt_b200.geometry import RigidTransform
from dpt_b200.projection import ProjectionSpec, ProjectionWorkspace
from dpt_b200.torch import Projector, _projection_ops
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


CAPTURING = 9  # handle of the stand-in stream that captures


class FakeStream:
    def __init__(self, handle: int) -> None:
        self.cuda_stream = handle

    def synchronize(self) -> None:
        pass


@pytest.fixture
def word(monkeypatch):
    """A status word on the host with stand-in streams; ``copies`` lists the stream each readback
    was queued on."""
    at = [1]

    @contextlib.contextmanager
    def stream(s):
        at.append(s.cuda_stream)
        yield
        at.pop()

    zeros = torch.zeros
    monkeypatch.setattr(torch, "zeros", lambda *a, pin_memory=False, **k: zeros(*a, **k))
    monkeypatch.setattr(torch.cuda, "stream", stream)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: at[-1] == CAPTURING)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda device: at[-1], raising=False)
    status = StatusWord(torch.device("cpu"))
    status.copies = []
    copy = status.host.copy_

    class Host:
        def copy_(self, source, non_blocking=False):
            status.copies.append(at[-1])
            return copy(source)

        def __getitem__(self, index):
            return status.host_values[index]

    status.host_values, status.host = status.host, Host()
    return status


def report(word, stream, address, handle) -> int:
    """A C-ABI call that reports 8."""
    assert (address, handle) == (word.word.data_ptr(), stream.cuda_stream)
    word.word.fill_(8)
    return 0


def test_status_word_is_read_on_the_stream_that_writes_it(word):
    side = FakeStream(2)
    word.launch(side, "report", lambda address, stream: report(word, side, address, stream))
    assert word.read(side) == 8 and word.pending(side) == 8  # sticky until reset
    assert word.pending(side, reset=True) == 8 and word.pending(side) == 0
    assert int(word.word) == 0 and word.copies == [2, 2, 2]


def test_status_word_stays_pending_until_its_own_stream_was_read_clean(word):
    side, other = FakeStream(2), FakeStream(3)
    assert word.pending(side) == 0 and word.copies == []  # no launch: no wait
    # another thread's read before the launch is queued
    word.launch(side, "nothing", lambda address, stream: word.read(side) and 1)
    assert word.pending(side) == 0 and word.copies == [2, 2]
    word.launch(side, "nothing", lambda address, stream: 0)
    word.read(other)  # ordered after another stream only
    word.clear(other)
    word.word.fill_(2)  # the launch reports now
    assert word.pending(other) == 2
    word.ptr  # given away: launches that are not followed
    word.read(side, reset=True)
    word.read(other)
    word.copies.clear()
    assert word.pending(side) == 0 and word.copies == [2]


def test_status_word_a_graph_was_given_is_read_at_every_checkpoint(word):
    side, capturing = FakeStream(2), FakeStream(CAPTURING)
    assert word.pending(capturing) == 0 and word.copies == [CAPTURING]  # where a real one refuses
    word.launch(capturing, "nothing", lambda address, stream: 0)
    assert word.read(capturing) == 0 and word.read(side) == 0
    word.word.fill_(8)  # a replay reports
    assert word.pending(side, reset=True) == 8
    word.copies.clear()
    assert word.pending(side) == 0 and word.copies == [2]


def test_every_operator_is_compliant_and_refuses_a_second_derivative():
    for name in ("project", "project_vjp", "project_out", "compose_pose", "compose_pose_vjp"):
        assert torch.Tag.pt2_compliant_tag in getattr(torch.ops.dpt, name).default.tags
    grid, geometry, _ = cone_scene(views=2)
    value = _projection_ops.configuration(grid, geometry, 4, "float32")
    field = torch.empty(grid.shape, device="meta", requires_grad=True)
    poses = torch.empty((2, 12), dtype=torch.float64, device="meta")
    cotangent = torch.empty(geometry.shape, device="meta", requires_grad=True)
    gradient, _ = torch.ops.dpt.project_vjp(field, poses, cotangent, value, True, False)
    with pytest.raises(RuntimeError, match="no autograd formula"):
        gradient.sum().backward()


def test_a_tangent_updated_in_place_before_the_backward_is_accepted():
    anchor = torch.tensor(RigidTransform().packed(), dtype=torch.float64)
    tangent = torch.full((6,), 0.1, dtype=torch.float64, requires_grad=True)
    poses = _projection_ops.compose_fixed_anchor(anchor, tangent)
    saved = poses.grad_fn.saved_tensors[1]
    with torch.no_grad():
        tangent.add_(1.0)
    assert poses.grad_fn.saved_tensors[1].tolist() == saved.tolist() == [0.1] * 6


@pytest.mark.parametrize("free,allocations", [(1000, 0), (10000, 1)])
def test_moments_that_do_not_fit_are_refused_once(monkeypatch, free, allocations):
    """Strict FP64 moments of 800 bytes: beside 1000 free bytes none is tried, and one allocation
    that fails all the same is not repeated at every step."""
    workspace = ProjectionWorkspace.__new__(ProjectionWorkspace)
    workspace.spec = ProjectionSpec(4, precision="float64", sampling_precision="float64")
    workspace.device, workspace._moments, workspace._moments_refused = torch.device("cuda:0"), None, False
    monkeypatch.setattr(ProjectionWorkspace, "_moment_bytes", lambda self: 800)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device: (free, 1 << 40))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda device: 0)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda device: 0)
    tried = []

    def empty(*args, **kwargs):
        tried.append(args)
        raise torch.OutOfMemoryError

    monkeypatch.setattr(torch, "empty", empty)
    assert [workspace._allocate_moments() for _ in range(3)] == [False] * 3
    assert len(tried) == allocations


def test_the_operators_can_be_reloaded():
    """As operators defined with custom_op can (in a process of its own: it replaces them)."""
    code = """
import importlib, torch
from dpt_b200.torch import _projection_ops as ops
for _ in range(2):
    importlib.reload(ops)
from scenes import cone_scene
grid, geometry, _ = cone_scene(views=2)
field = torch.empty(grid.shape, device="meta", requires_grad=True)
poses = torch.empty((2, 12), dtype=torch.float64, device="meta")
image = ops.project(field, poses, ops.configuration(grid, geometry, 4, "float32"), True, False)
image.sum().backward()
assert image.shape == geometry.shape and field.grad.shape == field.shape
"""
    root = Path(__file__).resolve().parents[1]
    environment = {**os.environ, "PYTHONPATH": os.pathsep.join((str(root), str(root / "tests")))}
    result = subprocess.run([sys.executable, "-c", code], env=environment, capture_output=True, text=True)
    assert result.returncode == 0, result.stderr
