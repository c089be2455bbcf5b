"""State kept between calls on the GPU: poses used from several streams, status words read across
streams and graph replays, and pose moments beside a caller's own memory."""

from __future__ import annotations

import pytest
import torch

from dpt_b200.contracts import NumericalError, TrialDomainError
from dpt_b200.objectives import ObjectiveSpec, evaluate_objective, prepare_objective
from dpt_b200.torch import Projector, _projection_ops
from dpt_b200.torch.operators import objective
from dpt_b200.transmission import TransmissionSpec, prepare_transmission, transmission_vjp, transmit
from scenes import cone_scene

pytestmark = pytest.mark.gpu
DEVICE = "cuda:0"


def busy(stream: torch.cuda.Stream) -> None:
    """Queue some tens of milliseconds of products on a stream."""
    with torch.cuda.stream(stream):
        a = torch.ones((4096, 4096), device=DEVICE)
        for _ in range(20):
            a = a @ a * 1e-4


def test_one_projector_on_two_streams_without_a_pose():
    grid, geometry, values = cone_scene(views=3)
    field = torch.tensor(values, dtype=torch.float32, device=DEVICE)
    expected = Projector(grid=grid, geometry=geometry, samples_per_ray=64)(field)
    shared = Projector(grid=grid, geometry=geometry, samples_per_ray=64)
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    busy(first)
    with torch.cuda.stream(first):
        poses = shared._packed_poses(field, None, None)  # made behind the queued work
    with torch.cuda.stream(second):
        torch.testing.assert_close(shared(field), expected, rtol=0, atol=0)
    with torch.cuda.stream(first):
        torch.testing.assert_close(shared(field), expected, rtol=0, atol=0)
    assert shared._packed_poses(field, None, None) is poses


def test_projector_first_called_in_inference_mode_trains():
    grid, geometry, values = cone_scene(views=3)
    field = torch.tensor(values, dtype=torch.float32, device=DEVICE)
    projector = Projector(grid=grid, geometry=geometry, samples_per_ray=64)
    with torch.inference_mode():
        expected = projector(field)
    volume = field.clone().requires_grad_()
    image = projector(volume)
    image.sum().backward()
    torch.testing.assert_close(image.detach(), expected.clone(), rtol=0, atol=0)
    assert float(volume.grad.abs().sum()) > 0


def test_an_error_on_an_owned_side_stream_reaches_its_checkpoint_once():
    side = torch.cuda.Stream()
    ws = prepare_transmission(TransmissionSpec(beam="scalar"), device=DEVICE, max_pixels=300, stream=side)
    depth, seed = torch.zeros(300, device=DEVICE), torch.full((300,), 1e38, device=DEVICE)
    out, gradient = torch.empty_like(depth), torch.empty_like(depth)
    torch.cuda.synchronize()
    busy(side)
    # -n0 exp(-L) seed is beyond FP32; the current stream is another one and idle
    transmission_vjp(depth, 1e5, cotangent_counts=seed, out_grad_L=gradient, workspace=ws, validate=False)
    with pytest.raises(NumericalError):
        ws.check_status()
    transmit(depth, 1e5, out_T=out, workspace=ws, validate=False)
    with pytest.raises(NumericalError):
        ws.settle()
    ws.settle()
    ws.check_status()
    torch.testing.assert_close(out, torch.ones_like(out), rtol=0, atol=0)


def test_an_error_of_a_replayed_graph_reaches_the_next_operator():
    ws = prepare_objective(ObjectiveSpec(kind="poisson", domain="counts"), device=DEVICE, max_pixels=300)
    observation = torch.full((300,), 5.0, device=DEVICE)
    prediction = torch.full((300,), 4.0, device=DEVICE)
    loss = torch.empty(1, dtype=torch.float64, device=DEVICE)

    def checked():
        mu = torch.full((300,), 4.0, device=DEVICE, requires_grad=True)
        return mu, objective(mu, observation, workspace=ws)

    evaluate_objective(prediction, observation, out_loss=loss, workspace=ws, validate=False)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        evaluate_objective(prediction, observation, out_loss=loss, workspace=ws, validate=False)
    graph.replay()
    mu, value = checked()
    prediction.fill_(-1.0)
    graph.replay()
    with pytest.raises(TrialDomainError):  # a zero cotangent launches nothing of its own
        (0.0 * value).backward()
    with pytest.raises(TrialDomainError):
        checked()
    ws.clear_status()
    mu, value = checked()
    value.backward()
    assert float(mu.grad.abs().sum()) > 0
    del graph


def test_a_pose_updated_in_place_before_the_backward_keeps_its_gradient():
    grid, geometry, values = cone_scene(views=3)
    field = torch.tensor(values, dtype=torch.float32, device=DEVICE)
    projector = Projector(grid=grid, geometry=geometry, samples_per_ray=64)
    poses = [torch.full((3, 6), 0.01, dtype=torch.float64, device=DEVICE, requires_grad=True) for _ in range(2)]
    images = [projector(field, pose) for pose in poses]
    with torch.no_grad():
        poses[1].add_(0.5)
    for image in images:
        image.sum().backward()
    torch.testing.assert_close(poses[1].grad, poses[0].grad, rtol=1e-12, atol=0)


def test_strict_fp64_step_without_room_for_its_moments(monkeypatch):
    """Beside little free memory the step samples twice: no kept moments, the same image and pose
    gradient, and a volume gradient to FP32 summation order."""
    grid, geometry, values = cone_scene(views=3)
    results, held = [], []
    for free in (None, 1 << 10):
        _projection_ops.clear_cache()
        if free is not None:
            monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device: (free, 1 << 40))
            monkeypatch.setattr(torch.cuda, "memory_reserved", lambda device: 0)
            monkeypatch.setattr(torch.cuda, "memory_allocated", lambda device: 0)
        field = torch.tensor(values, dtype=torch.float32, device=DEVICE, requires_grad=True)
        pose = torch.full((3, 6), 0.01, dtype=torch.float64, device=DEVICE, requires_grad=True)
        image = Projector(grid=grid, geometry=geometry, samples_per_ray=64, precision="fp64")(field, pose)
        image.sum().backward()
        results.append((image.detach(), pose.grad, field.grad))
        held.append([ws._moments is not None for ws in _projection_ops._CACHE.values()])
    assert held == [[True], [False]]
    torch.testing.assert_close(results[1][0], results[0][0], rtol=0, atol=0)
    torch.testing.assert_close(results[1][1], results[0][1], rtol=1e-9, atol=1e-12)
    assert float((results[1][2] - results[0][2]).norm()) <= 2e-6 * float(results[0][2].norm())
    _projection_ops.clear_cache()
