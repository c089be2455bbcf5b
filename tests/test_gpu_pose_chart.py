"""The tangent gradient of a Projector's pose chart (one kernel) against Torch's own reverse pass
of ``compose_pose``.

Both differ from the exact derivative by rounding of a few hundred FP64 operations on values of
the gradient's size, amplified at most by the cancellation of the closed-form coefficients just
above theta = 2 (a factor below 20): 1e-12 of the gradient's norm covers it."""

from __future__ import annotations

import pytest
import torch

from dpt_b200.torch import _projection_ops, compose_pose

pytestmark = pytest.mark.gpu

IDENTITY = [1.0, 0, 0, 0, 1.0, 0, 0, 0, 1.0, 0, 0, 0]


@pytest.mark.parametrize("angle", [0.0, 1e-9, 1e-3, 0.3, 1.9999, 2.0001, 3.1])
@pytest.mark.parametrize("anchors,tangents", [((12,), (6,)), ((12,), (5, 6)), ((300, 12), (300, 6)), ((1, 12), (1, 6))])
def test_tangent_gradient_equals_the_reverse_pass_of_the_chart(anchors, tangents, angle):
    g = torch.Generator(device="cuda").manual_seed(7)
    eye = torch.tensor(IDENTITY, dtype=torch.float64, device="cuda")

    def normal(shape):
        return torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)

    anchor = compose_pose(eye.expand(anchors), normal((*anchors[:-1], 6))).contiguous()
    axis = normal((*tangents[:-1], 3))
    tangent = torch.cat((10.0 * normal((*tangents[:-1], 3)), angle * axis / axis.norm(dim=-1, keepdim=True)), -1)
    expected_in, actual_in = (tangent.clone().requires_grad_() for _ in range(2))
    expected = compose_pose(anchor, expected_in)
    actual = _projection_ops.compose_fixed_anchor(anchor, actual_in)
    torch.testing.assert_close(actual, expected, rtol=0, atol=0)
    cotangent = normal(tuple(expected.shape))
    want, = torch.autograd.grad(expected, expected_in, cotangent)
    got, = torch.autograd.grad(actual, actual_in, cotangent)
    assert got.shape == want.shape
    assert float((got - want).norm()) <= 1e-12 * float(want.norm())


@pytest.mark.parametrize("angle", [3.2, 6.283184307, 6.283185307179586, 7.0, 20.0])
def test_tangent_gradient_beyond_a_half_turn(angle):
    """The closed form up to three turns, at the same bar: its cancellation only shrinks with theta."""
    test_tangent_gradient_equals_the_reverse_pass_of_the_chart((300, 12), (300, 6), angle)
