"""scale_cast: a bf16 product times a device scalar, in the dtype the gradient is returned in."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1), (3, 5), (7, 64), (1000, 769), (4096, 1024)])  # tails of 1 to 7, one CTA, all CTAs
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_scale_cast_is_exact(shape, dtype):
    from optimizers_b200.ops import build

    x = torch.randn(shape, device="cuda").bfloat16()
    scale = torch.tensor(0.3, device="cuda")
    got = build.load().scale_cast(x, scale, dtype == torch.bfloat16)
    assert got.dtype == dtype and torch.equal(got, (x.float() * scale).to(dtype))


def test_lm_head_loss_backward_can_be_recorded():
    """With create_graph the gradient stays differentiable with respect to the incoming gradient."""
    from optimizers_b200.models.fused_ops import lm_head_cross_entropy

    torch.manual_seed(0)
    x = torch.randn(32, 64, device="cuda").bfloat16().requires_grad_(True)
    w = torch.randn(100, 64, device="cuda").requires_grad_(True)
    t = torch.randint(0, 100, (32,), device="cuda")
    with torch.autocast("cuda", dtype=torch.bfloat16):
        loss = lm_head_cross_entropy(x, w, t)
    seed = torch.ones((), device="cuda", requires_grad=True)
    (dw,) = torch.autograd.grad(loss, (w,), grad_outputs=seed, create_graph=True)
    assert dw.requires_grad


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_lm_head_loss_backward_takes_a_batch_of_incoming_gradients(dtype):
    from optimizers_b200.models.fused_ops import lm_head_cross_entropy

    torch.manual_seed(0)
    x = torch.randn(32, 64, device="cuda").bfloat16().requires_grad_(True)
    w = (0.1 * torch.randn(100, 64, device="cuda")).to(dtype).requires_grad_(True)
    t = torch.randint(0, 100, (32,), device="cuda")
    with torch.autocast("cuda", dtype=torch.bfloat16):
        loss = lm_head_cross_entropy(x, w, t)
    seeds = torch.tensor([1.0, -2.0, 0.5], device="cuda")
    batched = torch.autograd.grad(loss, (x, w), grad_outputs=seeds, is_grads_batched=True, retain_graph=True)
    single = torch.autograd.grad(loss, (x, w))
    for many, one in zip(batched, single, strict=True):
        assert many.dtype == one.dtype and many.shape == (3, *one.shape)
        for seed, got in zip(seeds, many, strict=True):  # one more rounding to bf16
            assert float((got.float() - seed * one.float()).norm() / (seed * one.float()).norm()) < 2.0**-8
