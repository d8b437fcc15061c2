"""The preconditioned direction entry by entry against fp64, where rows and columns of the gradient differ by many decades
or are zero, and the inverse roots with them."""

import pytest
import torch

import optimizers_b200 as ob
from test_gpu_newton_range import _full

pytestmark = pytest.mark.gpu


def _gradient(shape, kind, gen):
    g = torch.randn(shape, device="cuda", generator=gen)
    rows, cols = shape
    if kind == "dead":
        g[-4:] = 0.0
        g[:, -4:] = 0.0
    elif kind != "plain":
        size = float(kind.split("_")[1])
        g[5] *= size
        g[:, 7] *= size
    return g


@pytest.mark.parametrize("exponent", [0.25, 0.5, 1.0])
@pytest.mark.parametrize("kind", ["plain", "dead", "scaled_1e-6", "scaled_1e-8", "scaled_1e-10"])
@pytest.mark.parametrize("scale", [1.0, 1e-4])
def test_direction_of_a_block_with_rows_and_columns_of_any_size(exponent, kind, scale):
    gen = torch.Generator(device="cuda").manual_seed(11)
    shape = (96, 120)
    p = torch.nn.Parameter(torch.zeros(shape, device="cuda"))
    config = ob.RootInvShampooPreconditionerConfig(inverse_exponent_override={2: exponent})
    opt = ob.DistributedShampoo(
        [p], lr=1.0, betas=(0.0, 1.0), epsilon=1e-12, max_preconditioner_dim=128, precondition_frequency=6, start_preconditioning_step=6,
        preconditioner_config=config, grafting_config=None,
    )
    for _ in range(7):
        p.grad = _gradient(shape, kind, gen) * scale
        before = p.detach().double()
        opt.step()
    state = next(v for k, v in opt.state[p].items() if str(k).startswith("block_"))["shampoo"]
    L, R = (_full(x) for x in state.inv_factor_matrices)
    F = p.grad.double()
    want, got = -(L @ F @ R), p.detach().double() - before
    # Two products with operands of 22 bits, summed 16 terms at a time; the update is added to the weight in fp32.  Entries of
    # the gradient or of the first product below 2^-28 of their row's bound are held to 2^-50 of it.
    terms = L.abs() @ F.abs() @ R.abs()
    steps = 2 * (3 * 2.0**-22 + 3 * (120 / 16 + 1) * 2.0**-24)
    bound = R.abs() @ F.abs().amax(0)
    floor = 4 * 2.0**-50 * (torch.outer(L.abs() @ F.abs().amax(1), R.abs().sum(1)) + torch.outer(L.abs().sum(1), bound))
    limit = 2 * steps * terms + 2 * floor + 2.0**-23 * (before.abs() + want.abs())
    error = (got - want).abs()
    assert bool((error <= limit).all()), (error / limit).max()
    if kind in ("plain", "dead", "scaled_1e-6", "scaled_1e-8"):
        # the floor does not show: rows and columns of these sizes are within the range of the pairs
        assert bool((error <= 4 * steps * terms + 2.0**-23 * (before.abs() + want.abs())).all()), (error / terms.clamp_min(1e-300)).max()


@pytest.mark.parametrize("kind", ["plain", "dead", "scaled_1e-6", "scaled_1e-8"])
def test_second_moments_in_the_eigenbasis_of_a_block_with_rows_and_columns_of_any_size(kind):
    """SOAP with eigenbases that are permutations: the projected gradient is the gradient itself, in another order, and each
    of its entries keeps its precision."""
    gen = torch.Generator(device="cuda").manual_seed(12)
    shape = (96, 120)
    p = torch.nn.Parameter(torch.zeros(shape, device="cuda"))
    opt = ob.DistributedShampoo(
        [p], lr=1.0, betas=(0.0, 1.0), epsilon=1e-15, max_preconditioner_dim=128, precondition_frequency=1000, start_preconditioning_step=1000,
        preconditioner_config=ob.EigenvalueCorrectedShampooPreconditionerConfig(), grafting_config=None,
    )
    orders = [torch.randperm(n, device="cuda", generator=gen) for n in shape]
    p.grad = _gradient(shape, "plain", gen)
    opt.step()
    state = opt.state_dict()
    block = next(v for k, v in state["state"][next(iter(state["state"]))].items() if str(k).startswith("block_"))["shampoo"]
    block["corrected_eigenvalues"].zero_()
    for basis, order in zip(block["factor_matrices_eigenvectors"].values(), orders, strict=True):
        basis.copy_(torch.eye(basis.shape[0], device="cuda")[:, order])
    opt.load_state_dict(state)
    for value in opt.state[p].values():
        if isinstance(value, torch.Tensor) and value.dtype == torch.int64:
            value.fill_(1001)
    p.grad = _gradient(shape, kind, gen)
    before = p.detach().double()
    opt.step()
    g = p.grad.double()
    got = p.detach().double() - before
    moments = next(v for k, v in opt.state[p].items() if str(k).startswith("block_"))["shampoo"].corrected_eigenvalues.double()
    # 2^-20: the rounding of two products with one term each and of the square; 2^-50: half a step of lo at the bound of the
    # gradient's row, then of the first product's (a column of the gradient)
    floor = 4 * 2.0**-50 * torch.maximum(g.abs().amax(1, keepdim=True), g.abs().amax(0, keepdim=True))
    want, slack = g[orders[0]][:, orders[1]], floor[orders[0]][:, orders[1]]
    assert bool(((moments.sqrt() - want.abs()).abs() <= 2.0**-20 * want.abs() + slack).all()), ((moments.sqrt() - want.abs()).abs() / want.abs()).max()
    direction = -torch.where(g == 0, 0.0, g / (g.abs() + 1e-15))
    limit = 2.0**-18 + torch.where(g == 0, 0.0, 2 * floor / g.abs().clamp_min(1e-30))
    assert bool(((got - direction).abs() <= limit).all()), (got - direction).abs().max()
