"""The coupled Newton refresh on factors whose diagonal spans many decades, row by row against fp64.

A dim that has never received a gradient has a zero row in its factor, so its eigenvalue is the ridge alone and its root is
``epsilon^(-1/p)``, many decades from the others'; the iteration starts from it at ``epsilon / |A|``."""

import pytest
import torch

import optimizers_b200 as ob

pytestmark = pytest.mark.gpu


def _full(packed):
    if packed.dim() == 2:
        return packed.double()
    d = int((2 * packed.numel()) ** 0.5)
    m = torch.zeros(d, d, device=packed.device, dtype=torch.float64)
    rows, cols = torch.triu_indices(d, d, device=packed.device)
    m[rows, cols] = packed.double()
    return m + m.triu(1).T


@pytest.mark.parametrize("epsilon", [1e-12, 1e-7])
@pytest.mark.parametrize("scale", [0.0, 1e-4])
def test_roots_of_dims_with_little_or_no_gradient(epsilon, scale):
    gen = torch.Generator(device="cuda").manual_seed(2)
    shape = (160, 192)
    p = torch.nn.Parameter(torch.zeros(shape, device="cuda"))
    opt = ob.DistributedShampoo(
        [p], lr=1.0, betas=(0.0, 1.0), epsilon=epsilon, max_preconditioner_dim=256, precondition_frequency=4, start_preconditioning_step=4,
        preconditioner_config=ob.RootInvShampooPreconditionerConfig(amortized_computation_config=ob.CoupledNewtonConfig()), grafting_config=None,
    )
    for _ in range(4):
        g = torch.randn(shape, device="cuda", generator=gen)
        for dim in range(2):
            g.narrow(dim, shape[dim] - 4, 4).mul_(scale)
        p.grad = g
        opt.step()
    state = next(v for k, v in opt.state[p].items() if str(k).startswith("block_"))["shampoo"]
    for factor, root in zip(state.factor_matrices, state.inv_factor_matrices, strict=True):
        A, got = _full(factor), _full(root)
        lam, Q = torch.linalg.eigh(A + epsilon * torch.eye(A.shape[0], device="cuda", dtype=torch.float64))
        want = (Q * lam.clamp_min(epsilon).pow(-0.25)) @ Q.T
        # In up to 60 iterations of p + 1 products each (p = 4), with a relative error of 5e-7 at these sizes: every row to its own size
        error = (got - want).norm(dim=1) / want.norm(dim=1)
        assert float(error.max()) < 60 * 5 * 5e-7, error.topk(5)
