"""Householder panels and Jacobi leaves at the sizes where their layouts change, against fp64."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ext():
    from optimizers_b200.ops import build

    return build.load()


def _pad4(n):
    return (n + 3) // 4 * 4


# Panels of up to 512, 1024 and 2048 rows live in registers (1, 2, 4 rows per thread), longer ones in shared memory; the
# lengths shrink by 16 from panel to panel, the last panel may be narrower than 16 columns.
@pytest.mark.parametrize("n,k", [(1, 1), (15, 15), (17, 17), (512, 33), (513, 20), (1024, 18), (1030, 40), (2048, 17), (2049, 35)])
def test_householder_panels_at_the_edges_of_their_layouts(ext, n, k):
    gen = torch.Generator(device="cuda").manual_seed(n)
    Y = torch.randn(n, k, device="cuda", generator=gen, dtype=torch.float64)
    Y[:, k // 2] *= 1e-3
    if k > 3:
        Y[:, 3] = 0.0  # a column that needs no reflector
    ct = torch.zeros(k, _pad4(n), device="cuda")[:, :n].copy_(Y.T)
    zt, hi, lo = (torch.full((n, _pad4(n)), float("nan"), device="cuda")[:, :n] for _ in range(3))
    ext.householder_qr([(ct, n, k, zt, hi, lo)])
    Q = zt.double().T
    eye = torch.eye(n, device="cuda", dtype=torch.float64)
    # k reflectors of n terms: rounding of about sqrt(n) 2^-24 each, summed like a random walk
    bound = 4 * (n * k) ** 0.5 * 2.0**-24 + 2.0**-21
    assert float((Q.T @ Q - eye).abs().max()) < bound
    R = torch.triu(ct.double().T[:k])
    assert float((Q[:, :k] @ R - Y.float().double()).norm() / Y.norm()) < bound


# Blocks of four columns, an even number of them: the sizes around their edges, and repeated or zero eigenvalues.
@pytest.mark.parametrize("n", [3, 4, 5, 8, 9, 12, 31, 33, 97, 124, 125, 127])
@pytest.mark.parametrize("kind", ["full", "identity", "low_rank", "graded"])
def test_jacobi_blocks_at_their_edges(ext, n, kind):
    gen = torch.Generator(device="cuda").manual_seed(n)
    B = torch.randn(n, 2 * n, device="cuda", generator=gen, dtype=torch.float64)
    A = {
        "full": B @ B.T / n,
        "identity": 3.0 * torch.eye(n, device="cuda", dtype=torch.float64),
        "low_rank": B[:, :2] @ B[:, :2].T + 1e-6 * torch.eye(n, device="cuda", dtype=torch.float64),
        "graded": B @ B.T / n * torch.logspace(0, -3, n, device="cuda", dtype=torch.float64).outer(torch.logspace(0, -3, n, device="cuda", dtype=torch.float64)),
    }[kind].float()
    lams, qs, sweeps = ext.jacobi_eigh([A], 24, 2e-6)
    assert int(sweeps[0]) <= 24
    want = torch.linalg.eigvalsh(A.double())
    scale = float(want.abs().max())
    # a column takes part in n rotations a sweep, in about 15 sweeps, and c^2 + s^2 is off by up to 2^-24 each time
    bound = (15 * n + 16) * 2.0**-24
    assert float((lams[0].double() - want).abs().max()) < bound * scale
    Q = qs[0].double()
    assert float((Q.T @ Q - torch.eye(n, device="cuda", dtype=torch.float64)).abs().max()) < 5e-6
    assert float(((Q * lams[0].double()) @ Q.T - A.double()).abs().max()) < bound * scale
