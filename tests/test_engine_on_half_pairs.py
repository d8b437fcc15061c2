"""The native engine on the CPU stand-in with its products on half pairs (tests/test_engine_host_logic.py runs the same
configurations on tf32 pairs; its multi-process tests run on half pairs too).  The stand-in holds fp32 values in the pairs'
layout and checks, for every product, the bounds of the rows that their scales follow."""

import pytest
import torch

import optimizers_b200 as ob
import test_engine_host_logic as host


@pytest.fixture
def cpu_engine(monkeypatch):
    return host.install_cpu_engine(monkeypatch.setattr)


def _on_pairs(opt):
    return [rec["native_engine"]._half for rec in opt._per_group_state_lists]


@pytest.mark.parametrize("name", list(host._configs()))
def test_engine_matches_the_torch_step(cpu_engine, name):
    host.test_engine_on_the_stand_in_matches_the_torch_step(cpu_engine, name)


def test_which_groups_run_on_half_pairs(cpu_engine):
    assert all(_on_pairs(host._train("native", steps=4, **host._configs()["kl_root_inverse"])[1]))
    for name in ("single_pass_gemm_mode", "rows_only"):
        assert not any(_on_pairs(host._train("native", steps=4, **host._configs()[name])[1]))


def test_engine_with_a_gradient_that_goes_missing(cpu_engine):
    host.test_engine_with_a_gradient_that_goes_missing(cpu_engine)


def test_engine_resumes_from_a_checkpoint(cpu_engine):
    host.test_engine_resumes_from_a_checkpoint(cpu_engine)


@pytest.mark.parametrize("soap", [False, True])
def test_order_3_blocks_match_the_torch_step(cpu_engine, soap):
    """First two dims in multiples of 32, as half pairs need; the re-viewed unfoldings share bounds among rows."""
    results = []
    for backend in ("torch", "native"):
        torch.manual_seed(3)
        p = torch.nn.Parameter(torch.randn(64, 32, 9) * 0.1)
        config = ob.EigenvalueCorrectedShampooPreconditionerConfig() if soap else ob.RootInvShampooPreconditionerConfig()
        opt = ob.DistributedShampoo(
            [p], lr=1e-2, betas=(0.9, 0.999), epsilon=1e-4, max_preconditioner_dim=64, precondition_frequency=40 if soap else 3,
            start_preconditioning_step=40 if soap else 3, preconditioner_config=config, grafting_config=ob.AdamPreconditionerConfig(),
            native_runtime_config=ob.NativeRuntimeConfig(backend=backend),
        )
        g = torch.Generator().manual_seed(5)
        sizes = torch.logspace(0, -1.5, 64).view(64, 1, 1) * torch.logspace(0, -1, 9)
        for _ in range(43 if soap else 8):
            p.grad = torch.randn(p.shape, generator=g) * sizes
            opt.step()
        if backend == "native":
            assert _on_pairs(opt) == [True]
        results.append(p.detach().clone())
    assert torch.allclose(*results, rtol=1e-4, atol=2e-4 if soap else 2e-6), (results[0] - results[1]).abs().max()


@pytest.mark.parametrize("kind", ["root_inverse", "eigendecomposed", "eigenvalue_corrected"])
def test_a_refresh_that_raises_leaves_the_mirrors_as_they_were(cpu_engine, monkeypatch, kind):
    """A refresh may stop after it has written fp32 matrices into the operands' memory; the caller catches the error and
    goes on with the preconditioner of the state."""
    import optimizers_b200.native_engine as engine_module

    config = {
        "root_inverse": ob.RootInvShampooPreconditionerConfig, "eigendecomposed": ob.EigendecomposedShampooPreconditionerConfig,
        "eigenvalue_corrected": ob.EigenvalueCorrectedShampooPreconditionerConfig,
    }[kind]()
    original = engine_module.NativeGroupEngine._refresh
    finals = []
    for scribble in (False, True):
        calls = []

        def refresh(self, blocks):
            calls.append(None)
            if len(calls) != 2:
                return original(self, blocks)
            if scribble:
                for b in blocks:
                    for mirror in b.inv_hi:
                        mirror.fill_(7.0)
            raise ValueError("refresh stopped half way")

        monkeypatch.setattr(engine_module.NativeGroupEngine, "_refresh", refresh)
        torch.manual_seed(0)
        p = torch.nn.Parameter(torch.randn(24, 40) * 0.1)
        opt = ob.DistributedShampoo(
            [p], lr=1e-2, betas=(0.9, 0.999), epsilon=1e-4, max_preconditioner_dim=64, precondition_frequency=4, start_preconditioning_step=4,
            preconditioner_config=config, native_runtime_config=ob.NativeRuntimeConfig(backend="native"),
        )
        g = torch.Generator().manual_seed(1)
        raised = 0
        for _ in range(11):
            p.grad = torch.randn(p.shape, generator=g)
            try:
                opt.step()
            except ValueError:
                raised += 1
        assert raised == 1 and len(calls) == 2 and _on_pairs(opt) == [True]
        finals.append(p.detach().clone())
    assert torch.equal(*finals)
