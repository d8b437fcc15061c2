"""Grouped products on scaled fp16 pairs (the operand format of the step) against fp64."""

import pytest
import torch

pytestmark = pytest.mark.gpu

_CHUNK = 32


@pytest.fixture(scope="module")
def ext():
    from optimizers_b200.ops import build

    return build.load()


def _pad(n):
    return (n + _CHUNK - 1) // _CHUNK * _CHUNK


def _scale(meta):
    return 2.0 ** (15.0 - torch.frexp(meta[0])[1].double()).clamp(max=110)


def _pairs(x):
    """(array of pairs, meta data) of a matrix, with the format restated in fp64."""
    rows, cols = x.shape
    meta = torch.stack([x.abs().max(), (x.double() ** 2).sum(1).max().float()])
    v = torch.zeros(rows, _pad(cols), device=x.device, dtype=torch.float64)
    v[:, :cols] = x.double() * _scale(meta)
    hi = v.half()
    lo = (v - hi.double()).half()
    return torch.stack([hi.view(rows, -1, _CHUNK), lo.view(rows, -1, _CHUNK)], 2).reshape(rows, -1).view(torch.float32), meta


def _value(pairs, meta, cols):
    h = pairs.contiguous().view(torch.float16).view(pairs.shape[0], -1, 2, _CHUNK).double()
    assert not (h.sum(2).reshape(pairs.shape[0], -1)[:, cols:]).any()  # padding
    return (h.sum(2).reshape(pairs.shape[0], -1) / _scale(meta))[:, :cols]


def _matrix(rows, cols, gen, decades):
    x = torch.randn(rows, cols, device="cuda", generator=gen)
    scales = [torch.pow(10.0, decades * torch.randn(n, device="cuda", generator=gen)) for n in (rows, cols)]
    return x * scales[0].unsqueeze(1) * scales[1] * 1e-4


def _bound(K):
    """Relative 2-norm error of a product with K terms: three dropped or rounded parts of 2^-22 each, and fp32
    accumulation truncated once per 16 terms and product, a drift of at most 2^-24 per step."""
    return 3 * 2.0**-22 + 3 * (K / 16 + 1) * 2.0**-24


# One tile and less; ragged tiles; a K loop long enough to be cut among CTAs (with few rows, with several tiles,
# with a length the parts do not divide); tiles of 256 columns.
@pytest.mark.parametrize(
    "M,N,K", [(1, 1, 1), (128, 128, 32), (10, 77, 33), (129, 257, 100), (3, 3, 98304), (130, 40, 5000), (64, 576, 1601), (1000, 4200, 65), (2100, 2100, 40)]
)
@pytest.mark.parametrize("decades", [0.0, 0.25])
def test_products_on_pairs_match_fp64(ext, M, N, K, decades):
    gen = torch.Generator(device="cuda").manual_seed(M + N + K)
    A, B = _matrix(M, K, gen, decades), _matrix(N, K, gen, decades)
    (a, a_meta), (b, b_meta) = _pairs(A), _pairs(B)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    old = torch.randn(M, N, device="cuda", generator=gen) * 1e-8
    c = old.clone()
    d, d_meta = torch.full((M, _pad(N)), float("nan"), device="cuda"), torch.zeros(2, device="cuda")
    norm = torch.zeros(1, device="cuda")
    plain = ext.build_gemm_plan([(a, None, b, None, c, None, None, norm, N, 0, ext.FLAG_SUMSQ, False, None, None, (a_meta, b_meta, None))])
    split = ext.build_gemm_plan([(
        a, None, b, None, None, d, None, None, 0, _pad(N), ext.FLAG_NO_C | ext.FLAG_SPLIT_OUT, False, None, None, (a_meta, b_meta, d_meta)
    )])
    ref = A.double() @ B.double().T
    first = None
    for _ in range(2):  # the counters of split tiles are ready for the next run
        c.copy_(old)
        norm.zero_()
        ext.run_gemm_plan(*plain, 0.5, 0.9, ext.HALF_PAIR, status)
        ext.run_gemm_plan(*split, 1.0, 0.0, ext.HALF_PAIR, status)
        want = 0.5 * ref + 0.9 * old.double()
        first = c.clone() if first is None else first
        assert torch.equal(c, first)
        assert float((c.double() - want).norm() / want.norm()) < _bound(K)
        assert abs(float(norm) / float((want**2).sum()) - 1) < 2 * _bound(K) + 1e-5  # 2-norm squared, summed in fp32
        assert float(d_meta[0]) >= float(ref.abs().max())
        assert float((_value(d, d_meta, N) - ref).norm() / ref.norm()) < _bound(K) + 2.0**-22
    assert int(status) == 0


@pytest.mark.parametrize("d,K", [(5, 1), (128, 700), (300, 96), (777, 2000), (2048, 64)])
def test_gram_of_pairs_in_the_packed_triangle(ext, d, K):
    gen = torch.Generator(device="cuda").manual_seed(d)
    X = _matrix(d, K, gen, 0.25)
    x, meta = _pairs(X)
    rows, cols = torch.triu_indices(d, d, device="cuda")
    state = torch.rand(d * (d + 1) // 2, device="cuda", generator=gen) * 1e-8
    want = 0.1 * (X.double() @ X.double().T)[rows, cols] + 0.9 * state.double()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    plan = ext.build_gemm_plan([(x, None, x, None, state, None, None, None, d, 0, ext.FLAG_PACKED_C, True, None, None, (meta, meta, None))])
    ext.run_gemm_plan(*plan, 0.1, 0.9, ext.HALF_PAIR, status)
    assert float((state.double() - want).norm() / want.norm()) < _bound(K)
    assert int(status) == 0


@pytest.mark.parametrize("d", [1, 31, 32, 33, 200])
@pytest.mark.parametrize("scale", [1e-30, 1.0, 1e37])
def test_mirrors_are_converted_in_place(ext, d, scale):
    gen = torch.Generator(device="cuda").manual_seed(d)
    X = torch.randn(d, d, device="cuda", generator=gen) * scale
    buf = torch.full((d, _pad(d)), float("nan"), device="cuda")
    buf[:, :d] = X
    t, meta = torch.full((d, _pad(d)), float("nan"), device="cuda"), torch.zeros(2, device="cuda")
    ext.pair_mirrors(*ext.build_pair_table([(buf[:, :d], buf, t, meta)]))
    assert float(meta[0]) == float(X.abs().max())
    for got, want in ((buf, X), (t, X.T)):  # 22 bits, or 2^-25 steps of the scaled value
        assert bool(((_value(got, meta, d) - want.double()).abs() <= 2.0**-22 * want.abs() + 2.0**-25 / _scale(meta)).all())


# The epilogues of the symmetric iterations: one tile, ragged edges, several tiles, wide tiles.
@pytest.mark.parametrize("sizes", [(1,), (33, 128), (200, 300, 31), (1500, 1500)])
def test_symmetric_products_on_pairs(ext, sizes):
    gen = torch.Generator(device="cuda").manual_seed(sum(sizes))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    bound = torch.tensor([8.0, 0.0], device="cuda")
    specs, finals, checks = [], [], []
    stats = torch.zeros(len(sizes), 2, device="cuda")
    for i, n in enumerate(sizes):
        X = torch.randn(n, n, device="cuda", generator=gen)
        X = (X + X.T) / (2.0 * n**0.5)
        x, meta = _pairs(X)
        c = torch.randn(n, n, device="cuda", generator=gen) / n**0.5
        c = (c + c.T) / 2
        d = torch.full((n, _pad(n)), float("nan"), device="cuda")
        pitch = (n + 3) // 4 * 4
        hi, lo = (torch.full((n, pitch), float("nan"), device="cuda") for _ in range(2))
        XX = X.double() @ X.double().T
        checks.append((c, d, hi, lo, 2.0 * XX - 0.5 * c.double() + 0.7 * torch.eye(n, device="cuda"), 0.5 * XX + 0.5 * torch.eye(n, device="cuda"), n))
        sym = ext.FLAG_MIRROR | ext.FLAG_SPLIT_OUT | ext.FLAG_ADD_DIAG
        specs.append((x, None, x, None, c, d, None, None, c.stride(0), d.stride(0), sym | ext.FLAG_FIXED_SCALE, True, None, None, (meta, meta, bound)))
        finals.append((x, None, x, None, None, hi, lo, stats[i], 0, pitch, sym | ext.FLAG_NO_C | ext.FLAG_SUMSQ | ext.FLAG_TRACE, True,
                       None, None, (meta, meta, None)))
    ext.run_gemm_plan(*ext.build_gemm_plan(specs), 2.0, -0.5, ext.HALF_PAIR_SYM, status, 0.7)
    ext.run_gemm_plan(*ext.build_gemm_plan(finals), 0.5, 0.0, ext.HALF_PAIR_SYM, status, 0.5)
    for i, (c, d, hi, lo, want, proj, n) in enumerate(checks):
        tol = _bound(n) + 2.0**-22
        value, split = _value(d, bound, n), hi[:, :n].double() + lo[:, :n].double()
        for got, ref in ((c.double(), want), (value, want), (split, proj)):
            assert float((got - ref).norm() / ref.norm()) < tol
            assert torch.equal(got, got.T)
        assert abs(float(stats[i, 0]) / float((proj**2).sum()) - 1) < 2 * tol + 1e-5
        assert abs(float(stats[i, 1]) - float(torch.trace(proj))) < (tol + 1e-5) * float(proj.norm()) * n**0.5
    assert int(status) == 0


def test_plans_of_one_format_are_not_run_in_another(ext):
    x, meta = _pairs(torch.ones(32, 32, device="cuda"))
    c, status = torch.zeros(32, 32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    spec = (x, None, x, None, c, None, None, None, 32, 0, 0, False)
    pairs = ext.build_gemm_plan([(*spec, None, None, (meta, meta, None))])
    plain = ext.build_gemm_plan([spec])
    with pytest.raises(RuntimeError, match="operand format"):
        ext.run_gemm_plan(*pairs, 1.0, 0.0, True, status)
    with pytest.raises(RuntimeError, match="operand format"):
        ext.run_gemm_plan(*plain, 1.0, 0.0, ext.HALF_PAIR, status)
