"""Grouped products on fp16 pairs with a scale per row (the operand format of the step) against fp64."""

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


def _scale(bound):
    return 2.0 ** (15.0 - torch.frexp(bound)[1].double()).clamp(max=110)


def _pairs(x, div=1):
    """(array of pairs, bounds of its rows, ``div`` rows to one) of a matrix, with the format restated in fp64."""
    rows, cols = x.shape
    bound = x.abs().amax(1).view(-1, div).amax(1)
    scale = _scale(bound.repeat_interleave(div)).unsqueeze(1)
    v = torch.zeros(rows, _pad(cols), device=x.device, dtype=torch.float64)
    v[:, :cols] = x.double() * scale
    hi = v.half()
    lo = ((v - hi.double()) * 2.0**11).half()
    return torch.stack([hi.view(rows, -1, _CHUNK), lo.view(rows, -1, _CHUNK)], 2).reshape(rows, -1).view(torch.float32), bound


def _value(pairs, bound, cols):
    h = pairs.contiguous().view(torch.float16).view(pairs.shape[0], -1, 2, _CHUNK).double()
    v = (h[:, :, 0] + 2.0**-11 * h[:, :, 1]).reshape(pairs.shape[0], -1)
    assert not v[:, cols:].any()  # padding
    return v[:, :cols] / _scale(bound).expand(pairs.shape[0]).unsqueeze(1)


def _outputs(A, B):
    """What a chained product is given to bound the rows of its result: (left, right, cap, bound)."""
    return (A.abs().sum(1), B.abs().max().view(1), None, torch.full((A.shape[0],), float("nan"), device="cuda"))


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
    (a, a_bound), (b, b_bound) = _pairs(A), _pairs(B)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    old = torch.randn(M, N, device="cuda", generator=gen) * 1e-8
    c = old.clone()
    d, out = torch.full((M, _pad(N)), float("nan"), device="cuda"), _outputs(A, B)
    norm = torch.zeros(1, device="cuda")
    plain = ext.build_gemm_plan([(a, None, b, None, c, None, None, norm, N, 0, ext.FLAG_SUMSQ, False, None, None, (a_bound, 1, b_bound, 1, None))])
    split = ext.build_gemm_plan([(
        a, None, b, None, None, d, None, None, 0, _pad(N), ext.FLAG_NO_C | ext.FLAG_SPLIT_OUT, False, None, None, (a_bound, 1, b_bound, 1, out)
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
        assert bool((out[3] * (1 + 1e-5) >= ref.abs().amax(1)).all())
        assert float((_value(d, out[3], N) - ref).norm() / ref.norm()) < _bound(K) + 2.0**-22
    assert int(status) == 0


@pytest.mark.parametrize("d,K", [(5, 1), (128, 700), (300, 96), (777, 2000), (2048, 64)])
def test_gram_of_pairs_in_the_packed_triangle(ext, d, K):
    gen = torch.Generator(device="cuda").manual_seed(d)
    X = _matrix(d, K, gen, 0.25)
    x, bound = _pairs(X)
    rows, cols = torch.triu_indices(d, d, device="cuda")
    state = torch.rand(d * (d + 1) // 2, device="cuda", generator=gen) * 1e-8
    want = 0.1 * (X.double() @ X.double().T)[rows, cols] + 0.9 * state.double()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    plan = ext.build_gemm_plan([(x, None, x, None, state, None, None, None, d, 0, ext.FLAG_PACKED_C, True, None, None, (bound, 1, bound, 1, None))])
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
    X[d // 2] *= 1e-7  # rows and columns keep scales of their own
    X[:, d // 3] = 0.0
    buf[:, :d] = X
    t = torch.full((d, _pad(d)), float("nan"), device="cuda")
    of_rows, of_cols = ((torch.full((d,), float("nan"), device="cuda"), torch.full((d,), float("nan"), device="cuda"), torch.zeros(1, device="cuda")) for _ in range(2))
    ext.pair_mirrors(*ext.build_pair_table([(buf[:, :d], buf, of_rows, t, of_cols)]))
    for got, (bound, l1, top), want in ((buf, of_rows, X), (t, of_cols, X.T)):
        assert torch.equal(bound, want.abs().amax(1))
        assert torch.allclose(l1, want.abs().sum(1), rtol=1e-5, atol=0.0) and float(top) == float(l1.max())
        # 22 bits, or half a step of lo at the end of its range
        limit = 2.0**-22 * want.double().abs() + (2.0**-36 / _scale(bound)).unsqueeze(1)
        assert bool(((_value(got, bound, d) - want.double()).abs() <= limit).all())


# The epilogues of the symmetric iterations: one tile, ragged edges, several tiles, wide tiles.
@pytest.mark.parametrize("sizes", [(1,), (33, 128), (200, 300, 31), (1500, 1500)])
def test_symmetric_products_on_pairs(ext, sizes):
    gen = torch.Generator(device="cuda").manual_seed(sum(sizes))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    bound = torch.tensor([8.0], device="cuda")
    fixed = (None, None, None, bound)
    specs, finals, checks = [], [], []
    stats = torch.zeros(len(sizes), 2, device="cuda")
    for i, n in enumerate(sizes):
        X = torch.randn(n, n, device="cuda", generator=gen)
        X = (X + X.T) / (2.0 * n**0.5)
        x, rows = _pairs(X)
        c = torch.randn(n, n, device="cuda", generator=gen) / n**0.5
        c = (c + c.T) / 2
        d = torch.full((n, _pad(n)), float("nan"), device="cuda")
        pitch = (n + 3) // 4 * 4
        hi, lo = (torch.full((n, pitch), float("nan"), device="cuda") for _ in range(2))
        XX = X.double() @ X.double().T
        checks.append((c, d, hi, lo, 2.0 * XX - 0.5 * c.double() + 0.7 * torch.eye(n, device="cuda"), 0.5 * XX + 0.5 * torch.eye(n, device="cuda"), n))
        sym = ext.FLAG_MIRROR | ext.FLAG_SPLIT_OUT | ext.FLAG_ADD_DIAG
        specs.append((x, None, x, None, c, d, None, None, c.stride(0), d.stride(0), sym | ext.FLAG_FIXED_SCALE, True, None, None, (rows, 1, rows, 1, fixed)))
        finals.append((x, None, x, None, None, hi, lo, stats[i], 0, pitch, sym | ext.FLAG_NO_C | ext.FLAG_SUMSQ | ext.FLAG_TRACE, True,
                       None, None, (rows, 1, rows, 1, None)))
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
    x, bound = _pairs(torch.ones(32, 32, device="cuda"))
    c, status = torch.zeros(32, 32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    spec = (x, None, x, None, c, None, None, None, 32, 0, 0, False)
    pairs = ext.build_gemm_plan([(*spec, None, None, (bound, 1, bound, 1, None))])
    plain = ext.build_gemm_plan([spec])
    with pytest.raises(RuntimeError, match="operand format"):
        ext.run_gemm_plan(*pairs, 1.0, 0.0, True, status)
    with pytest.raises(RuntimeError, match="operand format"):
        ext.run_gemm_plan(*plain, 1.0, 0.0, ext.HALF_PAIR, status)


# Rows and columns far below the others, in the Gram, in a product and in a chain of two.
@pytest.mark.parametrize("size", [1e-6, 1e-8, 1e-10, 1e-12])
@pytest.mark.parametrize("M,N", [(96, 120), (300, 260)])
def test_rows_and_columns_of_any_size_keep_their_precision(ext, M, N, size):
    gen = torch.Generator(device="cuda").manual_seed(M)
    F = torch.randn(M, N, device="cuda", generator=gen) * 1e-4
    F[3] *= size
    F[7] = 0.0
    F[:, 5] *= size
    L, R = (torch.eye(n, device="cuda") + torch.randn(n, n, device="cuda", generator=gen) * 1e-3 for n in (M, N))
    L, R = (L + L.T) / 2, (R + R.T) / 2
    for S, k in ((L, 3), (R, 5)):  # roots are large where gradients are small
        S[k] *= size**-0.5
        S[:, k] *= size**-0.5
    (f, f_bound), (l, l_bound), (r, r_bound) = _pairs(F), _pairs(L), _pairs(R)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    gram = torch.zeros(M, M, device="cuda")
    t, t_bound, top = torch.full((N, _pad(M)), float("nan"), device="cuda"), torch.full((N,), float("nan"), device="cuda"), torch.zeros(1, device="cuda")
    columns = torch.zeros(_pad(N), device="cuda")
    columns[:N] = F.abs().amax(0)
    ext.row_bounds(ext.build_row_bound_table([(r, r_bound, columns, t_bound, top)]))
    P = torch.zeros(M, N, device="cuda")
    for spec in (
        (f, None, f, None, gram, None, None, None, M, 0, 0, False, None, None, (f_bound, 1, f_bound, 1, None)),
        (r, None, f, None, None, t, None, None, 0, _pad(M), ext.FLAG_NO_C | ext.FLAG_SPLIT_OUT, False, None, None,
         (r_bound, 1, f_bound, 1, (None, None, None, t_bound))),
        (l, None, t, None, P, None, None, None, N, 0, 0, False, None, None, (l_bound, 1, t_bound, 1, None)),
    ):
        ext.run_gemm_plan(*ext.build_gemm_plan([spec]), 1.0, 0.0, ext.HALF_PAIR, status)
    L, F, R = L.double(), F.double(), R.double()
    want = R.abs() @ F.abs().amax(0)
    floor = 2.0**-38 * torch.outer(R.abs().amax(1), F.abs().amax(0)).sum(1)  # entries whose hi halves are subnormal
    assert bool((t_bound >= want).all()) and bool((t_bound <= 1.002 * (want + floor)).all()) and float(top) == float(t_bound.max())
    want = t_bound.double()
    # Every entry to the size of its own terms; below 2^-28 of its row's bound to half a step of lo, 2^-50 of the bound, per factor
    K, step = max(M, N), 2.0**-50
    norms = F.norm(dim=1)
    assert bool(((gram.double() - F @ F.T).abs() <= 2 * _bound(K) * torch.outer(norms, norms)).all())
    T_limit = _bound(K) * (R.abs() @ F.abs().T) + 3 * step * torch.outer(R.abs().sum(1), F.abs().amax(1)) + step * want.unsqueeze(1)
    assert bool(((_value(t, t_bound, M) - R @ F.T).abs() <= T_limit).all())
    limit = 2 * _bound(K) * (L.abs() @ F.abs() @ R.abs()) + L.abs() @ T_limit.T + 3 * step * torch.outer(L.abs().sum(1), want)
    assert bool(((P.double() - L @ F @ R).abs() <= limit).all())
    if size >= 1e-8:  # the range of the pairs: rows and columns of these sizes keep their precision, row by row and column by column
        for dim in (0, 1):
            norm = (L @ F @ R).norm(dim=dim).clamp_min(1e-300)
            assert float(((P.double() - L @ F @ R).norm(dim=dim) / norm).max()) < 4 * _bound(K) + 2.0**-20
    assert int(status) == 0


def test_rows_of_a_view_share_the_bound_of_the_row_they_were_written_with(ext):
    gen = torch.Generator(device="cuda").manual_seed(1)
    A = torch.randn(40, 64, device="cuda", generator=gen)
    B = torch.randn(5 * 6, 64, device="cuda", generator=gen) * torch.logspace(0, -9, 5, device="cuda").repeat_interleave(6).unsqueeze(1)
    (a, a_bound), (b, b_bound) = _pairs(A), _pairs(B, 6)
    c, status = torch.zeros(40, 30, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    spec = (a, None, b, None, c, None, None, None, 30, 0, 0, False, None, None)
    ext.run_gemm_plan(*ext.build_gemm_plan([(*spec, (a_bound, 1, b_bound, 6, None))]), 1.0, 0.0, ext.HALF_PAIR, status)
    ref = A.double() @ B.double().T
    assert float(((c.double() - ref).norm(dim=0) / ref.norm(dim=0)).max()) < _bound(64)
    with pytest.raises(RuntimeError, match="a bound per row"):
        ext.build_gemm_plan([(*spec, (a_bound, 1, b_bound, 5, None))])


# One tile, ragged tiles, a K loop cut among CTAs, wide tiles; two buffers of this GPU stand in for two ranks'.
@pytest.mark.parametrize("M,N,K", [(10, 77, 33), (3, 5, 98304), (130, 40, 5000), (2100, 2100, 40)])
@pytest.mark.parametrize("dtype,code", [(torch.float32, 0), (torch.bfloat16, 1), (torch.float16, 2)])
def test_pushed_products_on_pairs_are_the_stored_ones(ext, M, N, K, dtype, code):
    gen = torch.Generator(device="cuda").manual_seed(M + K)
    (a, a_bound), (b, b_bound) = (_pairs(torch.randn(n, K, device="cuda", generator=gen) * 0.1) for n in (M, N))
    status, norm, pushed_norm = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(1, device="cuda"), torch.zeros(1, device="cuda")
    c = torch.zeros(M, N, device="cuda")
    offset = 64  # elements in front of the problem's slot
    buffers = [torch.full((offset + M * N + 8,), 7.0, device="cuda", dtype=dtype) for _ in range(2)]
    bounds = (a_bound, 1, b_bound, 1, None)
    plain = ext.build_gemm_plan([(a, None, b, None, c, None, None, norm, N, 0, ext.FLAG_SUMSQ, False, None, None, bounds)])
    flags = ext.FLAG_SUMSQ | ext.FLAG_NO_C | ext.FLAG_PEER_PUSH
    push = ext.build_gemm_plan([(a, None, b, None, None, None, None, pushed_norm, N, 0, flags, False, offset * buffers[0].element_size(), None, bounds)])
    ext.run_gemm_plan(*plain, 1.0, 0.0, ext.HALF_PAIR, status)
    for _ in range(2):
        ext.run_gemm_plan_push(*push, 1.0, 0.0, ext.HALF_PAIR, status, [t.data_ptr() for t in buffers], code)
    for t in buffers:
        assert torch.equal(t[offset : offset + M * N].view(M, N), c.to(dtype))
        assert bool((t[:offset] == 7.0).all()) and bool((t[offset + M * N :] == 7.0).all())
    assert abs(float(pushed_norm) / (2 * float(norm)) - 1) < 1e-5
    assert int(status) == 0
