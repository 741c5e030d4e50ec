"""The FP32 product on the tensor cores (numbers cut in three): bits that do not depend on tile, split or neighbours, errors
against 64 bits, rows that TMA does not take, infinities and overflows, a wait that runs out."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _randn(*shape, seed=0, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(DEV)


def _exact(x, w):
    return x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()


def _bound(k, total):
    """Of an element's error, from the sum of |x| |w|: second parts are 2^-8 of a number at most, third ones 2^-16, so what is left out
    is 2^-23; 9 cuts (of 2^-23) of the large products while 64 columns are added up, 160 of the small ones, 2^-7 of them, in 256
    columns; a rounding (2^-24) per 64 and per 256 columns."""
    return total * (2.0 ** -23 + 9 * 2.0 ** -23 + 1.25 * 2.0 ** -23 + (k / 64 + k / 256 + 4) * 2.0 ** -24) + 1e-30


def _taken(m, k, rows, splits):
    """Whether a tile takes a split: a slice of 256 columns for each block, room for a block's sums and for those that arrive."""
    slices, (regions, ring) = -(-k // 256), {16: (18, 215040), 32: (8, 208896), 64: (4, 196608), 128: (2, 180224)}[rows]
    return splits == 1 or (splits <= slices and -(-slices // splits) <= regions
                           and slices * -(-min(m, rows) // splits) * 512 <= ring)


def _choices(ops, x, w, out):
    """Every tile and split that takes the product; the others, and no others, are refused."""
    for rows in (16, 32, 64, 128):
        for splits in (1, 2, 3, 4, 5, 8):
            if not _taken(x.shape[0], x.shape[1], rows, splits):
                with pytest.raises(ops.KernelError, match="bad argument"):
                    ops.gemm_f32_tc(x, w, out, rows, splits)
                continue
            ops.gemm_f32_tc(x, w, out, rows, splits)
            yield rows, splits


@pytest.mark.parametrize("m,n,k", [(1, 1, 4), (2, 128, 32), (15, 129, 64), (16, 127, 68), (17, 300, 256), (33, 5, 260), (64, 256, 1024),
                                   (64, 128, 2048), (128, 128, 2048), (177, 256, 2048), (65, 130, 1028), (130, 96, 2048), (3, 257, 8192), (129, 140, 4096), (40, 33, 1023)])
def test_every_tile_and_split_gives_the_same_bits(m, n, k):
    from nanoinfer_b200.kernels import ops
    x, w = _randn(m, k, seed=1), _randn(n, k, seed=2)
    want, total = _exact(x, w)
    first = torch.empty(m, n, device=DEV)
    ops.gemm_f32_tc(x, w, first)
    assert bool(((first.double() - want).abs() <= _bound(k, total)).all())
    out = torch.full((m, n), float("nan"), device=DEV)
    for choice in _choices(ops, x, w, out):
        assert torch.equal(out, first), choice
        out.fill_(float("nan"))
    row = torch.empty(1, n, device=DEV)
    ops.gemm_f32_tc(x[m - 1:], w, row)
    assert torch.equal(row[0], first[m - 1])
    ops.check_device_errors()


@pytest.mark.parametrize("k", [1024, 2048, 8192])
@pytest.mark.parametrize("positive", [False, True])
def test_errors_are_smaller_than_those_of_a_chain(k, positive):
    from nanoinfer_b200.kernels import ops
    x, w = _randn(48, k, seed=3), _randn(320, k, seed=4)
    if positive:
        x, w = x.abs(), w.abs()
    want, _ = _exact(x, w)
    cut, chain = torch.empty(48, 320, device=DEV), torch.empty(48, 320, device=DEV)
    ops.linear_f32(x, w, cut)
    ops.gemm_f32(x, w, chain)
    assert (cut.double() - want).norm() < (chain.double() - want).norm()


def _rows_of_few(kind, k):
    x, w = torch.zeros(64, k, device=DEV), _randn(320, k, seed=14)
    at = torch.arange(64, device=DEV)
    if kind == "one of 1":
        x[at, at * 13 % k] = 1.0
    elif kind == "one":
        x[at, at * 13 % k] = _randn(64, seed=13)
    elif kind == "ten":
        x = _randn(64, k, seed=13) * (torch.rand(64, k, generator=torch.Generator().manual_seed(15)).to(DEV) < 10 / k)
    elif kind == "one dominates":
        x = _randn(64, k, seed=13, scale=1e-4)
        x[at, at * 13 % k] = 3.0
    else:
        x, w = _randn(64, k, seed=13), torch.eye(320, k, device=DEV)
    return x, w


@pytest.mark.parametrize("k", [1024, 2048, 8192])
@pytest.mark.parametrize("kind", ["one of 1", "one", "ten", "one dominates", "identity"])
def test_rows_of_few_terms_are_as_exact_as_a_chain(kind, k):
    """Parts that hold whole numbers: a single product is rounded once, and weights (or activations) that meet a one come back as they
    were.  1.05: what is left out of a product, 2^-25 of it in the mean square, beside a rounding's 2^-24 / sqrt(3)."""
    from nanoinfer_b200.kernels import ops
    x, w = _rows_of_few(kind, k)
    want, _ = _exact(x, w)
    cut, chain = torch.empty(64, 320, device=DEV), torch.empty(64, 320, device=DEV)
    ops.linear_f32(x, w, cut)
    ops.gemm_f32(x, w, chain)
    assert (cut.double() - want).norm() <= 1.05 * (chain.double() - want).norm()
    if kind in ("one of 1", "identity"):
        assert torch.equal(cut, chain)


@pytest.mark.parametrize("rows,splits", [(16, 1), (16, 2), (32, 4), (64, 4), (128, 1), (128, 8)])
def test_numbers_near_the_ends_of_the_range(rows, splits):
    """Third parts of numbers below 2^-110 are beyond bfloat16: sums below 2^-80 (and from 2^100 on) are chains; beside ordinary
    numbers such ones lose 2^-133 at most."""
    from nanoinfer_b200.kernels import ops
    m, n, k = 40, 140, 2048
    x, w = _randn(m, k, seed=16), _randn(n, k, seed=17)
    x[3] *= 2.0 ** -120
    x[4] *= 2.0 ** -140                              # subnormal
    x[5] *= 2.0 ** 110
    x[6, ::2] *= 2.0 ** -122
    w[7, ::3] *= 2.0 ** -125
    w[8] = 0
    got, chain = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV)
    ops.gemm_f32_tc(x, w, got, rows, splits)
    ops.gemm_f32(x, w, chain)
    live = torch.arange(n, device=DEV) != 8
    for i in (3, 5):
        assert torch.equal(got[i, live], chain[i, live])
    assert (got[:, 8] == 0).all()
    want, total = _exact(x, w)
    lost = 2.0 ** -133 * (x.double().abs().sum(1)[:, None] + w.double().abs().sum(1)[None])
    ordinary = torch.ones(m, dtype=torch.bool, device=DEV)
    ordinary[5] = False
    assert bool(((got.double() - want).abs() <= _bound(k, total) - 1e-30 + lost)[ordinary].all())


@pytest.mark.parametrize("m,k,offset", [(3, 1040, 1), (20, 1036, 2), (70, 1024, 4), (5, 1031, 0)])
def test_heads_and_rows_of_a_wider_matrix(m, k, offset):
    """Rows off a 16-byte boundary are read number by number; the bits are those of aligned ones."""
    from nanoinfer_b200.kernels import ops
    h, n = 2, 137
    wide, w = _randn(m, h * k + 9, seed=5), _randn(h, n, k, seed=6)
    x = wide[:, offset:offset + h * k]
    out, rows = torch.empty(m, h * n, device=DEV), torch.empty(m, n, device=DEV)
    ops.linear_f32(x, w, out)
    for i in range(h):
        ops.linear_f32(x[:, i * k:(i + 1) * k].contiguous(), w[i].clone(), rows)
        assert torch.equal(out[:, i * n:(i + 1) * n], rows)


@pytest.mark.parametrize("rows,splits", [(16, 1), (16, 2), (64, 1), (128, 1)])
def test_what_is_not_finite_or_overflows_in_between(rows, splits):
    """Infinities, NaN and numbers whose parts overflow give what the chain gives; other rows are as without them."""
    from nanoinfer_b200.kernels import ops
    m, n, k = 19, 140, 512
    x, w = _randn(m, k, seed=7), _randn(n, k, seed=8)
    plain = torch.empty(m, n, device=DEV)
    ops.gemm_f32_tc(x, w, plain, rows, splits)
    x[2, 100], x[5, 3], x[7, 511] = float("inf"), float("-inf"), float("nan")
    x[9] = 2.0 ** 120 * x[9].sign()
    w[11, 17], w[12, 400] = float("inf"), float("nan")
    w[13] = 2.0 ** 110
    got, chain = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV)
    ops.gemm_f32_tc(x, w, got, rows, splits)
    ops.gemm_f32(x, w, chain)
    odd = torch.zeros(m, n, dtype=torch.bool, device=DEV)
    odd[[2, 5, 7, 9]] = True
    odd[:, [11, 12, 13]] = True
    assert torch.equal(got[~odd], plain[~odd])
    sure = torch.zeros_like(odd)                     # beyond FP32 in parts or in whole: recomputed as a chain
    sure[[2, 5, 7, 9]] = True
    sure[:, [11, 12]] = True
    torch.testing.assert_close(got[sure], chain[sure], rtol=0, atol=0, equal_nan=True)
    want, total = _exact(x, w)
    fine = odd & ~sure & want.isfinite()
    assert bool(((got.double() - want).abs()[fine] <= _bound(k, total)[fine]).all())


def test_rows_that_a_chain_takes_or_refuses():
    """One product's x is contiguous whatever its length; the strides of a single row do not matter."""
    from nanoinfer_b200.kernels import ops
    w = _randn(140, 1024, seed=18)
    with pytest.raises(ops.KernelError, match="contiguous"):
        ops.linear_f32(_randn(5, 1040, seed=19)[:, :1024], w, torch.empty(5, 140, device=DEV))
    column = _randn(1024, 1, seed=20)
    out, want = torch.empty(1, 140, device=DEV), torch.empty(1, 140, device=DEV)
    ops.linear_f32(column.t(), w, out)                # [1, 1024], strides 1 and 1
    ops.linear_f32(column.view(1, 1024), w, want)
    assert torch.equal(out, want)


def test_a_rule_by_the_length_of_a_row_alone():
    from nanoinfer_b200.kernels import ops
    for k in (1020, 1024):
        x, w = _randn(200, k, seed=9), _randn(260, k, seed=10)
        out = torch.empty(200, 260, device=DEV)
        ops.linear_f32(x, w, out)
        for m in (1, 9, 40, 100):
            rows = torch.empty(m, 260, device=DEV)
            ops.linear_f32(x[50:50 + m].contiguous(), w, rows)
            assert torch.equal(rows, out[50:50 + m])


def test_a_wait_that_runs_out_is_recorded_and_the_kernel_returns():
    from nanoinfer_b200.kernels import ops
    x, w = _randn(16, 1024, seed=11), _randn(256, 1024, seed=12)
    for splits in (1, 4):
        first, out = torch.empty(16, 256, device=DEV), torch.empty(16, 256, device=DEV)
        ops.gemm_f32_tc(x, w, first, 16, splits)
        torch.cuda.synchronize()
        ops.check_device_errors()
        ops.set_wait_limit("gemm_f32_tc", 2_000_000, extra_wait=True)           # about a millisecond
        try:
            ops.gemm_f32_tc(x, w, out, 16, splits)
            torch.cuda.synchronize()
            with pytest.raises(ops.KernelError, match="code 54"):
                ops.check_device_errors()
            assert torch.equal(out, first)
        finally:
            ops.set_wait_limit("gemm_f32_tc", 0, extra_wait=False)
        ops.gemm_f32_tc(x, w, out.zero_(), 16, splits)
        torch.cuda.synchronize()
        ops.check_device_errors()
        assert torch.equal(out, first)
