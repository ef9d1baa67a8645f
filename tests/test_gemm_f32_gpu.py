"""The float32 product on the tensor cores (``ops.gemm_f32_tcgen05``) against 64 bits and against the library's float32 product:
one element past and short of a tile, K short of a slab, of one group of slabs and of many, with K in shares."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,n,k,splits", [(1, 4, 4, 1), (127, 132, 60, 1), (128, 128, 64, 1), (129, 260, 132, 1), (300, 384, 1024, 1),
                                             (300, 384, 1024, 3), (64, 1024, 2048, 5), (595, 4096, 1024, 1), (2, 132, 1028, 17), (1500, 2560, 196, 2)])
def test_against_64_bits(rows, n, k, splits):
    from tiny_llm_infer_b200 import ops
    from tiny_llm_infer_b200.engine.runner import strict_float32
    strict_float32()
    g = torch.Generator(device="cuda").manual_seed(rows + k)
    x = torch.randn(rows, k, generator=g, device="cuda") * torch.exp(torch.randn(rows, 1, generator=g, device="cuda") * 3)
    w = torch.randn(n, k, generator=g, device="cuda") * 0.02
    want = x.double() @ w.double().t()
    y, lib = ops.gemm_f32_tcgen05(x, w, splits), torch.mm(x, w.t())
    ops.check_error_word("cuda")
    scale = want.norm(dim=1, keepdim=True)
    error, lib_error = (((t.double() - want) / scale).norm() / rows ** 0.5 for t in (y, lib))
    # a few roundings of 2^-24 whatever K is: 128 terms at a time are cut off at most 8 ulps below their sum, their sums add up rounded
    assert error <= max(1.2 * float(lib_error), 3e-7), (float(error), float(lib_error))
    # rows and columns keep to themselves: a row of no numbers and an infinite weight spoil nothing else
    if rows > 1:
        x2, w2 = x.clone(), w.clone()
        x2[rows // 2] = float("nan")
        w2[n // 2, k // 2] = float("inf")
        y2 = ops.gemm_f32_tcgen05(x2, w2, splits)
        keep_r, keep_c = torch.arange(rows, device="cuda") != rows // 2, torch.arange(n, device="cuda") != n // 2
        assert torch.equal(y2[keep_r][:, keep_c], y[keep_r][:, keep_c])
        assert torch.isnan(y2[rows // 2]).all() and not torch.isfinite(y2[:, n // 2]).any()


@pytest.mark.parametrize("rows,n,k,splits", [(129, 260, 132, 1), (300, 384, 1024, 1), (300, 384, 1024, 3), (64, 1024, 2048, 5)])
def test_infinities_and_overflows_are_those_of_a_float32_product(rows, n, k, splits):
    """Infinite operands, among them beside weights that one bfloat16 holds whole, sums that overflow, and finite numbers that no
    bfloat16 is as large as: infinite, not a number or finite wherever the library's product is, of the same sign."""
    from tiny_llm_infer_b200 import ops
    from tiny_llm_infer_b200.engine.runner import strict_float32
    strict_float32()
    g = torch.Generator(device="cuda").manual_seed(rows + k)
    x = torch.randn(rows, k, generator=g, device="cuda")
    w = torch.randn(n, k, generator=g, device="cuda") * 0.02
    plain = ops.gemm_f32_tcgen05(x, w, splits)
    w[:, 5] = 0.5
    w[1::2, 5] = -0.5
    x[3, 5] = float("inf")                                         # an infinity of each sign per column
    x[7, 5], x[7, 9] = float("inf"), -float("inf")                 # and both, by the column no number
    x[11, 5] = 3.4e38                                              # rounds to an infinity in bfloat16; its products are finite
    x[12, 5], x[13, 5] = 3.4e38, float("nan")
    w[n // 2, 5] = 4.0                                             # overflows with row 11
    w[n - 1, 5] = 0.0                                              # infinity times zero
    w[2, k - 1] = -float("inf")
    want, got = torch.mm(x, w.t()), ops.gemm_f32_tcgen05(x, w, splits)
    ops.check_error_word("cuda")
    assert torch.isinf(want).any() and torch.isnan(want).any() and torch.isinf(want[3]).sum() >= n - 2
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    assert torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
    fine = torch.isfinite(want)
    assert ((got - want)[fine].abs() <= 1e-5 * want[fine].abs() + 1e-5).all()      # sums of k products, in another order
    # rows and columns that have none of it keep their bits
    w2, rest = w.clone(), torch.ones(rows, dtype=torch.bool, device="cuda")
    w2[2, k - 1] = 0.0
    rest[[3, 7, 11, 12, 13]] = False
    columns = torch.arange(n, device="cuda") != 2
    assert torch.equal(got[rest][:, columns], ops.gemm_f32_tcgen05(x, w2, splits)[rest][:, columns]) and torch.isfinite(plain).all()
