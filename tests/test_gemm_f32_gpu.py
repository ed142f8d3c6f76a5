"""The true float32 product at the edges of its tiles and variants: against float64, and the same
bits for a row whatever rows it is computed with."""

import pytest
import torch

from mini_llm_stack_b200.ops.kernels import Runtime

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    return Runtime("cuda:0", torch.bfloat16).ops


@pytest.mark.parametrize("a_type", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("m, n, k", [
    (1, 257, 16), (31, 300, 17), (33, 5120, 40), (65, 19000, 64), (97, 9473, 33), (64, 9472, 4),
    (1, 1, 1), (3, 1000, 132), (8, 260, 64), (5, 19001, 72), (63, 65, 130), (64, 65, 132), (65, 9, 36), (700, 65, 256), (130, 256, 1028), (2100, 8, 24),
    (1501, 64, 132), (1200, 64, 65)])
def test_product(ops, a_type, m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m * n + k)
    a = torch.randn(m, k, device="cuda", generator=g).to(a_type)
    w = torch.randn(n, k, device="cuda", generator=g)
    out = torch.full((m, n), float("nan"), device="cuda")
    ops.linear(a, w, out)
    want = a.double() @ w.double().T
    # float32 sums of k products of unit size: k roundings of a partial sum, 2^-24 each
    bound = 2.0 ** -24 * (k + 2) * (a.double().abs() @ w.double().abs().T)
    assert ((out.double() - want).abs() <= bound + 1e-30).all()
    some = sorted({0, m // 2, m - 1})
    few = torch.empty(len(some), n, device="cuda")
    ops.linear(a[some].contiguous(), w, few)
    assert torch.equal(few, out[some])


@pytest.mark.parametrize("a_type", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("off_a, off_w", [(1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("m, n, k", [(5, 33, 64), (100, 33, 64), (1500, 70, 64), (90, 300, 64)])
def test_rows_between_addresses(ops, a_type, off_a, off_w, m, n, k):
    """Operands that cannot be read four entries at a time although their rows are whole quads."""
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn(m * k + 1, device="cuda", generator=g).to(a_type)[off_a:][:m * k].view(m, k)
    w = torch.randn(n * k + 1, device="cuda", generator=g)[off_w:][:n * k].view(n, k)
    out = torch.full((m, n), float("nan"), device="cuda")
    ops.linear(a, w, out)
    bound = 2.0 ** -24 * (k + 2) * (a.double().abs() @ w.double().abs().T)
    assert ((out.double() - a.double() @ w.double().T).abs() <= bound + 1e-30).all()
