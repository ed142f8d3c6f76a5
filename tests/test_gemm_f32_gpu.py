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


@pytest.mark.parametrize("a_type", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("m, n, k", [
    (1, 257, 2048), (16, 300, 2052), (17, 260, 2304), (33, 2048, 2080), (161, 385, 2056), (170, 4100, 2048),
    (700, 1000, 8196), (16, 4096, 4096), (200, 300, 5000), (1, 257, 8188), (5, 16384, 512), (321, 16500, 548), (1, 64, 4096), (129, 65, 4100), (1030, 130, 4104)])
def test_product_on_tensor_cores(ops, a_type, off, m, n, k):
    """Sizes around the edges of its tiles, blocks and groups: nearer to float64 than a chain over k could
    be, and the same bits for a row whatever rows it is computed with (cut along K or not)."""
    g = torch.Generator(device="cuda").manual_seed(m * n + k + off)
    a = torch.randn(m * k + 1, device="cuda", generator=g).to(a_type)[off:][:m * k].view(m, k)
    w = torch.randn(n, k, device="cuda", generator=g)
    out = torch.full((m, n), float("nan"), device="cuda")
    ops.linear(a, w, out)
    want = a.double() @ w.double().T
    # parts left out: 3 of a product's 9, 2^-25 of it together at the most in the root mean square of many;
    # sums: 2^-23 a step of four cut ones over 64 of k, 2^-24 rounded a block of 64 and a group
    steps = 4 * 2 + (k + 63) // 64 / 8 + 8
    size = (a.double().abs() @ w.double().abs().T)
    assert ((out.double() - want).abs() <= 2.0 ** -24 * (2 + steps) * size).all()
    assert (out.double() - want).norm() <= 2e-7 * want.norm()
    some = sorted({0, m // 2, m - 1})
    few = torch.empty(len(some), n, device="cuda")
    ops.linear(a[some].contiguous(), w, few)
    assert torch.equal(few, out[some])
    ops.check_status()


@pytest.mark.parametrize("m", [4, 200])
def test_odd_values_on_tensor_cores(ops, m):
    """Infinities, values that are no numbers, and values at both ends of float32's range: what a chain
    of float32 products and sums gives."""
    n, k = 300, 2048
    g = torch.Generator(device="cuda").manual_seed(m)
    a, w = torch.randn(m, k, device="cuda", generator=g), torch.randn(n, k, device="cuda", generator=g)
    a[0, 5], a[1, 7], a[2, :] = float("inf"), float("nan"), a[2] * 1e37
    a[3] *= 2.0 ** -60
    w[4, 9], w[6, 2], w[8] = 3.4e38, float("-inf"), w[8] * 2.0 ** -40
    out = torch.empty(m, n, device="cuda")
    ops.linear(a, w, out)
    want = a.double() @ w.double().T
    size = a.double().abs() @ w.double().abs().T
    plain = size < 3e38                                   # no partial sum beyond float32's range
    assert ((out.double() - want).abs()[plain] <= 2.0 ** -24 * 24 * size[plain]).all()
    assert (out[0, 0].isinf() or out[0, 0].isnan()) and out[1].isnan().all()
    # an infinite product decides a sum as in a chain: infinite where no other one is of the other sign
    sure = torch.ones(m, n, dtype=torch.bool, device="cuda")
    sure[:, 4] = sure[:, 6] = False
    sure[1:] = False
    assert (out[sure] == torch.where(a[0, 5] * w[:, 5] > 0, float("inf"), float("-inf")).expand(m, n)[sure]).all()
    ops.check_status()


@pytest.mark.parametrize("a_type", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("m", [3, 200])
@pytest.mark.parametrize("power_a, power_w, chain", [
    (-112, 100, False), (-120, 100, False), (-130, 100, False), (100, -112, False), (100, -120, False), (100, -140, False),
    (-60, -62, False), (30, 40, False), (-130, 120, True), (60, 60, True)])   # from 2^112, sums from 2^96 on
def test_operands_of_all_sizes_on_tensor_cores(ops, a_type, m, power_a, power_w, chain):
    """Operands whose lower parts would lie below bfloat16's smallest number, down to float32's own smallest, against
    large ones (the products are ordinary numbers): all 24 bits count.  What is too large goes to a chain over k."""
    n, k = 300, 2048
    g = torch.Generator(device="cuda").manual_seed(m + power_a)
    a = (torch.randn(m, k, device="cuda", generator=g) * 2.0 ** power_a).to(a_type)
    w = torch.randn(n, k, device="cuda", generator=g) * 2.0 ** power_w
    want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert a.any() and w.any() and want.abs().max() < 3e38
    out = torch.empty(m, n, device="cuda")
    ops.linear(a, w, out)
    # as in test_product_on_tensor_cores (4 steps a 64 of k of 2^-23, k / 64 / 8 and 8 of 2^-24); a chain's k roundings
    steps = k + 2 if chain else 2 + 8 + k / 512 + 8
    assert ((out.double() - want).abs() <= 2.0 ** -24 * steps * size).all()
    assert chain or (out.double() - want).norm() <= 2e-7 * want.norm()
    ops.check_status()


@pytest.mark.parametrize("a_type, m, n, k, share", [(torch.float32, 700, 300, 2048, 8), (torch.bfloat16, 333, 300, 2052, 8),
                                                    (torch.float32, 40, 2048, 8192, 2)])
def test_scratch_has_a_bound_and_memory_may_run_out(ops, monkeypatch, a_type, m, n, k, share):
    """Rows in parts give the same bits: by the bound, and after the allocator has refused what the whole takes."""
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn(m, k, device="cuda", generator=g).to(a_type)
    w = torch.randn(n, k, device="cuda", generator=g)
    whole, out = torch.empty(m, n, device="cuda"), torch.full((m, n), float("nan"), device="cuda")
    monkeypatch.setattr(ops, "_scratch", {})
    ops.linear(a, w, whole)
    most = ops._scratch["gemm_f32"].numel()
    assert most & (most - 1) == 0                         # grows by powers of two
    # a bound
    limit = most // share
    monkeypatch.setattr(ops, "F32_SCRATCH", limit, raising=False)
    monkeypatch.setattr(ops, "_scratch", {})
    ops.linear(a, w, out)
    assert torch.equal(out, whole) and ops._scratch["gemm_f32"].numel() <= max(limit, 1 << 16)
    # an allocator that has less than the whole takes
    monkeypatch.setattr(ops, "F32_SCRATCH", 1 << 26, raising=False)
    monkeypatch.setattr(ops, "_scratch", {})
    real = ops.scratch

    def scratch(tag, floats):
        if floats > limit:
            raise torch.cuda.OutOfMemoryError("none left")
        return real(tag, floats)
    monkeypatch.setattr(ops, "scratch", scratch)
    out.fill_(float("nan"))
    ops.linear(a, w, out)
    assert torch.equal(out, whole) and ops.F32_SCRATCH < most
    ops.check_status()


@pytest.mark.parametrize("a_type, m, n, k, count", [
    (torch.float32, 700, 3000, 2048, 2),       # rows split, product
    (torch.float32, 1, 2048, 2048, 3),         # and sums of the groups of a cut product
    (torch.bfloat16, 1, 64, 4096, 2),          # rows that are their own part
    (torch.bfloat16, 3000, 4000, 2048, 1),
    (torch.float32, 5, 300, 64, 1)])           # CUDA cores
def test_launches_are_counted(ops, a_type, m, n, k, count):
    """As many as a captured call has nodes."""
    from cuda.bindings import runtime
    a = torch.ones(m, k, device="cuda", dtype=a_type)
    w, out = torch.ones(n, k, device="cuda"), torch.empty(m, n, device="cuda")
    ops.linear(a, w, out)
    before, graph = ops.launches, torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        ops.linear(a, w, out)
    error, _, nodes = runtime.cudaGraphGetNodes(runtime.cudaGraph_t(graph.raw_cuda_graph()), 0)
    assert int(error) == 0 and ops.launches - before == count == nodes


@pytest.mark.parametrize("what", ["every value", "one value a row", "one row of weights"])
@pytest.mark.parametrize("m, n, k", [(515, 2048, 2048), (16, 2048, 8192)])
def test_values_that_are_no_numbers_do_not_hold_a_product_up(ops, what, m, n, k):
    """Right, and at most ninety times the time of ordinary values (up to 35; an output at a time took 220)."""
    a, w = torch.randn(m, k, device="cuda"), torch.randn(n, k, device="cuda")
    odd, odd_w = a.clone(), w.clone()
    if what == "every value":
        odd[:] = float("nan")
    elif what == "one value a row":
        odd[:, k // 2] = float("inf")
    else:
        odd_w[5, 7] = float("nan")
    out = torch.empty(m, n, device="cuda")

    def time(a, w):
        best = float("inf")
        for _ in range(4):
            begin, end = torch.cuda.Event(True), torch.cuda.Event(True)
            begin.record()
            ops.linear(a, w, out)
            end.record()
            torch.cuda.synchronize()
            best = min(best, begin.elapsed_time(end))
        return best
    plain = time(a, w)
    assert time(odd, odd_w) <= 90 * plain
    if what == "every value":
        assert out.isnan().all()
    elif what == "one value a row":
        assert (out == torch.where(w[:, k // 2] > 0, float("inf"), float("-inf"))).all()
    else:
        assert out[:, 5].isnan().all() and out[:, :5].isfinite().all() and out[:, 6:].isfinite().all()
    ops.check_status()
