"""The float32 product of large matrices on the tensor cores (three bfloat16 parts a number): against float64 within a bound of its sums,
the same bits for a row in every batch, and what is no finite number as the kernel of fused multiply-adds has it."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from stride_b200.csrc import ops as _ops
    kept, _ops.F32_TC_WEIGHTS = _ops.F32_TC_WEIGHTS, 0          # small matrices too
    yield _ops
    _ops.F32_TC_WEIGHTS = kept


def plain_kernel(ops, a, w, out):
    (m, k), n = a.shape, w.shape[0]
    assert ops._fn("stride_gemm_nt_f32")(a.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, k, k, n, ops._stream()) == 0


# smallest sizes, a broken tile of W and of K, a broken last part, parts of more than 1,024 (K above 8,192), a part of one block
@pytest.mark.parametrize("n,k", [(512, 512), (513, 520), (700, 1032), (1280, 3080), (640, 8264), (514, 2056)])
def test_bits_do_not_depend_on_the_batch_and_the_error_is_bounded(ops, n, k):
    g = torch.Generator(device="cuda").manual_seed(n + k)
    a, w = torch.randn(337, k, generator=g, device="cuda"), torch.randn(n, k, generator=g, device="cuda")
    full = torch.empty(337, n, device="cuda")
    ops.linear(a, w, full)
    # Of sum |a_i w_i|: 2^-24 for every rounded sum of 64 terms and every part; inside 64 terms four steps of 16 that cut off at most a
    # last place (2^-23) each, as much for what a step of 16 loses inside, and the products that are left out (2^-22 at most)
    blocks = -(-k // 64)
    bound = (-(-blocks // min(8, -(-k // 1024))) + 8 + 16 + 4) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    error = (full.double() - a.double() @ w.double().T).abs()
    assert bool((error <= bound).all())
    chains = torch.empty_like(full)
    plain_kernel(ops, a, w, chains)
    assert float(error.square().mean()) <= float((chains.double() - a.double() @ w.double().T).square().mean()), "further off than multiply-adds"
    for m in (1, 15, 16, 17, 48, 49, 96, 97, 160, 161, 336):
        out = torch.full((m + 1, n), 7.0, device="cuda")
        ops.linear(a[:m], w, out[:m])
        assert torch.equal(out[:m], full[:m]) and bool((out[m] == 7.0).all()), m
    assert ops.tc_status() == 0


@pytest.mark.parametrize("m", [3, 70, 200])
def test_what_is_not_finite_comes_out_as_from_multiply_adds(ops, m):
    g = torch.Generator(device="cuda").manual_seed(m)
    a, w = torch.randn(m, 1024, generator=g, device="cuda"), torch.randn(600, 1024, generator=g, device="cuda")
    a[1, 1000], a[2, 3], a[0, 9], w[3, 5], w[77, 1], w[500, 8] = 3.4e38, float("nan"), 1e-42, float("inf"), -3.4e38, float("-inf")
    out, want = torch.empty(m, 600, device="cuda"), torch.empty(m, 600, device="cuda")
    ops.linear(a, w, out)
    plain_kernel(ops, a, w, want)
    finite = want.isfinite()
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out[want.isinf()], want[want.isinf()]) and bool(out[finite].isfinite().all())
    close = finite & (want.abs() < 1e30)
    assert float((out[close] - want[close]).abs().max()) < 1e-3         # sums of 1,024 terms of about 1


def test_slabs_of_rows_give_the_same_bits(ops):
    a, w = torch.randn(1500, 8192, device="cuda"), torch.randn(512, 8192, device="cuda")       # 64 MB of parts: 1,280 rows at a time
    full, out = torch.empty(1500, 512, device="cuda"), torch.empty(300, 512, device="cuda")
    ops.linear(a, w, full)
    ops.linear(a[1200:], w, out)
    assert torch.equal(full[1200:], out)
