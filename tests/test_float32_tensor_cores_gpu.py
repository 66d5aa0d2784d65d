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


@pytest.fixture
def ran(ops, monkeypatch):
    """The launchers that ``linear`` asks for, in order: a refused size would come out of the other kernel, right and unseen."""
    names, fn = [], ops._fn
    monkeypatch.setattr(ops, "_fn", lambda name, what=None: (names.append(name), fn(name, what))[1])
    return names


def plain_kernel(ops, a, w, out):
    (m, k), n = a.shape, w.shape[0]
    assert ops._fn("stride_gemm_nt_f32")(a.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, k, k, n, ops._stream()) == 0


# smallest sizes, a broken tile of W and of K, a broken last part, parts of more than 1,024 (K above 8,192), a part of one block
@pytest.mark.parametrize("n,k", [(512, 512), (513, 520), (700, 1032), (1280, 3080), (640, 8264), (514, 2056)])
def test_bits_do_not_depend_on_the_batch_and_the_error_is_bounded(ops, ran, n, k):
    g = torch.Generator(device="cuda").manual_seed(n + k)
    a, w = torch.randn(337, k, generator=g, device="cuda"), torch.randn(n, k, generator=g, device="cuda")
    full = torch.empty(337, n, device="cuda")
    ops.linear(a, w, full)
    # Of sum |a_i w_i|: 2^-24 for every rounded sum of 64 terms, every part of K and the last; inside 64 terms four steps of 16 that cut off at most
    # a last place (2^-23) each and as much for what a step of 16 loses inside; the same for the other products (7 times as many steps in a
    # whole part), 2^-5 of the sum at most; and the product that is left out (2^-30)
    blocks = -(-k // 64)
    bound = (blocks + 10 + 16 + 7 * 16 * blocks / 32) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    error = (full.double() - a.double() @ w.double().T).abs()
    assert bool((error <= bound).all())
    chains = torch.empty_like(full)
    plain_kernel(ops, a, w, chains)
    other = (chains.double() - a.double() @ w.double().T).square().mean()
    assert float(error.square().mean()) < 0.36 * float(other), "not 0.6 of the multiply-adds' error (measured: 0.43 at K = 512, less beyond)"
    for m in (1, 15, 16, 17, 48, 49, 96, 97, 160, 161, 336):
        out = torch.full((m + 1, n), 7.0, device="cuda")
        ops.linear(a[:m], w, out[:m])
        assert torch.equal(out[:m], full[:m]) and bool((out[m] == 7.0).all()), m
    assert ops.tc_status() == 0 and set(ran) == {"stride_gemm_nt_f32_tc", "stride_gemm_nt_f32"} and ran.count("stride_gemm_nt_f32") == 1


# Rows and weights of one sign, of one term, and far apart from one another; short K too: no further from float64 than the multiply-adds, but for
# one rounding where there is nothing else (one term: 2^-24 and the 2^-30 that is left out).
@pytest.mark.parametrize("k", [512, 1024, 3072])
@pytest.mark.parametrize("kind", ["normal", "uniform", "near one", "constant", "one term", "four terms", "either sign, far apart"])
def test_error_beside_the_multiply_adds(ops, ran, kind, k):
    g = torch.Generator(device="cuda").manual_seed(k)
    m, n = 200, 1024
    r, u = (lambda *s: torch.randn(*s, generator=g, device="cuda")), (lambda *s: torch.rand(*s, generator=g, device="cuda"))
    a, w = {"normal": lambda: (r(m, k).abs(), r(n, k).abs()), "uniform": lambda: (u(m, k), u(n, k)), "near one": lambda: (1 + u(m, k), 1 + u(n, k)),
            "constant": lambda: (torch.full((m, k), 1 / 3, device="cuda"), 1 + u(n, k)), "one term": lambda: (torch.zeros(m, k, device="cuda"), 1 + u(n, k)),
            "four terms": lambda: (torch.zeros(m, k, device="cuda"), 1 + u(n, k)),
            "either sign, far apart": lambda: (torch.exp(3 * r(m, k)) * r(m, k).sign(), torch.exp(3 * r(n, k)) * r(n, k).sign())}[kind]()
    for _ in range({"one term": 1, "four terms": 4}.get(kind, 0)):
        a[torch.arange(m, device="cuda"), torch.randint(0, k, (m,), generator=g, device="cuda")] = 1 + u(m)
    out, chains = torch.empty(m, n, device="cuda"), torch.empty(m, n, device="cuda")
    ops.linear(a, w, out)
    plain_kernel(ops, a, w, chains)
    want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    mine, theirs = (((x.double() - want) / size) for x in (out, chains))
    assert float(mine.square().mean().sqrt()) <= 1.01 * float(theirs.square().mean().sqrt())
    assert float(mine.abs().max()) <= max(float(theirs.abs().max()), 2.0 ** -24 + 2.0 ** -28)       # the sum of the other products has 2^-28 of its own
    assert ran == ["stride_gemm_nt_f32_tc", "stride_gemm_nt_f32"]


@pytest.mark.parametrize("exponent", [-140, -125, -110, -60, 60, 100])
def test_numbers_far_from_one_keep_their_bits(ops, ran, exponent):
    """Numbers whose bfloat16 parts would be subnormal, and subnormal float32 themselves, lose nothing; from 2^70 on the multiply-adds do it."""
    g = torch.Generator(device="cuda").manual_seed(5)
    a, w = torch.randn(70, 1024, generator=g, device="cuda"), torch.randn(512, 1024, generator=g, device="cuda")
    far_a, far_w = a.double().mul(2.0 ** exponent).float(), w.double().mul(2.0 ** min(-exponent, 60)).float()
    out, chains = torch.empty(70, 512, device="cuda"), torch.empty(70, 512, device="cuda")
    ops.linear(far_a, far_w, out)
    plain_kernel(ops, far_a, far_w, chains)
    want = far_a.double() @ far_w.double().T
    size = far_a.double().abs() @ far_w.double().abs().T
    assert float(((out.double() - want) / size).square().mean()) <= 1.02 * float(((chains.double() - want) / size).square().mean())
    assert ran[0] == "stride_gemm_nt_f32_tc"


@pytest.mark.parametrize("m", [3, 40, 70, 200])
def test_rows_off_a_16_byte_boundary(ops, ran, m):
    g = torch.Generator(device="cuda").manual_seed(m)
    memory, w = torch.randn(m * 1024 + 1, generator=g, device="cuda"), torch.randn(600, 1024, generator=g, device="cuda")
    odd = memory[1:].view(m, 1024)
    out, want = torch.empty(m, 600, device="cuda"), torch.empty(m, 600, device="cuda")
    ops.linear(odd, w, out)
    ops.linear(odd.clone(), w, want)
    assert odd.data_ptr() % 16 == 4 and torch.equal(out, want) and ran == ["stride_gemm_nt_f32_tc"] * 2


def test_what_the_kernel_does_not_take_runs_as_multiply_adds_without_scratch(ops, ran):
    for n, k, off in ((600, 1028, 0), (600, 1024, 1), (500, 1024, 0), (600, 504, 0)):
        a, memory = torch.randn(100, k, device="cuda"), torch.randn(n * k + 1, device="cuda")
        w, out, want = memory[off:off + n * k].view(n, k), torch.empty(100, n, device="cuda"), torch.empty(100, n, device="cuda")
        plain_kernel(ops, a, w, want)
        del ran[:]
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        ops.linear(a, w, out)
        assert torch.cuda.max_memory_allocated() == before
        assert ran == ["stride_gemm_nt_f32"] and torch.equal(out, want)


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
