"""The float32 product on the tensor cores (operands split into three bfloat16 values): every form of it against float64 and against each
other, rows of a single term, and the values that have no split."""
import pytest
import torch

from x0ne_engine_b200.csrc import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
FORMS = [(16, 1), (16, 2), (16, 4), (16, 8), (32, 1), (32, 4), (32, 8), (64, 1), (64, 4), (64, 8), (96, 1)]
# Of a sum of |x w|: 2^-32 for what the split leaves out of each product (its two lowest parts, 2^-16 times 2^-16), 2^-22 for the tensor core cutting
# off the sums of a slab of 32 values (two products of 16), 2^-24 for each float32 addition of a slab or a part, and of the part's small products
# (2^-7 of the sum) 2^-23 for each of their 10 sums a slab.
BOUND = lambda k: 2.0 ** -32 + 2.0 ** -22 + (-(-k // 256) + 10) * 2.0 ** -24 + 10 * -(-k // 256) * 2.0 ** -30


def product(x, w, y, m, nx=0, cl=0):
    lib = ops._lib("core")
    ops._check(lib, lib.x0ne_gemm_f32_split(ops._ptr(x), ops._ptr(w), ops._ptr(y), m, w.shape[0], w.shape[1], w.shape[1], w.shape[1], w.shape[0], 1, 0, 0, 0,
                                            nx * 16 + cl, ops._ptr(ops.gemm_tc_status(x.device)), ops._stream()), "gemm_f32_split")


def normal(shape, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.randn(shape, device=DEV, generator=g)


# slabs of 32 values of k: 16, a ragged 17th, parts without a slab (17 in parts of 3), rows of W that TMA cannot address; ragged tiles of both operands
@pytest.mark.parametrize("n,k", [(1, 512), (128, 516), (257, 541), (384, 1000), (129, 2048)])
def test_every_form_gives_the_same_bits(n, k):
    rows = 131
    x, w = normal((rows, k), 1), normal((n, k), 2)
    exact, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    want = None
    for nx, cl in FORMS:
        y = torch.full((rows + 1, n), 3.0, device=DEV)
        product(x, w, y, rows, nx, cl)
        want = y[:rows].clone() if want is None else want
        assert torch.equal(y[:rows], want) and bool((y[rows] == 3.0).all()), (nx, cl)
    assert bool(((want.double() - exact).abs() <= BOUND(k) * size).all())
    for m in (1, 8, 9, 17, 33, 65, 97, 128):            # the rule's choices, of rows alone
        y = torch.full((m + 1, n), 3.0, device=DEV)
        ops.gemm_f32_nt(x[rows - m:].contiguous(), w, y, m)
        assert torch.equal(y[:m], want[rows - m:]) and bool((y[m] == 3.0).all()), m
    odd = torch.zeros((rows * k + 1,), device=DEV)[1:].view(rows, k)        # rows that do not start on 16 bytes
    odd.copy_(x)
    y = torch.zeros((rows, n), device=DEV)
    ops.gemm_f32_nt(odd, w, y, rows)
    assert torch.equal(y, want)
    ops.check_tc_status(x.device)


def test_rows_of_a_single_term():
    """Nothing is lost where there is nothing to add: an identity gives x back, and a product alone is rounded once (2^-24, and 2^-29 in the
    sum of its small parts), in a row of zeros and beside terms that do not reach its last bit."""
    k = 640
    x = normal((33, k), 10)
    for nx, cl in FORMS:
        y = torch.zeros((33, k), device=DEV)
        product(x, torch.eye(k, device=DEV), y, 33, nx, cl)
        assert torch.equal(y, x), (nx, cl)
    w = normal((200, k), 11)
    at = torch.arange(33, device=DEV) * 19
    alone, beside = torch.zeros((33, k), device=DEV), normal((33, k), 12) * 2.0 ** -40
    for rows, slack in ((alone, 0.0), (beside, 2.0 ** -24)):
        rows[torch.arange(33), at] = normal((33,), 13) + 3.0
        y = torch.zeros((33, 200), device=DEV)
        ops.gemm_f32_nt(rows, w, y, 33)
        exact = rows.double() @ w.double().T
        term = (rows[torch.arange(33), at].double()[:, None] * w.double()[:, at].T).abs()
        rest = rows.double().abs() @ w.double().abs().T - term
        assert bool(((y.double() - exact).abs() <= (2.0 ** -24 + 2.0 ** -29) * exact.abs() + rest + slack * term).all())
    ops.check_tc_status(x.device)


def test_operands_of_far_apart_sizes():
    """Operands near the low end of the float32 range whose products are of ordinary size: no room for their last bits below."""
    k = 512
    x, w = normal((20, k), 14), normal((140, k), 15)
    x[3], w[100:110] = x[3] * 2.0 ** -112, w[100:110] * 2.0 ** 90
    x[4] *= 2.0 ** -130
    want = x.double() @ w.double().T
    size = x.double().abs() @ w.double().abs().T
    for nx, cl in [(0, 0)] + FORMS:
        y = torch.zeros((20, 140), device=DEV)
        product(x, w, y, 20, nx, cl)
        assert bool(((y.double() - want).abs() <= k * 2.0 ** -24 * size + k * 2.0 ** -149).all()), (nx, cl)
    ops.check_tc_status(x.device)


@pytest.mark.parametrize("n,k", [(4096, 2048), (12288, 2048), (2048, 6144)])
def test_more_blocks_than_multiprocessors(n, k):
    """Launches of several rounds of blocks, many of them one behind the other: a block of every form ends whatever order its warps end in."""
    rows = 700
    x, w = normal((rows, k), 7), normal((n, k), 8)
    want = torch.zeros((rows, n), device=DEV)
    product(x, w, want, rows, 16, 1)
    at = torch.randint(0, rows, (40,), generator=torch.Generator().manual_seed(9)).to(DEV)
    exact, size = x[at].double() @ w.double().T, x[at].double().abs() @ w.double().abs().T
    assert bool(((want[at].double() - exact).abs() <= BOUND(k) * size).all())
    for nx, cl in FORMS:
        y = torch.full((rows + 1, n), 3.0, device=DEV)
        for _ in range(20):
            product(x, w, y, rows, nx, cl)
        assert torch.equal(y[:rows], want) and bool((y[rows] == 3.0).all()), (nx, cl)
    y = torch.zeros((rows, n), device=DEV)
    for _ in range(1000):
        ops.gemm_f32_nt(x, w, y, rows)
    assert torch.equal(y, want)
    ops.check_tc_status(x.device)


def test_strided_batches():
    b, m, n, k = 3, 21, 150, 576
    a, w = normal((m, b, k), 3).transpose(0, 1), normal((b, n, k), 4)
    out = torch.zeros((m, b, n), device=DEV).transpose(0, 1)
    ops.batched_product(a, w, out)
    for i in range(b):
        y = torch.zeros((m, n), device=DEV)
        ops.gemm_f32_nt(a[i].contiguous(), w[i], y, m)
        assert torch.equal(out[i], y)
    ops.check_tc_status(a.device)


def test_values_without_a_split():
    """Infinities, NaN and results near the ends of the float32 range are what a chain of multiply-adds gives; rows beside them stay."""
    x, w = normal((20, 512), 5), normal((70, 512), 6)
    clean = torch.zeros((20, 70), device=DEV)
    ops.gemm_f32_nt(x, w, clean, 20)
    x[3, 7], x[4, 9], x[5] = float("inf"), float("nan"), 0.0
    x[6] *= 1e-38                                        # results of 1e-37, operands without room for a low half
    x[7, 0], w[:, 0] = torch.finfo(torch.float32).max, 0.25   # rounds to an infinite TF32 value
    w[11, 2] = -float("inf")
    y = torch.zeros((20, 70), device=DEV)
    ops.gemm_f32_nt(x, w, y, 20)
    exact = x.double() @ w.double().T
    assert torch.equal(y.isnan(), exact.isnan()) and torch.equal(y.isposinf(), exact.isposinf()) and torch.equal(y.isneginf(), exact.isneginf())
    keep = torch.arange(70, device=DEV) != 11
    assert not y[5][keep].any()
    size = x.double().abs() @ w.double().abs().T
    for r in (6, 7):
        assert bool(((y[r].double() - exact[r]).abs() <= 512 * 2.0 ** -24 * size[r] + 512 * 2.0 ** -150)[keep].all()), r
    y2 = torch.zeros((20, 70), device=DEV)
    w[:, 0], w[11, 2] = normal((70, 512), 6)[:, 0], normal((70, 512), 6)[11, 2]
    ops.gemm_f32_nt(x, w, y2, 20)
    assert torch.equal(y2[8:], clean[8:])
    ops.check_tc_status(x.device)
