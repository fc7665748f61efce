"""The float32 product on the tensor cores (operands split into two TF32 values): every form of it against float64 and against each
other, and the values that have no split."""
import pytest
import torch

from x0ne_engine_b200.csrc import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
FORMS = [(16, 1), (16, 2), (16, 4), (16, 8), (32, 1), (32, 4), (32, 8), (64, 1), (64, 4), (64, 8), (96, 1), (128, 1), (128, 8)]
# Of a sum of |x w|: 2^-23 for what the split leaves out of each product (two low halves cut off at 2^-12 times 2^-11, and their own
# product), 2^-22 for the tensor core cutting off 4 sums of a slab of 32 values, and 2^-24 for each float32 addition of a slab or a part.
BOUND = lambda k: 2.0 ** -23 + 2.0 ** -22 + (-(-k // 256) + 8) * 2.0 ** -24


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
    x[7, 0], w[:, 0] = 3.4e38, 0.25                       # rounds to an infinite TF32 value
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
