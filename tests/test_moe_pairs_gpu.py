"""The experts' products on pairs of blocks against float64, and their choice beside single blocks: experts without pairs, with a tile's edge
(128, 129, 256, 257 pairs) and with several tiles, widths that end inside a tile."""
import pytest
import torch

from x0ne_engine_b200.csrc import ops

DEV = "cuda:0"


@pytest.mark.gpu
@pytest.mark.parametrize("which,n,k", [(0, 200, 72), (0, 512, 256), (1, 136, 320), (1, 260, 64), (1, 514, 128), (2, 512, 200)])
def test_products_of_listed_pairs(which, n, k):
    counts = [0, 1, 128, 129, 256, 257, 600]
    experts, pairs = len(counts), sum(counts)
    g = torch.Generator().manual_seed(n + k)
    chosen = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)])[torch.randperm(pairs, generator=g)].view(pairs, 1)
    a, w = torch.randn(pairs, k, generator=g).bfloat16(), (torch.randn(experts, n, k, generator=g) / k ** 0.5).bfloat16()
    i32 = lambda *shape: torch.empty(shape, dtype=torch.int32, device=DEV)
    got, listed = {}, i32(pairs)               # (the order of an expert's pairs is the grouping's own)
    for pair in (False, True):
        tile = ops.MOE_TC_TILE_ROWS * (2 if pair else 1)
        n_tiles = ops.moe_max_tiles(pairs, experts, tile)
        offsets, tiles, n_real = i32(experts + 1), i32(n_tiles, 3), i32(1)
        ops.moe_group(chosen.to(DEV), pairs, experts, offsets, listed, tiles, tile, n_real)
        out = torch.full((pairs + 1, n // 2 if which == 2 else n), 3.0, dtype=torch.float32 if which == 1 else torch.bfloat16, device=DEV)
        ops.moe_product_tc(which, a.to(DEV), w.to(DEV), listed, tiles, n_real, n_tiles, out[:pairs], pair)
        ops.check_tc_status(torch.device(DEV))
        assert bool((out[pairs] == 3.0).all())
        got[pair] = out[listed.long()] if which == 1 else out[:pairs]          # (the down product writes by pair)
    assert torch.equal(got[True], got[False])            # by place, the same order of sums
    of = chosen[listed.cpu().long(), 0]                   # a place's expert; a's row p is place p's
    z = torch.empty(pairs, n, dtype=torch.float64)
    for e in range(experts):
        at = of == e
        z[at] = a[at].double() @ w[e].double().T
    if which == 0:
        want = torch.relu(z) ** 2
    elif which == 1:
        want = z
    else:
        blocks = z.view(pairs, -1, 2, ops.MOE_PAIR_BLOCK)
        want = (torch.nn.functional.silu(blocks[:, :, 0]) * blocks[:, :, 1]).reshape(pairs, n // 2)
    err = (got[True].double().cpu() - want).abs().max() / want.abs().max()
    assert err <= (2.0 ** -19 * k ** 0.5 if which == 1 else 2.0 ** -8)      # float32 sums of k products of unit size; one rounding to bfloat16


@pytest.mark.gpu
@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("which,n", [(0, 264), (1, 264), (2, 512)])
def test_results_that_do_not_start_on_16_bytes(which, n, pair):
    experts, pairs, k = 2, 150, 64
    g = torch.Generator().manual_seed(n)
    a, w = torch.randn(pairs, k, generator=g).bfloat16().to(DEV), torch.randn(experts, n, k, generator=g).bfloat16().to(DEV)
    tile = ops.MOE_TC_TILE_ROWS * (2 if pair else 1)
    i32 = lambda *shape: torch.empty(shape, dtype=torch.int32, device=DEV)
    n_tiles = ops.moe_max_tiles(pairs, experts, tile)
    offsets, listed, tiles, n_real = i32(experts + 1), i32(pairs), i32(n_tiles, 3), i32(1)
    ops.moe_group(torch.randint(0, experts, (pairs, 1), generator=g, dtype=torch.int32).to(DEV), pairs, experts, offsets, listed, tiles, tile, n_real)
    width, dtype = n // 2 if which == 2 else n, torch.float32 if which == 1 else torch.bfloat16
    got = []
    for first in (0, 1):
        out = torch.full((pairs * width + 8,), 3.0, dtype=dtype, device=DEV)
        ops.moe_product_tc(which, a, w, listed, tiles, n_real, n_tiles, out[first:first + pairs * width].view(pairs, width), pair)
        assert bool((out[:first] == 3.0).all()) and bool((out[first + pairs * width:] == 3.0).all())
        got.append(out[first:first + pairs * width].clone())
    ops.check_tc_status(torch.device(DEV))
    assert torch.equal(got[0], got[1])


def test_the_choice():
    take = lambda pairs, experts, ff=1024: ops.moe_tc_in_pairs(pairs, experts, 2 * ff, 2048, ff, 148)
    assert take(4096, 16) and take(16384, 16) and take(8192, 8, 1792)
    assert not take(8192, 16) and not take(4096, 32)
