"""The 32-bit attention kernel of passes with several rows per sequence: the plain kernel's bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# q heads, kv heads, keys, values, values out of the keys, window, chunk, what else
FORMS = [(16, 8, 128, None, 0, 0, 0, ""), (4, 4, 16, None, 0, 5, 0, "sink"), (6, 2, 20, 12, 0, 0, 37, ""), (20, 1, 48, 80, 0, 70, 0, "gate"), (6, 1, 144, 0, 128, 0, 0, "sink wide"),
         (3, 1, 64, 256, 0, 33, 0, "slope"), (5, 5, 72, 200, 0, 0, 64, "sig inside"), (32, 1, 320, 0, 256, 0, 0, "gate"), (8, 2, 32, None, 0, 40, 50, "slope sink")]


@pytest.mark.parametrize("H,G,dk,dv,vfk,window,chunk,what", FORMS)
def test_same_bits_as_the_plain_kernel(H, G, dk, dv, vfk, window, chunk, what):
    """Sequences of 1, 2, 31, 64 and 150 rows that start anywhere, a padding row of no sequence, pages that a sequence does not have."""
    from test_rovurax_gpu import scattered_cache
    from x0ne_engine_b200.csrc import ops
    storage, table, view = scattered_cache(G, dk, 0 if vfk else dv, 5, 5, seed=dk + H)
    table[3, 1] = -1
    s32 = storage.float()
    cache = ops.PagedCacheArg(s32.data_ptr(), table.data_ptr(), view.page_stride, view.table_stride, view.ring_pages, 64, G, dk, view.n_pages, view.v_dim)
    vd = vfk or (dk if dv is None else dv)
    seqs = [(0, 7, 1), (3, 100, 2), (1, 0, 31), (-1, 0, 1), (2, 33, 64), (4, 11, 150)]
    n_rows = sum(n for _, _, n in seqs)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    slots, pos = i32([s for s, _, n in seqs for _ in range(n)]), i32([p + r for _, p, n in seqs for r in range(n)])
    g = torch.Generator().manual_seed(5)
    inside = "inside" in what
    q_ld = H * dk + (8 if inside else 0)
    q = torch.randn(n_rows, q_ld, generator=g).to(DEV)
    kw = dict(chunk=chunk, v_from_k=vfk)
    if "sink" in what:
        kw["sink"] = torch.randn(H, generator=g).to(DEV)
    if "slope" in what:
        kw["slope"] = (torch.rand(H, generator=g) * 0.3).to(DEV)
    if "gate" in what or "wide" in what:
        kw.update(gate=torch.randn(n_rows, H * vd + 8, generator=g).to(DEV), gate_ld=H * vd + 8, gate_wide="wide" in what)
    if "sig" in what:
        kw["sig_bias"] = torch.randn(H, generator=g).to(DEV)
    if inside:
        kw.update(q_ld=q_ld, out_ld=H * vd + 6, out_col=3, out_scale=0.5)
    extra = ops.attn_extra(**kw)
    got = []
    for prompt in (False, True):
        out = torch.zeros((n_rows, H * vd + (6 if inside else 0)), device=DEV)
        ops.attention_rows(q, out, cache, slots, pos, n_rows, H, 0.3, window, extra, prompt=prompt)
        got.append(out)
    assert torch.isfinite(got[0]).all() and torch.equal(got[0], got[1])


@pytest.mark.parametrize("tile_rows", [16, 64, 128])
@pytest.mark.parametrize("H,G,dk,dv,window,chunk", [(16, 8, 128, None, 0, 0), (4, 4, 16, None, 5, 0), (6, 2, 20, 12, 0, 37), (3, 1, 64, 256, 33, 0), (20, 1, 48, 80, 70, 0)])
def test_same_bits_over_a_pass_table_of_tiles(H, G, dk, dv, window, chunk, tile_rows):
    """Single rows of many sequences beside longer ones, as a pass's tiles cut them (and as larger and smaller tiles would); rows of no tile are left alone."""
    from test_rovurax_gpu import scattered_cache
    from x0ne_engine_b200.csrc import ops
    lens, starts = [1, 1, 2, 150, 1, 64, 65, 1, 3, 129, 1], [70, 0, 63, 5, 255, 0, 64, 128, 31, 100, 299]
    storage, table, view = scattered_cache(G, dk, dv, len(lens), 5, seed=dk + H)
    s32 = storage.float()
    cache = ops.PagedCacheArg(s32.data_ptr(), table.data_ptr(), view.page_stride, view.table_stride, view.ring_pages, 64, G, dk, view.n_pages, view.v_dim)
    vd = dk if dv is None else dv
    first, tiles = [0], []
    for s, n in enumerate(lens):
        tiles += [(s, first[-1] + r) for r in range(0, n, tile_rows)]
        first.append(first[-1] + n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)      # noqa: E731
    n_rows = first[-1] + 2                                               # two padding rows behind the last sequence
    slots = i32(sum(([s] * n for s, n in enumerate(lens)), []) + [-1, -1])
    pos = i32(sum((list(range(p, p + n)) for p, n in zip(starts, lens)), []) + [0, 0])
    q = torch.randn(n_rows, H * dk, generator=torch.Generator().manual_seed(6)).to(DEV)
    extra = ops.attn_extra(chunk=chunk)
    plain, out = torch.zeros((n_rows, H * vd), device=DEV), torch.full((n_rows, H * vd), 3.0, device=DEV)
    ops.attention_rows(q, plain, cache, slots, pos, n_rows, H, 0.3, window, extra)
    ops.attention_rows(q, out, cache, slots, pos, n_rows, H, 0.3, window, extra, prompt=True,
                       tiles=(i32([t[0] for t in tiles]), i32([t[1] for t in tiles]), len(tiles), i32(first)))
    assert torch.isfinite(plain).all() and torch.equal(out[:-2], plain[:-2]) and bool((out[-2:] == 3.0).all())
