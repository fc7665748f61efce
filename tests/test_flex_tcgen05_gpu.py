"""The general prefill attention on tcgen05 beside the mma.sync kernel and the plain kernel, over the forms it takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# keys, values, values out of the keys, window, chunk, kept first keys, what else
FORMS = [
    (128, 128, 0, 0, 0, 0, ""), (64, 64, 0, 70, 0, 0, "sink"), (8, 8, 0, 0, 0, 0, "slope"), (96, 40, 0, 0, 100, 0, "gate"),
    (128, 256, 0, 150, 0, 67, "wide f32"), (72, 200, 0, 0, 64, 0, "sink f32 inside"), (320, 0, 256, 90, 0, 0, "sink gate"), (160, 0, 128, 0, 0, 3, "wide"),
    (128, 64, 0, 0, 130, 0, "sig inside"), (64, 136, 0, 0, 0, 0, "slope late"), (128, 128, 0, 0, 0, 0, "late inside"), (24, 16, 0, 1, 0, 0, "sig"),
    (128, 128, 0, 0, 0, 0, "gone"), (64, 64, 0, 70, 0, 67, "gone sink"), (320, 0, 256, 0, 0, 0, "gone gate"), (128, 64, 0, 0, 130, 0, "gone sig"),
]


@pytest.mark.parametrize("dk,dv,vfk,window,chunk,keep,what", FORMS)
def test_both_kernels_give_the_plain_kernels_results(dk, dv, vfk, window, chunk, keep, what, monkeypatch):
    """Sequences of 1, 127, 128, 129 and 300 rows that start inside and at the start of pages, scattered pages, and rows of the last
    page past a sequence's end that hold NaN.  `late`: keys that grow along the sequence, so that accumulators are rescaled.
    `gone`: pages that the table does not name or names past the last one, and a page number 0 that is nobody's and holds NaN."""
    from test_rovurax_gpu import plain_kernel_in_float32, scattered_cache
    from x0ne_engine_b200.csrc import ops
    G, H, pages = (1 if vfk else 2), 6, 8
    vd = vfk or dv
    storage, table, view = scattered_cache(G, dk, 0 if vfk else (None if dv == dk else dv), 5, pages, seed=dk + vd)
    view_args = (view.page_stride, view.table_stride, view.ring_pages, 64, G, dk, view.n_pages, view.v_dim)
    seqs = [(3, 0, 1), (0, 65, 127), (1, 128, 128), (4, 37, 129), (2, 0, 300)]
    pool = storage.view(-1, view.page_stride)
    keys = lambda page: page[:G * 64 * dk].view(G, 64, dk)
    for slot, p0, n in seqs:
        for lp in range(pages):
            page = pool[int(table[slot, lp])]
            if "late" in what:
                keys(page).mul_(0.2 + 1.5 * lp)
            past = p0 + n - lp * 64
            if past < 64:
                keys(page)[:, max(past, 0):] = float("nan")
                if not vfk:
                    page[G * 64 * dk:G * 64 * (dk + vd)].view(G, 64, vd)[:, max(past, 0):] = float("nan")
    if "gone" in what:
        own = torch.nonzero(table == 0)
        if len(own):
            spare = next(p for p in range(view.n_pages) if not bool((table == p).any()))
            pool[spare] = pool[0]
            table[own[0, 0], own[0, 1]] = spare
        pool[0] = float("nan")
        table[0, 0], table[2, 1], table[4, 0] = -1, view.n_pages + 3, -1          # (slot 4's first rows see no key at all)
    g = torch.Generator().manual_seed(3)
    n_rows = sum(n for _, _, n in seqs)
    inside = "inside" in what
    q_ld = H * dk + (24 if inside else 0)
    q = torch.randn(n_rows, q_ld, generator=g).bfloat16().to(DEV)
    kw = dict(keep_first=keep, chunk=chunk)
    if vfk:
        kw["v_from_k"] = vfk
    if "sink" in what:
        kw["sink"] = torch.randn(H, generator=g).to(DEV)
    if "slope" in what:
        kw["slope"] = (torch.rand(H, generator=g) * 0.3).to(DEV)
    if "gate" in what or "wide" in what:
        wide = "wide" in what
        kw["gate"], kw["gate_ld"], kw["gate_wide"] = torch.randn(n_rows, H * vd + 8, generator=g).bfloat16().to(DEV), H * vd + 8, wide
    if "sig" in what:
        kw["sig_bias"] = torch.randn(H, generator=g).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    first, tiles = [0], []
    for k, (_, _, n) in enumerate(seqs):
        tiles += [(k, first[-1] + r0) for r0 in range(0, n, 128)]
        first.append(first[-1] + n)
    slots, pos = i32([s for s, _, n in seqs for _ in range(n)]), i32([p + r for _, p, n in seqs for r in range(n)])
    scale = 1.3 * dk ** -0.5
    clean = storage.clone()
    torch.nan_to_num_(clean, nan=0.0)
    want, _ = plain_kernel_in_float32(q[:, :H * dk].contiguous(), view_args, clean, table, slots, pos, H, scale, window,
                                      {k: (v.float() if k == "gate" else v) for k, v in kw.items()}, vd)
    if inside:
        kw.update(q_ld=q_ld, out_ld=H * vd + 16, out_col=8, out_scale=0.5)
        want = want * 0.5
    extra = ops.attn_extra(out_f32="f32" in what, **kw)
    assert ops.attention_flex_tc_takes(q, view, H, scale, extra)
    got = []
    for tensor_memory in (True, False):
        if not tensor_memory:
            monkeypatch.setattr(ops, "attention_flex_tc_takes", lambda *a: False)
        out = torch.zeros((n_rows, H * vd + (16 if inside else 0)), dtype=torch.float32 if "f32" in what else torch.bfloat16, device=DEV)
        ops.attention_flex_prefill(q, out, view, i32([t[0] for t in tiles]), i32([t[1] for t in tiles]), len(tiles), i32(first), i32([s for s, _, _ in seqs]),
                                   i32([p for _, p, _ in seqs]), H, scale, window, extra)
        assert int(ops.gemm_tc_status(out.device)[0]) == 0
        if inside:
            assert bool((out[:, :8] == 0).all()) and bool((out[:, 8 + H * vd:] == 0).all())
            out = out[:, 8:8 + H * vd]
        got.append(out.float())
        # weights carry 16 bits, sums are float32: what is left is the result's rounding (2^-9 of a value; 2^-14 without it)
        bound = (2 ** -13 if "f32" in what else 2 ** -8) * want.abs().max().item()
        assert (got[-1] - want).abs().max().item() <= bound, "tcgen05" if tensor_memory else "mma.sync"


def test_rows_that_cannot_be_copied_16_bytes_at_a_time_take_the_other_kernel():
    from test_rovurax_gpu import scattered_cache
    from x0ne_engine_b200.csrc import ops
    q = torch.zeros(4, 2 * 64 + 4, dtype=torch.bfloat16, device=DEV)
    _, _, view = scattered_cache(1, 64, None, 1, 2, seed=1)
    assert ops.attention_flex_tc_takes(q[:, :128].contiguous(), view, 2, 0.1, ops.attn_extra())
    assert not ops.attention_flex_tc_takes(q, view, 2, 0.1, ops.attn_extra(q_ld=132))
    assert not ops.attention_flex_tc_takes(q[:, :128].contiguous(), view, 2, 0.0, ops.attn_extra())
    _, _, odd = scattered_cache(1, 60, None, 1, 2, seed=1)
    assert not ops.attention_flex_tc_takes(torch.zeros(4, 120, dtype=torch.bfloat16, device=DEV), odd, 2, 0.1, ops.attn_extra())
