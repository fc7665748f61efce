"""The matrix-state scan by chunks against float64 token by token, at the places where a chunk (64 tokens) or a block (8) ends, and its
choice beside the walk."""
import types

import pytest
import torch

from x0ne_engine_b200.csrc import ops
from x0ne_engine_b200.parts.recurrent import by_chunks

DEV = "cuda:0"


def exact(r, k, v, w, u, S):
    """Outputs and final state of one sequence: r, k, v, w [T, H, 64], u [H, 64], S [H, 64, 64], all float64."""
    out = torch.empty_like(v)
    for t in range(r.shape[0]):
        kv = k[t][:, :, None] * v[t][:, None, :]
        out[t] = ((S + u[:, :, None] * kv) * r[t][:, :, None]).sum(1)
        S = S * w[t][:, :, None] + kv
    return out, S


@pytest.mark.gpu
@pytest.mark.parametrize("lens,heads,decay", [([1], 1, 1.0), ([8, 64], 2, 1.0), ([7, 9, 63, 65], 3, 0.1), ([128, 57, 200], 2, 4.0), ([515], 1, 0.01)])
def test_chunks_against_float64(lens, heads, decay):
    g = torch.Generator(device=DEV)
    g.manual_seed(11)
    rows, hn, width = sum(lens), heads * 64, heads * 64
    normal = lambda *s: torch.randn(*s, device=DEV, generator=g)
    r, k, v, h = (normal(rows, hn).bfloat16() for _ in range(4))
    z, w0, u = normal(rows, hn), torch.full((hn,), decay, device=DEV).log(), normal(hn)
    state = normal(len(lens) + 2, heads * 4096 + width)
    slots, first = list(range(len(lens), 0, -1)) + [-1], [0]
    for n in lens + [0]:
        first.append(first[-1] + n)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    before, o = state.clone(), torch.full((rows + 1, hn), 3.0, device=DEV)
    scratch = torch.full(((rows // 64 + len(lens) + 1) * heads * ops.WKV_CHUNK_UNIT,), float("nan"), device=DEV)
    run = lambda st, out, vv: ops.wkv_chunk_scan(r, k, vv, z, w0, u, h, out, st, i32(first), i32(slots), len(lens) + 1, rows, max(lens), heads, scratch)
    run(state, o, v)
    assert bool((o[rows] == 3.0).all())
    d = lambda x: x.double().view(rows, heads, 64)
    w = torch.exp(-torch.exp(d(z) + w0.double().view(heads, 64)))
    for s, n in enumerate(lens):
        a, b, slot = first[s], first[s] + n, slots[s]
        S = before[slot, :heads * 4096].double().view(heads, 64, 64)
        args = [x[a:b] for x in (d(r), d(k), d(v), w)]
        want, last = exact(*args, u.double().view(heads, 64), S)
        size, grown = exact(*[x.abs() for x in args], u.double().abs().view(heads, 64), S.abs())
        # of a term: its decays, at most n of two functions (2^-22 each and the argument's own rounding, which the exponent scales) and a
        # product each; sums of 16 in the tensor core and in float32 2^-20
        bound = 2.0 ** -20 + n * 2.0 ** -21 * (1 + 4 * decay)
        assert bool(((o[a:b].double().view(n, heads, 64) - want).abs() <= bound * size).all()), s
        assert bool(((state[slot, :heads * 4096].double().view(heads, 64, 64) - last).abs() <= bound * grown).all()), s
        assert torch.equal(state[slot, heads * 4096:], h[b - 1].float())
    untouched = [x for x in range(len(lens) + 2) if x not in slots]
    assert torch.equal(state[untouched], before[untouched])
    again, o2 = before.clone(), torch.zeros_like(o)
    run(again, o2, v)
    assert torch.equal(o2[:rows], o[:rows]) and torch.equal(again, state)
    # a value that is not finite reaches no earlier token
    bad, o3 = v.clone(), torch.zeros_like(o)
    at = first[len(lens) - 1] + lens[-1] // 2
    bad[at] = float("inf")
    run(before.clone(), o3, bad)
    assert torch.isfinite(o3[:at]).all() and (torch.equal(o3[:max(0, at - 64)], o[:max(0, at - 64)]))


@pytest.mark.gpu
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["r", "k", "v", "z", "state"])
def test_values_that_are_not_finite_reach_what_they_reach_token_by_token(where, value):
    """One value in the middle of the second of four chunks (or in the state the sequence starts from)."""
    g = torch.Generator(device=DEV)
    g.manual_seed(17)
    rows, heads, width = 230, 2, 128
    normal = lambda *s: torch.randn(*s, device=DEV, generator=g)
    rkv = {s: normal(rows, 128).bfloat16() for s in "rkv"}
    h, z, w0, u = normal(rows, width).bfloat16(), normal(rows, 128) * 0.1, torch.full((128,), 0.01, device=DEV).log(), normal(128)
    state = normal(1, heads * 4096 + width)
    if where == "state":
        state[0, 64 * 5 + 7] = value
    elif where == "z":
        z[100, 70] = value
    else:
        rkv[where][100, 70] = value
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    scratch = torch.empty(((rows // 64 + 1) * heads * ops.WKV_CHUNK_UNIT,), device=DEV)
    got = []
    for chunks in (False, True):
        st, o = state.clone(), torch.zeros(rows, 128, device=DEV)
        args = (rkv["r"], rkv["k"], rkv["v"], z, w0, u, h, o, st, i32([0, rows]), i32([0]), 1)
        if chunks:
            ops.wkv_chunk_scan(*args, rows, rows, heads, scratch)
        else:
            ops.wkv_scan(*args, heads, 64)
        got.append((o, st))
    (o1, s1), (o2, s2) = got
    assert not bool(torch.isfinite(o1).all()) or where == "z"           # (a decay of zero is finite)
    assert torch.equal(torch.isfinite(o1), torch.isfinite(o2)) and torch.equal(torch.isfinite(s1), torch.isfinite(s2))
    if value != value:
        assert torch.equal(o1.isnan(), o2.isnan()) and torch.equal(s1.isnan(), s2.isnan())
    fine = torch.isfinite(o1)
    assert float((o1 - o2)[fine].abs().max()) <= 1e-4 * float(o1[fine].abs().max())     # (two orders of float32 sums of a few hundred terms)


def test_the_choice():
    def ctx(n_seqs, longest, decode=False):
        return types.SimpleNamespace(decode=decode, n_seqs=n_seqs, max_seq_rows=longest, sm_count=148)
    state = torch.zeros(2, 4 * 100)
    take = lambda c, heads, rows, dtype=torch.bfloat16, dim=64, st=state: by_chunks(c, dtype, heads, dim, rows, st)
    assert take(ctx(1, 2048), 32, 2048) and take(ctx(16, 128), 32, 2048) and take(ctx(1, 512), 16, 512)
    assert not take(ctx(1, 256), 32, 256) and not take(ctx(1, 64), 64, 64) and not take(ctx(64, 40), 32, 2048)
    assert not take(ctx(1, 2048), 32, 2048, torch.float32) and not take(ctx(1, 2048), 32, 2048, dim=32) and not take(ctx(1, 2048, True), 32, 2048)
    assert not take(ctx(1, 2048), 32, 2048, st=torch.zeros(2, 4 * 100 + 2))
