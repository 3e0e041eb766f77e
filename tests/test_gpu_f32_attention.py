"""float32 attention: rows in tiles of 64 and rows one by one give the same bits, and both hold to 64 bits."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rows,prior,H,G,hd,vd,window,cap,gated,sink,page", [
    ([9], [0], 4, 4, 128, 128, 0, 0.0, False, None, 16),                      # the fewest rows a tile takes
    ([64, 63, 1], [0, 64, 63], 4, 4, 128, 128, 64, 0.0, True, 1.5, 16),       # a whole tile, one short, a row by itself; window = a chunk
    ([130, 9, 8, 70], [0, 5, 200, 33], 6, 2, 64, 64, 0, 0.0, False, None, 16),
    ([130, 9, 70, 3], [50, 5, 33, 100], 6, 2, 128, 64, 40, 30.0, True, None, 16),
    ([65, 200], [7, 90], 4, 1, 24, 100, 33, 0.0, False, 0.0, 4),
    ([12], [600], 2, 1, 4, 128, 0, 0.0, False, None, 16),
    ([640, 9, 65], [0, 700, 10], 32, 4, 128, 128, 0, 0.0, False, None, 16),
    ([640, 9, 65], [0, 700, 10], 32, 4, 96, 96, 0, 0.0, False, None, 16),        # tiles of 64 rows (so the next; the others: of 32)
    ([600, 12], [3, 0], 32, 32, 60, 64, 50, 20.0, True, 0.5, 16)])
def test_tiles_and_rows_agree(rows, prior, H, G, hd, vd, window, cap, gated, sink, page):
    from cajeta_llm_b200.csrc import kernels as K
    g = torch.Generator().manual_seed(7)
    total = [a + b for a, b in zip(rows, prior)]
    width = max(-(-t // page) for t in total)
    pages = sum(-(-t // page) for t in total) + 1
    perm, at = torch.randperm(pages - 1, generator=g) + 1, 0
    table = torch.full((len(rows), width), -1, dtype=torch.int32)
    for r, t in enumerate(total):
        n = -(-t // page)
        table[r, :n] = perm[at:at + n].int()
        at += n
    kp, vp = (torch.randn(pages, G, page, d, generator=g).to(DEV) for d in (hd, vd))
    T = sum(rows)
    q = torch.randn(T, H, hd, generator=g).to(DEV)
    gate = torch.randn(T, H + 3, generator=g).to(DEV) if gated else None
    starts = [sum(rows[:i]) for i in range(len(rows) + 1)]
    pos = torch.cat([torch.arange(p, p + n) for n, p in zip(rows, prior)]).int().to(DEV)
    req = torch.cat([torch.full((n,), i) for i, n in enumerate(rows)]).int().to(DEV)
    table, start = table.to(DEV), torch.tensor(starts, dtype=torch.int32, device=DEV)
    scale = hd ** -0.5
    kw = dict(value_dim=vd, softcap=cap, head_gate=gate, gate_offset=3 if gated else 0, sink=K.NO_SINK if sink is None else sink)
    tiled, single = torch.empty(T, H, vd, device=DEV), torch.empty(T, H, vd, device=DEV)
    K.paged_attention(q, tiled, kp, vp, pos, req, table, page, H, G, hd, window, scale, req_start=start, h_req_start=starts, **kw)
    K.paged_attention(q, single, kp, vp, pos, req, table, page, H, G, hd, window, scale, **kw)
    assert torch.equal(tiled, single)
    for r, (n, p0) in enumerate(zip(rows, prior)):
        held = table[r].long()[:-(-total[r] // page)]
        k, v = (t[held].permute(1, 0, 2, 3).reshape(G, -1, t.shape[-1])[:, :total[r]].double() for t in (kp, vp))
        i, j = torch.arange(p0, p0 + n, device=DEV)[:, None], torch.arange(total[r], device=DEV)[None]
        seen = (j <= i) & ((j > i - window) if window else torch.ones_like(j, dtype=torch.bool))
        for h in range(H):
            s = q[starts[r]:starts[r + 1], h].double() @ k[h * G // H].t() * scale
            s = (cap * torch.tanh(s / cap) if cap else s).masked_fill(~seen, -math.inf)
            if sink is not None:
                s = torch.cat([s, torch.full((n, 1), sink, dtype=torch.float64, device=DEV)], 1)
            o = torch.softmax(s, 1)[:, :total[r]] @ v[h * G // H]
            if gated:
                o = o * torch.sigmoid(gate[starts[r]:starts[r + 1], 3 + h].double())[:, None]
            assert torch.allclose(single[starts[r]:starts[r + 1], h].double(), o, atol=2e-5, rtol=1e-4)


def test_a_later_rows_infinite_value_stays_with_the_rows_that_see_it():
    from cajeta_llm_b200.csrc import kernels as K
    T, H, hd = 40, 2, 64
    g = torch.Generator().manual_seed(8)
    kp, vp = (torch.randn(4, H, 16, hd, generator=g).to(DEV) for _ in range(2))
    vp[1, :, 15] = float("inf")                                               # position 31
    q, out = torch.randn(T, H, hd, generator=g).to(DEV), torch.empty(T, H, hd, device=DEV)
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    K.paged_attention(q, out, kp, vp, pos, torch.zeros_like(pos), torch.arange(4, dtype=torch.int32, device=DEV)[None], 16, H, H, hd, 0, 0.125,
                      req_start=torch.tensor([0, T], dtype=torch.int32, device=DEV), h_req_start=[0, T])
    assert bool(torch.isfinite(out[:31]).all()) and not bool(torch.isfinite(out[31:]).any())


def test_rows_by_request_have_to_cover_the_rows():
    """A list that shares out other rows than the step's is refused; an empty one is none at all."""
    from cajeta_llm_b200.csrc import kernels as K
    T, H, hd = 20, 2, 64
    g = torch.Generator().manual_seed(9)
    kp, vp = (torch.randn(2, H, 16, hd, generator=g).to(DEV) for _ in range(2))
    q = torch.randn(T, H, hd, generator=g).to(DEV)
    pos = torch.arange(T, dtype=torch.int32, device=DEV)

    def run(**kw):
        out = torch.full((T, H, hd), 7.0, device=DEV)
        K.paged_attention(q, out, kp, vp, pos, torch.zeros_like(pos), torch.arange(2, dtype=torch.int32, device=DEV)[None], 16, H, H, hd, 0, 0.125, **kw)
        return out

    start = torch.tensor([0, T], dtype=torch.int32, device=DEV)
    plain = run()
    assert torch.equal(run(req_start=start, h_req_start=[]), plain) and torch.equal(run(req_start=start, h_req_start=[0, T]), plain)
    for wrong in ([0], [0, T - 1], [0, T + 1], [1, T], [0, 12, 11, T], [0, 5, T]):
        with pytest.raises(K.KernelError):
            run(req_start=start, h_req_start=wrong)


@pytest.mark.parametrize("tiled", [False, True])
def test_keys_whose_scores_are_minus_infinity_have_no_weight(tiled):
    """Whole chunks of such keys at a row's end, in its middle and at its beginning (the first score of all finite or not)."""
    from cajeta_llm_b200.csrc import kernels as K
    T, prior, H, hd = 9, 320, 2, 64
    n = T + prior
    g = torch.Generator().manual_seed(10)
    kp, vp = (torch.randn(21, H, 16, hd, generator=g).to(DEV) for _ in range(2))
    q = torch.randn(T, H, hd, generator=g).to(DEV)
    q[..., 0] = 1.0
    q[4:, :, 0] = 0.0                                                         # (0 x -inf is no number: the other rows' keys are finite)
    kp[..., 0] = kp[..., 0].abs()
    keys = kp.permute(1, 0, 2, 3).reshape(H, -1, hd)
    dead = torch.zeros(keys.shape[1], dtype=torch.bool)
    dead[:64], dead[128:192], dead[320:] = True, True, True
    big = torch.zeros(hd, device=DEV)
    big[0] = -3e38
    keys[:, dead.to(DEV)] = big
    kp = keys.reshape(H, 21, 16, hd).permute(1, 0, 2, 3).contiguous()
    pos = torch.arange(prior, n, dtype=torch.int32, device=DEV)
    out = torch.empty(T, H, hd, device=DEV)
    more = dict(req_start=torch.tensor([0, T], dtype=torch.int32, device=DEV), h_req_start=[0, T]) if tiled else {}
    K.paged_attention(q, out, kp, vp, pos, torch.zeros_like(pos), torch.arange(21, dtype=torch.int32, device=DEV)[None], 16, H, H, hd, 0, 2.0, **more)
    values = vp.permute(1, 0, 2, 3).reshape(H, -1, hd).double()
    for h in range(H):
        s = (q[:4, h] @ kp.permute(1, 0, 2, 3).reshape(H, -1, hd)[h].t() * 2.0).double()
        s = s.masked_fill(torch.arange(336, device=DEV)[None] > pos[:4, None], -math.inf)
        assert bool(torch.isinf(s[:, :64]).all())
        assert torch.allclose(out[:4, h].double(), torch.softmax(s, 1) @ values[h], atol=2e-5, rtol=1e-4)


@pytest.mark.parametrize("rows,heads,hd,vd", [(37, 4, 128, 128), (70, 4, 128, 96), (130, 4, 100, 128), (180, 4, 128, 128), (300, 4, 64, 64), (260, 8, 64, 128)])
@pytest.mark.parametrize("window", [0, 41])
def test_rows_in_pieces_of_any_size(monkeypatch, rows, heads, hd, vd, window):
    """One row a request, as many blocks as go with chunks whole and in pieces of 32, 24 and 16 keys; keys that end at pieces' and chunks' edges."""
    from cajeta_llm_b200.csrc import kernels as K
    g, page = torch.Generator().manual_seed(13), 16
    ends = [(0, 1, 15, 16, 17, 23, 24, 25, 31, 32, 47, 48, 49, 63, 64, 65, 87, 88, 111, 112, 130, 191, 192, 300, 450)[i % 25] for i in range(rows)]
    pages = [e // page + 1 for e in ends]
    kp, vp = (torch.randn(sum(pages), heads, page, d, generator=g).to(DEV) for d in (hd, vd))
    table, at = torch.full((rows, max(pages)), -1, dtype=torch.int32), 0
    for r, n in enumerate(pages):
        table[r, :n] = torch.arange(at, at + n)
        at += n
    q, pos, req = torch.randn(rows, heads, hd, generator=g).to(DEV), torch.tensor(ends).int().to(DEV), torch.arange(rows).int().to(DEV)
    starts, outs = list(range(rows + 1)), []
    for few in (K.F32_FEW_ROWS, 0):
        monkeypatch.setattr(K, "F32_FEW_ROWS", few)
        out = torch.full((rows, heads, vd), math.nan, device=DEV)
        K.paged_attention(q, out, kp, vp, pos, req, table.to(DEV), page, heads, heads, hd, window, hd ** -0.5, value_dim=vd,
                          req_start=torch.tensor(starts, dtype=torch.int32, device=DEV), h_req_start=starts)
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
