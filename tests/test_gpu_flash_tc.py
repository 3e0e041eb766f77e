"""Differential and latent attention of prompt portions on tcgen05: against the formula in 64 bits, at the edges of tiles of 128 rows and
keys, of halves of 64 and of windows.  What is no key of a row is NaN in memory where another request, or nobody, owns it.

Tolerance: what leaves is bfloat16 (2^-9 of itself) of a weighted mean of bfloat16 values; with weights rounded to bfloat16 the mean is
off by at most 2^-9 of the largest value besides.  The differential form's weights keep 16 bits, but its norm divides by the size of a
difference: its bound is the tiled form's own, 0.02."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
NAN = float("nan")


def _visible(p, r, n, window):
    """[rows, n]: whether a row of a request (p tokens before its r rows) sees key k."""
    pos, key = torch.arange(p, p + r)[:, None], torch.arange(n)[None]
    return (key <= pos) & ((key > pos - window) if window else True)


def _attend(q, k, v, see, scale, sink=None):
    """q [r, d], k [n, d], v [n, e] in 64 bits."""
    s = (q @ k.T * scale).masked_fill(~see, float("-inf"))
    m = s.amax(1, keepdim=True)
    e = torch.exp(s - m)
    return (e @ v) / (e.sum(1, keepdim=True) + (torch.exp(sink - m) if sink is not None else 0.0))


@pytest.mark.parametrize("H,G,hd,vd,page,window,requests", [
    (2, 1, 64, 128, 16, 0, [(0, 128), (0, 129), (0, 1), (65, 127)]),
    (4, 2, 64, 64, 32, 0, [(255, 1), (256, 130), (0, 300), (63, 65)]),
    (2, 2, 128, 128, 16, 100, [(0, 260), (500, 40), (99, 1), (100, 2)]),
    (3, 1, 128, 64, 48, 1, [(0, 140), (127, 3)]),
    (16, 8, 64, 128, 16, 0, [(0, 700)]),
])
def test_differential(H, G, hd, vd, page, window, requests):
    from cajeta_llm_b200.csrc import kernels as K
    g = torch.Generator().manual_seed(H + hd + vd)
    totals = [p + r for p, r in requests]
    need = [-(-t // page) for t in totals]
    order = torch.randperm(sum(need) + 2, generator=g).int()
    table = torch.full((len(requests), max(need) + 1), -1, dtype=torch.int32)
    kp, vp = (torch.full((sum(need) + 2, G, page, w), NAN, dtype=torch.bfloat16) for w in (2 * hd, vd))
    keys, values, at = [], [], 0
    for i, n in enumerate(need):
        table[i, :n] = order[at:at + n]
        at += n
        k, v = (torch.randn((totals[i], G, w), generator=g).bfloat16() for w in (2 * hd, vd))
        k[::5] *= 2.0
        for t in range(totals[i]):
            kp[int(table[i, t // page]), :, t % page], vp[int(table[i, t // page]), :, t % page] = k[t], v[t]
        keys.append(k.double()), values.append(v.double())
        gone = max(0, requests[i][0] + 1 - window) // page if window else 0      # pages behind the window have been given back
        table[i, :gone] = -1
    T = sum(r for _, r in requests)
    q = torch.randn((T, H, 2 * hd), generator=g).bfloat16()
    scale, lam, eps, out_scale = hd ** -0.5, 0.55, 1e-5, 0.4
    want, row = torch.zeros((T, H, vd), dtype=torch.float64), 0
    starts = [0]
    for i, (p, r) in enumerate(requests):
        see = _visible(p, r, totals[i], window)
        for h in range(H):
            a = [_attend(q[row:row + r, h, m * hd:(m + 1) * hd].double(), keys[i][:, h * G // H, m * hd:(m + 1) * hd], values[i][:, h * G // H],
                         see, scale) for m in range(2)]
            o = a[0] - lam * a[1]
            want[row:row + r, h] = o / torch.sqrt((o * o).mean(1, keepdim=True) + eps) * out_scale
        row += r
        starts.append(row)
    out = torch.full((T, H, vd), NAN, dtype=torch.bfloat16, device=DEV)
    K.diff_attention_tc(q.to(DEV), out, kp.to(DEV), vp.to(DEV), torch.tensor(starts, dtype=torch.int32, device=DEV),
                        torch.tensor([p for p, _ in requests], dtype=torch.int32, device=DEV), len(requests), table.to(DEV), page, H, G, hd, vd,
                        window, scale, lam, eps, out_scale)
    err = (out.cpu().double() - want).abs()
    assert float(err.max()) < 0.02 * max(1.0, float(want.abs().max())), float(err.max())
    assert float((err / want.abs().clamp_min(want.pow(2).mean().sqrt())).mean()) < 2.0 ** -8
    assert not K.wait_errors()


@pytest.mark.parametrize("requests,tcgen05", [([(0, 128), (40, 127)], False), ([(0, 128), (40, 128)], True), ([(0, 8)] * 33, False), ([(300, 8)] * 33, True)])
def test_the_forms_of_differential_attention_agree(monkeypatch, requests, tcgen05):
    """What the entry takes on both sides of its lines, against the tiles of 64 rows."""
    from cajeta_llm_b200.csrc import kernels as K
    g, H, G, hd, vd, page = torch.Generator().manual_seed(5), 8, 4, 64, 128, 16
    T, totals, taken = sum(r for _, r in requests), [p + r for p, r in requests], []
    real = K.diff_attention_tc
    monkeypatch.setattr(K, "diff_attention_tc", lambda *a: (taken.append(1), real(*a)))
    need = [-(-t // page) for t in totals]
    kp, vp = (torch.randn((sum(need), G, page, w), generator=g).bfloat16().to(DEV) for w in (2 * hd, vd))
    table, at = torch.full((len(requests), max(need)), -1, dtype=torch.int32), 0
    for i, n in enumerate(need):
        table[i, :n] = torch.arange(at, at + n)
        at += n
    q, starts = torch.randn((T, H, 2 * hd), generator=g).bfloat16().to(DEV), [sum(r for _, r in requests[:i]) for i in range(len(requests) + 1)]
    i32 = [torch.tensor(x, dtype=torch.int32, device=DEV) for x in (
        [p + j for p, r in requests for j in range(r)], [i for i, (_, r) in enumerate(requests) for _ in range(r)], starts, [p for p, _ in requests])]
    outs = []
    for kw in (dict(h_rows=[r for _, r in requests], h_prior=[p for p, _ in requests]), dict(splits=1)):
        out = torch.full((T, H, vd), NAN, dtype=torch.bfloat16, device=DEV)
        K.diff_attention(q, out, kp, vp, i32[0], i32[1], table.to(DEV), page, H, G, hd, vd, 0, hd ** -0.5, 0.55, 1e-5, 0.4, i32[2], i32[3], len(requests),
                         table.shape[1] * page, **kw)
        outs.append(out.double())
    assert bool(taken) == tcgen05
    assert float((outs[0] - outs[1]).abs().max()) < 2 * 0.02 * max(1.0, float(outs[1].abs().max()))        # (each within 0.02 of the formula)
    assert not K.wait_errors()


@pytest.mark.parametrize("H,dim,rot,vdim,window,sink,gate,requests", [
    (2, 128, 64, 128, 0, True, "none", [(0, 256), (0, 257), (0, 1), (65, 127)]),
    (2, 128, 64, 128, 0, False, "head", [(100, 300), (0, 640)]),
    (3, 128, 40, 64, 64, False, "entry", [(0, 130), (500, 70), (63, 66), (64, 1)]),
    (2, 64, 64, 128, 200, True, "entry", [(0, 420), (7, 2), (1000, 3)]),
    (2, 64, 32, 64, 1, False, "none", [(0, 200), (200, 65)]),
    (16, 128, 64, 128, 1024, False, "entry", [(0, 1500)]),
])
def test_latent(H, dim, rot, vdim, window, sink, gate, requests):
    from cajeta_llm_b200.csrc import kernels as K
    g = torch.Generator().manual_seed(H + dim + rot + vdim)
    T, gap = sum(r for _, r in requests), 5                                       # tokens between requests that nobody owns
    q = torch.zeros((T, H, dim + 64))
    q[..., :dim + rot] = torch.randn((T, H, dim + rot), generator=g)
    q = q.bfloat16()
    starts, base, n = [0], [], 0
    for p, r in requests:
        first = max(0, p + 1 - window) if window else 0
        base.append(n - first)
        n += p + r - first + gap
        starts.append(starts[-1] + r)
    kp, kr, vp = torch.full((n, H * dim), NAN), torch.full((n, 64), NAN), torch.full((n, H * vdim), NAN)
    for (p, r), b in zip(requests, base):
        lo, hi = b + (max(0, p + 1 - window) if window else 0), b + p + r
        kp[lo:hi], vp[lo:hi] = torch.randn((hi - lo, H * dim), generator=g), torch.randn((hi - lo, H * vdim), generator=g)
        kr[lo:hi, :rot], kr[lo:hi, rot:] = torch.randn((hi - lo, rot), generator=g), 0.0
    kp, kr, vp = kp.bfloat16(), kr.bfloat16(), vp.bfloat16()
    sinks = torch.randn(H, generator=g) if sink else None
    gates = torch.randn((T, 4 + (H * vdim if gate == "entry" else H)), generator=g)
    scale, want = 1.5 * (dim + rot) ** -0.5, torch.zeros((T, H, vdim), dtype=torch.float64)
    for i, (p, r) in enumerate(requests):
        first = max(0, p + 1 - window) if window else 0
        rows, toks = slice(starts[i], starts[i + 1]), slice(base[i] + first, base[i] + p + r)
        see = _visible(p, r, p + r, window)[:, first:]
        for h in range(H):
            k = torch.cat([kp[toks, h * dim:(h + 1) * dim], kr[toks]], 1).double()
            o = _attend(q[rows, h].double(), k, vp[toks, h * vdim:(h + 1) * vdim].double(), see, scale, sinks[h].double() if sink else None)
            if gate != "none":
                z = gates[rows, 3 if gate == "head" else 4:].double()
                o = o * torch.sigmoid(z[:, h * vdim:(h + 1) * vdim] if gate == "entry" else z[:, h:h + 1])
            want[rows, h] = o
    errs = []
    for exact in (False, True):
        out = torch.full((T, H * vdim), NAN, dtype=torch.bfloat16, device=DEV)
        # (a gate from the fourth column on lies on 16 bytes: eight entries a thread)
        K.latent_attention_tc(q.to(DEV), out, kp.to(DEV), kr.to(DEV), vp.to(DEV), torch.tensor(starts, dtype=torch.int32, device=DEV),
                              torch.tensor([p for p, _ in requests], dtype=torch.int32, device=DEV),
                              torch.tensor(base, dtype=torch.int32, device=DEV), len(requests), H, dim, vdim, scale,
                              sink=sinks.to(DEV) if sink else None, window=window, exact_weights=exact,
                              gate=gates.to(DEV) if gate == "head" else None, gate_offset=3)
        if gate == "entry":
            K.latent_gate_rows(out.view(T, H, vdim), gates.to(DEV), 4, H, vdim, out, by_entry=True)
        err = (out.cpu().double().view(T, H, vdim) - want).abs()
        assert float(err.max()) < 2.0 ** -8 * 5.0, float(err.max())                # values of at most about five
        errs.append(float(err.pow(2).mean().sqrt()))
    assert errs[1] <= errs[0] * 1.001
    assert not K.wait_errors()


@pytest.mark.parametrize("dim,rot,rotary,halves", [(128, 64, 64, False), (128, 64, 64, True), (64, 40, 16, True), (64, 24, 24, False), (60, 20, 12, True)])
def test_latent_queries_and_gather(dim, rot, rotary, halves):
    """Queries eight entries a thread and one a thread, the latent and the rotated key part sixteen bytes and one entry a thread."""
    from cajeta_llm_b200.csrc import kernels as K
    g = torch.Generator().manual_seed(dim + rot)
    T, H, DK, rank, page = 7, 3, 256, 48 if dim != 60 else 50, 16
    q, pos = torch.randn((T, H * (dim + rot) + 4), generator=g), torch.randint(0, 3000, (T,), generator=g).int()
    f = (10000.0 ** (-torch.arange(rotary // 2) / (rotary / 2.0))).float()
    qx = torch.full((T, H, DK), NAN, dtype=torch.bfloat16, device=DEV)
    K.latent_q_pack(q.to(DEV), H, dim, rot, rotary, f.to(DEV), pos.to(DEV), qx, halves=halves, magnitude=1.1)
    want = torch.zeros((T, H, DK), dtype=torch.float64)
    want[..., :dim + rot] = q[:, :H * (dim + rot)].view(T, H, dim + rot).double()
    a = (pos.float()[:, None] * f).double()[:, None]
    x = want[..., dim:dim + rotary].clone()
    u, w = (x[..., :rotary // 2], x[..., rotary // 2:]) if halves else (x[..., 0::2], x[..., 1::2])
    y = [1.1 * (u * torch.cos(a) - w * torch.sin(a)), 1.1 * (w * torch.cos(a) + u * torch.sin(a))]
    want[..., dim:dim + rotary] = torch.cat(y, -1) if halves else torch.stack(y, -1).flatten(-2)
    assert float((qx.cpu().double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())
    plane = torch.randn((4, 1, page, rank + rot), generator=g).bfloat16()
    table, tok_req, tok_pos = torch.tensor([[2, 0], [3, -1]]).int(), torch.tensor([0, 0, 1, 1]).int(), torch.tensor([0, 17, 15, 3]).int()
    c, kr = (torch.full((4, n), NAN, dtype=torch.bfloat16, device=DEV) for n in (rank, 64))
    K.latent_gather(plane.to(DEV), rank, tok_req.to(DEV), tok_pos.to(DEV), table.to(DEV), page, c, kr)
    rows = torch.stack([plane[int(table[r, p // page]), 0, p % page] for r, p in zip(tok_req.tolist(), tok_pos.tolist())])
    assert torch.equal(c.cpu(), rows[:, :rank]) and torch.equal(kr.cpu()[:, :rot], rows[:, rank:]) and not kr.cpu()[:, rot:].any()
