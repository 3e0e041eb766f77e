"""Latent attention over a bfloat16 cache of 16-byte pieces (and over other sizes): against the plain formula in 64 bits."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rank,rot", [(64, 8), (512, 64), (448, 64), (576, 8), (1024, 16), (128, 4), (96, 32)])
@pytest.mark.parametrize("heads,window,sink,most", [(8, 0, False, 0), (9, 0, True, 4096), (3, 40, True, 700), (16, 100, False, 0)])
def test_latent_attention(rank, rot, heads, window, sink, most):
    from cajeta_llm_b200.csrc import kernels as K
    g = torch.Generator().manual_seed(13)
    positions = [0, 31, 32, 33, 700, 64, 129]
    T, page = len(positions), 16
    width = max(positions) // page + 1
    table = (torch.randperm(T * width, generator=g) + 1).view(T, width).int()
    plane = torch.randn(T * width + 1, 1, page, rank + rot, generator=g).to(torch.bfloat16)
    plane[0] = float("nan")                                   # a page that no row sees
    q_abs, q_rot = torch.randn(heads, T, rank, generator=g) * 0.3, torch.randn(T, heads, rot, generator=g)
    s = torch.randn(heads, generator=g) if sink else None
    if window:
        for r, p in enumerate(positions):                     # pages before the window may be gone
            table[r, :max(0, p + 1 - window) // page] = 0
    out = torch.empty(heads, T, rank, dtype=torch.bfloat16, device=DEV)
    scale = (rank + rot) ** -0.5
    K.latent_attention(q_abs.to(DEV), q_rot.to(DEV), plane.to(DEV), rank, rot, heads, torch.tensor(positions, dtype=torch.int32, device=DEV),
                       torch.arange(T, dtype=torch.int32, device=DEV), table.to(DEV), page, scale, out, max_context=most,
                       sink=None if s is None else s.to(DEV), window=window)
    for r, p in enumerate(positions):
        lo = max(0, p + 1 - window) if window else 0
        keys = plane[table[r].long()].reshape(-1, rank + rot)[lo:p + 1].double()
        q = torch.cat([q_abs[:, r], q_rot[r]], 1).double()
        sc = q @ keys.t() * scale
        if s is not None:
            sc = torch.cat([sc, s.double()[:, None]], 1)
        want = torch.softmax(sc, 1)[:, :p + 1 - lo] @ keys[:, :rank]
        assert torch.allclose(out[:, r].double().cpu(), want, atol=1e-2, rtol=1e-2), (r, float((out[:, r].double().cpu() - want).abs().max()))
        assert math.isfinite(float(out[:, r].float().sum()))


@pytest.mark.parametrize("rank,rot,dtype,window", [(64, 8, torch.bfloat16, 0), (200, 4, torch.float32, 0), (1024, 16, torch.bfloat16, 4400), (130, 2, torch.float32, 4000)])
def test_any_number_of_stretches_is_merged(rank, rot, dtype, window):
    """More stretches than the merge has threads, their maxima and sums at an address that is a multiple of four alone."""
    from cajeta_llm_b200.csrc import kernels as K
    g = torch.Generator().manual_seed(14)
    heads, page, positions, split = 3, 16, [4500, 31, 4127], 32
    T, pages = len(positions), 4500 // 16 + 1
    plane = torch.randn(pages, 1, page, rank + rot, generator=g).to(dtype)
    q_abs, q_rot = torch.randn(heads, T, rank, generator=g) * 0.3, torch.randn(T, heads, rot, generator=g)
    scale, most = (rank + rot) ** -0.5, min(4501, window or 4501)
    splits = -(-most // split)
    assert splits > 121
    acc = torch.full((T, heads, splits, rank), float("nan"), device=DEV)
    ml = torch.full((T * heads * splits * 2 + 1,), float("nan"), device=DEV)[1:]
    out = torch.empty(heads, T, rank, dtype=dtype, device=DEV)
    on = [t.to(DEV) for t in (q_abs, q_rot, plane, torch.tensor(positions, dtype=torch.int32), torch.zeros(T, dtype=torch.int32),
                              torch.arange(pages, dtype=torch.int32)[None])]
    P, I = K._ptr, K._i
    st = K.library("latent_attention").cj_latent_attention(
        P(on[0]), P(on[1]), P(on[2]), I(K._code(plane)), I(rank), I(rot), I(heads), I(T), P(on[3]), P(on[4]), P(on[5]), I(pages), I(page),
        I(window), K._f(scale), P(out), I(split), I(splits), P(acc), P(ml), P(None), K._stream())
    assert st == 0
    flat = plane.reshape(-1, rank + rot).double()
    for r, p in enumerate(positions):
        keys = flat[max(0, p + 1 - window) if window else 0:p + 1]
        want = torch.softmax(torch.cat([q_abs[:, r], q_rot[r]], 1).double() @ keys.t() * scale, 1) @ keys[:, :rank]
        assert torch.allclose(out[:, r].double().cpu(), want, atol=1e-2 if dtype == torch.bfloat16 else 1e-5, rtol=1e-2 if dtype == torch.bfloat16 else 1e-4)
