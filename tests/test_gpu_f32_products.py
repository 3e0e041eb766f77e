"""The float32 product on the tensor cores (three bfloat16 parts an operand) against 64 bits, at the edges of its tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def K():
    from cajeta_llm_b200.csrc import kernels
    return kernels


def rnd(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


def held(got, a, w, want):
    """The sum's error is at most, in units of 2^-24 of the sum of magnitudes: two roundings a block of 32 products, one for the terms left
    out, two for each of the leading products' two truncated adds inside a block, and one for the smaller terms'."""
    bound = (a.shape[-1] / 16 + 6) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t())
    assert bool(((got.double() - want).abs() <= bound).all()), float(((got.double() - want).abs() / bound).max())


@pytest.mark.parametrize("M,N,Kd", [(1, 64, 128), (16, 128, 132), (17, 129, 160), (33, 200, 2048), (64, 130, 1000), (65, 1408, 256),
                                     (129, 96, 1028), (300, 257, 136), (600, 260, 192)])
def test_plain_bias_accumulate_scale(K, M, N, Kd):
    a, w, b = rnd(M, Kd, seed=1), rnd(N, Kd, seed=2), rnd(N, seed=3)
    out = torch.empty(M, N, device=DEV)
    assert K.f32_tc_takes(a, w, None, out)
    want = a.double() @ w.double().t()
    K.gemm(a, w, out)
    held(out, a, w, want)
    base = rnd(M, N, seed=4)
    acc = base.clone()
    K.gemm(a, w, acc, bias=b, accumulate=True, out_scale=0.5)
    assert torch.allclose(acc.double(), 0.5 * (want + b.double()) + base.double(), atol=1e-4, rtol=1e-5)
    # rows do not depend on the batch: the same bits from a tile of any width
    for lo, hi in ((0, 1), (M // 2, M)):
        part = torch.empty(hi - lo, N, device=DEV)
        K.gemm(a[lo:hi], w, part)
        assert torch.equal(part, out[lo:hi])
    assert K.wait_errors() == {}


def low_bits(t):
    """Operands that three bfloat16 parts hold worst: the low 15 bits all set."""
    return (t.view(torch.int32) | 0x7FFF).view(torch.float32)


def on_the_fma_pipe(K, monkeypatch, a, w):
    out = torch.empty(a.shape[0], w.shape[0], device=DEV)
    with monkeypatch.context() as m:
        m.setattr(K, "f32_tc_takes", lambda *x: False)
        K.gemm(a, w, out)
    return out


@pytest.mark.parametrize("kind", ["given", "normal", "low bits"])
def test_rows_with_a_single_entry_are_right_to_their_last_place(K, kind):
    """One product: half a place for its rounding and at most as much for the terms left out."""
    n, Kd = 256, 128
    x, y = rnd(n, seed=17), rnd(n, seed=18)
    if kind == "given":
        x, y = torch.full_like(x, 1 + 2.0 ** -7 - 2.0 ** -23), torch.full_like(y, 1 + 2.0 ** -7 - 2.0 ** -23)
    if kind == "low bits":
        x, y = low_bits(x), low_bits(y)
    a = torch.zeros(n, Kd, device=DEV)
    a[torch.arange(n), torch.arange(n) % Kd] = x
    out = torch.empty(n, n, device=DEV)
    K.gemm(a, y[:, None].expand(n, Kd).contiguous(), out)
    want = x.double()[:, None] * y.double()[None, :]
    assert bool(((out.double() - want).abs() <= 2.0 ** -23 * want.abs()).all())


@pytest.mark.parametrize("Kd", [128, 2048])
def test_sums_of_one_sign_are_no_further_off_than_the_fma_pipes(K, monkeypatch, Kd):
    for low in (False, True):
        a, w = rnd(64, Kd, seed=19).abs(), rnd(128, Kd, seed=20).abs()
        if low:
            a, w = low_bits(a), low_bits(w)
        out, want = torch.empty(64, 128, device=DEV), a.double() @ w.double().t()
        K.gemm(a, w, out)
        held(out, a, w, want)
        assert float((out.double() - want).norm()) <= float((on_the_fma_pipe(K, monkeypatch, a, w).double() - want).norm())


@pytest.mark.parametrize("ea,ew", [(-124, 60), (-112, 60), (-104, 10), (-60, -58), (-149, 100), (126, -60), (64, 62)])
def test_operands_and_products_near_the_ends_of_the_range(K, monkeypatch, ea, ew):
    """Numbers that are not the sum of three parts, and products whose parts are not float32's, are as right as on the FMA pipe."""
    n, Kd = 64, 128
    g = torch.Generator().manual_seed(21)
    x, y = ((1 + torch.rand(n, generator=g)).double().mul(2.0 ** e).float().to(DEV) for e in (ea, ew))
    a = torch.zeros(n, Kd, device=DEV)
    a[torch.arange(n), torch.arange(n)] = x
    w = y[:, None].expand(n, Kd).contiguous()
    out, want = torch.empty(n, n, device=DEV), x.double()[:, None] * y.double()[None, :]
    K.gemm(a, w, out)
    fma = on_the_fma_pipe(K, monkeypatch, a, w)
    near = (out.double() - want).abs() <= 2.0 ** -23 * want.abs() + 2.0 ** -150
    assert bool((near | (torch.isinf(out) & torch.isinf(fma))).all())
    assert torch.equal(torch.isinf(out), torch.isinf(fma))


@pytest.mark.parametrize("n_tok", [16, 32, 64, 128])
@pytest.mark.parametrize("feat_tile", [64, 128])
def test_every_tile_gives_the_same_bits(K, monkeypatch, n_tok, feat_tile):
    a, w = rnd(150, 292, seed=12), rnd(200, 292, seed=13)
    out, other = torch.empty(150, 200, device=DEV), torch.empty(150, 200, device=DEV)
    K.gemm(a, w, out)
    monkeypatch.setattr(K, "f32_tc_tile", lambda *x: (n_tok, feat_tile))
    K.gemm(a, w, other)
    assert torch.equal(out, other)


@pytest.mark.parametrize("T,inter", [(1, 64), (7, 100), (70, 192), (200, 65), (800, 64)])
def test_gated_and_grouped(K, T, inter):
    H, E, k = 260, 5, 2
    x, wg, wu, wd = rnd(T, H, seed=5), rnd(E, inter, H, seed=6), rnd(E, inter, H, seed=7), rnd(E, H, inter, seed=8)
    sel = torch.randint(0, E - 1, (T * k,), generator=torch.Generator().manual_seed(9))       # the last group is empty
    order = torch.argsort(sel, stable=True)
    offsets = torch.cat([torch.zeros(1, dtype=torch.long), torch.bincount(sel, minlength=E).cumsum(0)]).int().to(DEV)
    index = (order // k).int().to(DEV)
    out = torch.empty(T * k, inter, device=DEV)
    K.gemm(x, wg, out, w_up=wu, group_offsets=offsets, a_row_index=index)
    down = torch.empty(T * k, H, device=DEV)
    K.gemm(out, wd, down, group_offsets=offsets)
    for e in range(E):
        lo, hi = int(offsets[e]), int(offsets[e + 1])
        rows = x[index[lo:hi].long()].double()
        g, u = rows @ wg[e].double().t(), rows @ wu[e].double().t()
        assert torch.allclose(out[lo:hi].double(), g * torch.sigmoid(g) * u, atol=1e-3, rtol=1e-4)
        assert torch.allclose(down[lo:hi].double(), out[lo:hi].double() @ wd[e].double().t(), atol=5e-3, rtol=1e-4)
    assert K.wait_errors() == {}


@pytest.mark.parametrize("n_tok", [16, 32, 64, 128])
@pytest.mark.parametrize("feat_tile", [64, 128])
def test_a_row_that_is_not_finite_changes_no_other_rows_bits(K, monkeypatch, n_tok, feat_tile):
    monkeypatch.setattr(K, "f32_tc_tile", lambda *x: (n_tok, feat_tile))
    a, w = rnd(140, 192, seed=22), rnd(200, 192, seed=23)
    plain, out = torch.empty(140, 200, device=DEV), torch.empty(140, 200, device=DEV)
    K.gemm(a, w, plain)
    rows, feats = [3, 64, 139], [0, 70, 199]
    a[3, 7], a[64, 100], a[139, 0], w[0, 9], w[70, 191], w[199, 31] = float("inf"), float("nan"), 2.0 ** -126, float("-inf"), 1e-40, float("nan")
    K.gemm(a, w, out)
    r, f = torch.ones(140, dtype=torch.bool), torch.ones(200, dtype=torch.bool)
    r[rows], f[feats] = False, False
    assert torch.equal(out[r][:, f], plain[r][:, f])
    want = a.double() @ w.double().t()
    assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(torch.isinf(out), torch.isinf(want))


@pytest.mark.parametrize("feat_tile", [32, 64])
def test_another_groups_weights_change_no_bits(K, monkeypatch, feat_tile):
    """Features that do not fill a group's last tile: the tile holds rows of the next group's weights too."""
    monkeypatch.setattr(K, "f32_tc_tile", lambda *x: (16, feat_tile))
    x, wg, wu = rnd(20, 128, seed=24), rnd(2, 72, 128, seed=25), rnd(2, 72, 128, seed=26)
    offsets = torch.tensor([0, 11, 20], dtype=torch.int32, device=DEV)
    plain, out = torch.empty(20, 72, device=DEV), torch.empty(20, 72, device=DEV)
    for gated in (False, True):
        K.gemm(x, wg, plain, w_up=wu if gated else None, group_offsets=offsets)
        bad_g, bad_u = wg.clone(), wu.clone()
        bad_g[1, 0, 3] = bad_u[1, 1, 5] = float("inf")
        K.gemm(x, bad_g, out, w_up=bad_u if gated else None, group_offsets=offsets)
        assert torch.equal(out[:11], plain[:11]) and torch.equal(out[11:, 2:], plain[11:, 2:])


def test_infinite_and_missing_numbers_are_summed_as_the_fma_pipe_sums_them(K):
    a, w = rnd(40, 192, seed=10), rnd(140, 192, seed=11)
    a[3, 7], a[20, 100], a[21, 0], w[5, 9] = float("inf"), float("nan"), 3.4e38, float("-inf")
    out = torch.empty(40, 140, device=DEV)
    K.gemm(a, w, out)
    want = a.double() @ w.double().t()
    want = torch.where(want.abs() > 3.4028235e38, torch.sign(want) * float("inf"), want)
    same = torch.isnan(out) == torch.isnan(want)
    assert bool(same.all()) and torch.equal(torch.isinf(out), torch.isinf(want.float()))


def test_rows_by_index_of_a_column_slice_and_slots_outside_the_groups(K):
    """Rows may be a column slice of a wider matrix; an index below 0 names a row of zeros; slots that no group holds are neither read nor
    written, and x need not have rows for them."""
    H, E, N, slots = 128, 3, 64, 40
    x, w = rnd(20, H + 16, seed=14)[:, 8:8 + H], rnd(E, N, H, seed=15)
    offsets = torch.tensor([2, 9, 9, 30], dtype=torch.int32, device=DEV)
    index = torch.full((slots,), -1, dtype=torch.int32, device=DEV)
    index[2:30] = torch.randint(0, 20, (28,), generator=torch.Generator().manual_seed(16)).int().to(DEV)
    index[5] = -1
    out = torch.full((slots, N), 7.0, device=DEV)
    assert K.f32_tc_takes(x, w, None, out)
    K.gemm(x, w, out, group_offsets=offsets, a_row_index=index)
    assert bool((out[:2] == 7.0).all()) and bool((out[30:] == 7.0).all()) and bool((out[5] == 0.0).all())
    rows = torch.where(index[:, None] >= 0, x[index.clamp(min=0).long()], 0.0)
    for e, (lo, hi) in enumerate(((2, 9), (9, 9), (9, 30))):
        held(out[lo:hi], rows[lo:hi], w[e], rows[lo:hi].double() @ w[e].double().t())
    again = torch.full((slots, N), 7.0, device=DEV)
    K.gemm(rows[:30].contiguous(), w, again, group_offsets=offsets, rows=slots)
    assert torch.equal(out, again)


@pytest.mark.parametrize("n_tok", [64, 128])
@pytest.mark.parametrize("Kd", [132, 192])
def test_rows_split_ahead_follow_their_index(K, monkeypatch, n_tok, Kd):
    """Tiles of many tokens take rows that were split once, through the index: the bits of tiles that split their own, rows of zeros and
    rows that are not finite among them."""
    x, w, up = rnd(90, Kd, seed=24), rnd(3, 70, Kd, seed=25), rnd(3, 70, Kd, seed=26)
    x[5, 3], x[60, 131], w[1, 9, 0] = float("inf"), 1e-40, float("nan")
    index = torch.randint(-1, 90, (300,), generator=torch.Generator().manual_seed(27)).int().to(DEV)
    index[:2] = torch.tensor([5, 60])
    offsets = torch.tensor([0, 130, 131, 290], dtype=torch.int32, device=DEV)
    index[290:] = 1 << 20                                       # outside the groups: never followed
    outs = []
    for n in (16, n_tok):
        monkeypatch.setattr(K, "f32_tc_tile", lambda *a, n=n: (n, 64))
        out = torch.zeros(300, 70, device=DEV)
        K.gemm(x, w, out, w_up=up, group_offsets=offsets, a_row_index=index)
        outs.append(out)
    assert torch.equal(outs[0].view(torch.int32), outs[1].view(torch.int32))
    finite = torch.isfinite(outs[0][:130][index[:130] != 5])
    assert bool(finite.all()) and bool(torch.isnan(outs[0][130, 9])) and not bool(outs[0][290:].any())
    assert K.wait_errors() == {}


@pytest.mark.parametrize("Kd", [132, 260])                      # five and nine blocks of K: the rings' places and phases move from tile to tile
def test_blocks_that_take_many_tiles(K, monkeypatch, Kd):
    """More tiles than the machine has blocks, the last ones part-filled, a row and a feature that are not finite in the middle ones."""
    a, w = rnd(2100, Kd, seed=28), rnd(1500, Kd, seed=29)
    plain, want = torch.empty(2100, 1500, device=DEV), a.double() @ w.double().t()
    K.gemm(a, w, plain)
    held(plain, a, w, want)
    a[1000, 5], w[700, 100] = float("inf"), 1e-40
    rows, feats = torch.arange(2100, device=DEV) != 1000, torch.arange(1500, device=DEV) != 700
    for n_tok in (16, 32, 64, 128):
        monkeypatch.setattr(K, "f32_tc_tile", lambda *x: (n_tok, 64))
        out = torch.empty(2100, 1500, device=DEV)
        K.gemm(a, w, out)
        assert torch.equal(out[rows][:, feats], plain[rows][:, feats]) and not bool(torch.isfinite(out[1000]).any())
        # gated and in groups: the two weights' sums cross while the next tile is under way
        offsets = torch.tensor([0, 1, 1, 700, 2100], dtype=torch.int32, device=DEV)
        wg, wu = w[:1480].view(4, 370, Kd), w[20:].view(4, 370, Kd)
        got = torch.empty(2100, 370, device=DEV)
        K.gemm(a, wg, got, w_up=wu, group_offsets=offsets)
        for g in range(4):
            lo, hi = int(offsets[g]), int(offsets[g + 1])
            x, y = (a[lo:hi].double() @ t[g].double().t() for t in (wg, wu))
            fine = torch.arange(lo, hi, device=DEV) != 1000
            assert torch.allclose(got[lo:hi].double()[fine], (x * torch.sigmoid(x) * y)[fine], atol=1e-3, rtol=1e-4)
    assert K.wait_errors() == {}


@pytest.mark.parametrize("n_tok", [16, 32, 64, 128])
@pytest.mark.parametrize("rows", [1, 17, 33])
def test_tokens_past_the_rows_of_x_are_rows_of_zeros(K, monkeypatch, n_tok, rows):
    """Fewer rows than tokens, and a row and a feature that send a tile to look for entries that are not the sum of three parts: the rows that
    x does not have are not read (memory behind them holds what no number is)."""
    monkeypatch.setattr(K, "f32_tc_tile", lambda *x: (n_tok, 64))
    behind, w = torch.full((160, 192), float("nan"), device=DEV), rnd(70, 192, seed=34)
    x = behind[:rows]
    x.copy_(rnd(rows, 192, seed=35))
    x[0, 5], w[66, 9] = 1e-40, 2.0 ** -126
    out = torch.full((150, 70), 7.0, device=DEV)
    K.gemm(x, w, out, rows=150)
    want = x.double() @ w.double().t()
    assert torch.allclose(out[:rows].double(), want, atol=1e-4, rtol=1e-5) and not bool(out[rows:].any())
    offsets = torch.tensor([0, 40, 150], dtype=torch.int32, device=DEV)
    K.gemm(x, torch.stack([w, w]), out, w_up=torch.stack([w, w]), group_offsets=offsets, rows=150)
    assert torch.allclose(out[:rows].double(), want * torch.sigmoid(want) * want, atol=1e-3, rtol=1e-4) and not bool(out[rows:].any())
    assert K.wait_errors() == {}


@pytest.mark.parametrize("groups", [1023, 1024, 1025, 2500])
def test_any_number_of_groups(K, monkeypatch, groups):
    """More groups than a block holds places for, empty ones at both ends and in runs, one with several tiles: the bits of the groups alone."""
    H, N = 128, 64
    g = torch.Generator().manual_seed(36)
    sizes = torch.randint(0, 3, (groups,), generator=g)
    sizes[:5], sizes[-40:], sizes[groups // 2:groups // 2 + 70] = 0, 0, 0
    sizes[7], sizes[groups - 41] = 150, 33
    offsets = torch.cat([torch.zeros(1, dtype=torch.long), sizes.cumsum(0)])
    T = int(offsets[-1])
    x, w = rnd(T, H, seed=37), rnd(groups, N, H, seed=38)
    want = torch.empty(T, N, device=DEV)
    for e in range(groups):
        lo, hi = int(offsets[e]), int(offsets[e + 1])
        if hi > lo:
            K.gemm(x[lo:hi], w[e], want[lo:hi])
    for n_tok in (16, 64):
        monkeypatch.setattr(K, "f32_tc_tile", lambda *a: (n_tok, 64))
        out = torch.empty(T, N, device=DEV)
        K.gemm(x, w, out, group_offsets=offsets.int().to(DEV))
        assert torch.equal(out, want)
    assert K.wait_errors() == {}
