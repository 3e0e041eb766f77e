"""What the kernels' Python face hands to the libraries, on the CPU: the libraries are stood in for, nothing is launched."""
import ctypes

import pytest
import torch

from cajeta_llm_b200.csrc import kernels as K


class Calls:
    """A library whose every function takes its arguments down and succeeds; ``answers``: what a function returns instead of 0."""

    def __init__(self, **answers):
        self.answers, self.made = answers, []

    def __getattr__(self, name):
        def call(*args):
            self.made.append((name, [a.value if isinstance(a, ctypes._SimpleCData) else a for a in args]))
            answer = self.answers.get(name, 0)
            return answer(args) if callable(answer) else answer
        return call


@pytest.fixture
def calls(monkeypatch):
    lib = Calls()
    monkeypatch.setattr(K, "library", lambda name: lib)
    monkeypatch.setattr(K, "_need", lambda *a: None)
    monkeypatch.setattr(K, "_stream", lambda: ctypes.c_void_p(0))
    monkeypatch.setattr(K, "_sm_count", lambda: 148)
    real = K._libs.get("recurrent") or ctypes.CDLL(K._build.build("recurrent"))
    lib.answers["cj_state_scan_walks"] = lambda args: real.cj_state_scan_walks(*args)
    scratch = ctypes.CDLL(K._build.build("gemm_f32_tc")).cj_gemm_f32_tc_scratch
    scratch.restype = ctypes.c_longlong
    lib.answers["cj_gemm_f32_tc_scratch"] = lambda args: scratch(*args)
    return lib


def scan(mode, tokens, raw_rows, requests, **kw):
    heads, rows, cols = 4, 128, 256
    x, raw = torch.zeros(tokens, heads * (2 * rows + cols)), torch.zeros(raw_rows, heads * rows)
    K.state_scan(mode, x, 0, heads * rows, 2 * heads * rows, raw, 0, heads, *[torch.zeros(heads)] * 3, torch.zeros(2, K.state_scan_floats(heads, rows, cols, mode)),
                 0, torch.zeros(requests + 1, dtype=torch.int32), torch.zeros(requests, dtype=torch.int32), torch.zeros(tokens, heads * cols), requests, heads,
                 heads, rows, cols, c0=0.25, **kw)


def test_decays_of_all_rows_only_where_all_rows_have_them(calls):
    """Gated linear attention works the decays of all of x's rows out ahead; the scan alone needs those of the requests' rows."""
    scan(K.SCAN_GLA, 64, 64, 1)
    scan(K.SCAN_GLA, 64, 40, 1)
    scan(K.SCAN_DELTA, 64, 64, 1)
    scan(K.SCAN_GLA, 64, 64, 9)                                               # (seven rows a request: too few to walk)
    pointers = [args[-3] for name, args in calls.made if name == "cj_state_scan"]
    assert pointers[0] and not any(pointers[1:])


def test_a_few_requests_with_many_tokens_are_not_single_ones(calls):
    """62 rows in a layout of 64 requests: 32 single tokens and one request of 30, say.  The caller knows; without it no more rows than requests
    count as single tokens."""
    scan(K.SCAN_SSD, 62, 62, 64, single=False)
    scan(K.SCAN_SSD, 62, 62, 64, single=True)
    scan(K.SCAN_SSD, 62, 62, 64)
    scan(K.SCAN_SSD, 65, 65, 64)
    assert [args[-2] for name, args in calls.made if name == "cj_state_scan"] == [0, 1, 1, 0]


def counted(call, *args, **kw):
    before = K.launches
    call(*args, **kw)
    return K.launches - before


def test_every_kernel_of_a_call_is_counted(calls, monkeypatch):
    """A product that splits or gathers its rows first, and a scan whose decays are worked out first, are two kernels."""
    x, w, out = torch.zeros(300, 256), torch.zeros(3, 128, 256), torch.zeros(300, 128)
    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda t: True))
    offsets, index = torch.tensor([0, 100, 200, 300], dtype=torch.int32), torch.arange(300, dtype=torch.int32)
    for n_tok, many, index_given, kernels in ((16, False, None, 1), (16, True, None, 1), (32, True, index, 2), (64, False, None, 2), (128, True, index, 2)):
        monkeypatch.setattr(K, "f32_tc_tile", lambda *a: (n_tok, 64))
        assert counted(K.gemm, x, w if many else w[0], out, group_offsets=offsets if many else None, a_row_index=index_given) == kernels
    assert counted(scan, K.SCAN_GLA, 64, 64, 1) == 2 and counted(scan, K.SCAN_GLA, 64, 40, 1) == 1 and counted(scan, K.SCAN_SSD, 64, 64, 1) == 1


@pytest.mark.parametrize("n_tok,indexed", [(16, False), (32, True), (64, False), (128, True)])
def test_a_float32_product_refuses_scratch_that_is_too_small(n_tok, indexed):
    """The library's own entry (its host side launches nothing before the check): a byte short, and no scratch at all."""
    lib, one = K.library("gemm_f32_tc"), ctypes.c_void_p(1 << 20)
    need = K._f32_tc_scratch(100, 260, n_tok, indexed)
    assert need == (100 * (6 * 288 + 4) if n_tok >= 64 else 100 * 260 * 4 if indexed else 0)

    def call(scratch, size):
        null = ctypes.c_void_p(0)
        return lib.cj_gemm_f32_tc(one, K._ll(260), K._i(100), one if indexed else null, scratch, K._ll(size), one, null, null, null, one, K._ll(64), K._i(100),
                                  K._i(64), K._i(260), K._i(0), null, K._i(0), K._f(0), K._f(1), K._f(0), K._i(0), K._i(0), K._f(1), K._i(n_tok), K._i(64),
                                  null)

    if need:
        assert call(one, need - 1) == -5 and call(ctypes.c_void_p(0), need) == -5


@pytest.mark.parametrize("rows,features,groups,gated,tile", [
    (1, 2048, 0, False, (16, 128)), (8, 6144, 0, False, (16, 128)), (60, 2048, 0, False, (16, 128)), (60, 6144, 0, False, (32, 128)),
    (264, 2048, 0, False, (32, 128)), (264, 6144, 0, False, (128, 128)), (512, 2048, 0, False, (64, 128)), (1777, 2048, 0, False, (128, 128)),
    (8, 5632, 0, True, (16, 64)), (60, 5632, 0, True, (64, 64)), (264, 5632, 0, True, (128, 64)),
    (64, 512, 16, True, (16, 64)), (500, 512, 16, True, (64, 64)), (8, 1408, 8, True, (16, 64)), (16, 1024, 16, False, (16, 128)),
    (1056, 1408, 60, True, (32, 64)), (7108, 1408, 60, True, (128, 64))])
def test_tiles_of_float32_products(rows, features, groups, gated, tile):
    """Tiles as measured; no tile is cut in half along its features: that makes rounds, not shorter blocks."""
    assert K.f32_tc_tile(rows, features, groups, gated, 148) == tile


@pytest.mark.parametrize("heads,requests,split_keys,tcgen05", [
    # (tokens before, rows) of the requests; what the tiles of 64 rows cut the keys into; which form was the faster one
    (16, [(3000, 256)], 2048, True), (8, [(3000, 256)], 1024, False), (2, [(3000, 256)], 320, False), (8, [(1000, 256)], 1024, True),
    (4, [(2000, 512)], 832, False), (4, [(3000, 512)], 832, False), (8, [(3000, 1024)], 0, True), (16, [(0, 256)], 2048, True),
    (16, [(0, 8)] * 32, 0, False), (16, [(0, 32)] * 8, 0, False), (16, [(0, 100)] * 8, 0, True), (16, [(500, 8)] * 32, 0, True),
    (16, [(0, 256)] + [(500, 1)] * 60, 0, True), (16, [(0, 256)] + [(2000, 1)] * 16, 0, True), (16, [(0, 256)] + [(50, 1)] * 60, 0, False),
    (16, [(0, 1000)] + [(50, 1)] * 30, 0, True), (32, [(100, 16)] * 16, 0, False), (16, [(0, 256), (7, 0), (0, 0)], 2048, True)])
def test_which_form_differential_attention_takes(heads, requests, split_keys, tcgen05):
    assert K.diff_tc_pays([r for _, r in requests], [p for p, _ in requests], heads, 0, split_keys, 148) == tcgen05


def test_a_window_bounds_what_a_tile_reads():
    """Far behind its window a portion costs what its window costs."""
    near, far = ([K.diff_tc_pays([256] * n, [p] * n, h, 512, 0, 148) for n in (1, 4, 16) for h in (2, 8, 32)] for p in (512, 100000))
    assert near == far


def test_differential_attention_asks_from_256_rows_on(calls, monkeypatch):
    asked = []
    monkeypatch.setattr(K, "diff_tc_pays", lambda *a: asked.append(a) or False)
    for rows, given in (([255], True), ([256], True), ([200, 56], True), ([256], False)):
        T, H = sum(rows), 16
        start = torch.tensor([0] + list(torch.tensor(rows).cumsum(0)), dtype=torch.int32)
        q, out = torch.zeros(T, H, 128, dtype=torch.bfloat16), torch.zeros(T, H, 128, dtype=torch.bfloat16)
        k, v = torch.zeros(40, 8, 16, 128, dtype=torch.bfloat16), torch.zeros(40, 8, 16, 128, dtype=torch.bfloat16)
        z = torch.zeros(T, dtype=torch.int32)
        K.diff_attention(q, out, k, v, z, z, torch.zeros(len(rows), 4, dtype=torch.int32), 16, H, 8, 64, 128, 0, 0.125, 0.5, 1e-6, 0.5, start,
                         torch.zeros(len(rows), dtype=torch.int32), len(rows), 64, h_rows=rows if given else None, h_prior=[0] * len(rows) if given else None)
    assert [a[0] for a in asked] == [[256], [200, 56]]
    assert [name for name, _ in calls.made] == ["cj_diff_attention_tile"] * 3 + ["cj_diff_attention_tc"]


@pytest.mark.parametrize("rows,columns,a_block", [(40, 61, 8), (99, 61, 8), (264, 61, 8), (512, 61, 16), (1000, 61, 32), (1777, 61, 61), (33, 257, 8), (264, 257, 32),
                                                  (512, 257, 32), (1000, 257, 32), (1000, 129, 32), (1777, 257, 257), (4000, 17, 17), (600, 3, 8), (5000, 3, 8)])
def test_experts_of_a_router_block(rows, columns, a_block):
    """Many experts are spread over blocks until the row blocks by themselves fill the machine."""
    lib = ctypes.CDLL(K._build.build("moe_route"))
    assert lib.cj_router_experts_a_block(-(-rows // 8), columns, 2 * 148) == a_block


@pytest.mark.parametrize("rows,columns,a_block", [(700, 16, 16), (1000, 16, 16), (512, 61, 32), (264, 129, 32), (99, 61, 8), (2000, 61, 61)])
def test_experts_of_a_router_block_that_has_an_sm_to_itself(rows, columns, a_block):
    lib = ctypes.CDLL(K._build.build("moe_route"))
    assert lib.cj_router_experts_a_block(-(-rows // 8), columns, 148) == a_block


def test_products_and_scans_run_without_room_for_scratch(calls, monkeypatch):
    """Where the memory for split rows or for decays is not there, the forms that need none (or the gathered rows alone) run."""
    real, limit = torch.empty, [0]

    def empty(*size, **kw):
        n = 1
        for d in size[0]:
            n *= d
        if n * (4 if kw.get("dtype") == torch.float32 else 1) > limit[0]:
            raise torch.OutOfMemoryError("no room")
        return real(*size, **kw)

    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda t: True))
    monkeypatch.setattr(torch, "empty", empty)
    x, w, out = torch.zeros(300, 256), torch.zeros(3, 128, 256), torch.zeros(300, 128)
    offsets, index = torch.tensor([0, 100, 200, 300], dtype=torch.int32), torch.arange(300, dtype=torch.int32)
    monkeypatch.setattr(K, "f32_tc_tile", lambda *a: (128, 64))
    K.gemm(x, w[0], out)
    K.gemm(x, w, out, group_offsets=offsets)
    with pytest.raises(torch.OutOfMemoryError):
        K.gemm(x, w, out, group_offsets=offsets, a_row_index=index)
    limit[0] = 300 * 256 * 4
    K.gemm(x, w, out, group_offsets=offsets, a_row_index=index)
    limit[0] = 300 * (256 * 6 + 4)
    K.gemm(x, w, out, group_offsets=offsets, a_row_index=index)
    products = [args for name, args in calls.made if name == "cj_gemm_f32_tc"]
    assert [args[-3] for args in products] == [32, 32, 32, 128] and [bool(args[4]) for args in products] == [False, False, True, True]
    limit[0] = 0
    scan(K.SCAN_GLA, 64, 64, 1)
    assert not calls.made[-1][1][-3]


@pytest.mark.parametrize("heads,dim,vdim,window,requests,tcgen05", [
    # (tokens before, rows) of the requests; which form was the faster one
    (16, 128, 128, 0, [(0, 4)] * 64, False), (32, 64, 64, 0, [(0, 4)] * 64, False), (16, 128, 128, 0, [(0, 8)] * 32, False), (32, 128, 128, 512, [(0, 8)] * 32, False),
    (16, 128, 128, 0, [(0, 16)] * 16, True), (16, 128, 128, 0, [(0, 256)], True), (16, 128, 128, 0, [(0, 2000)], True), (8, 128, 128, 0, [(3000, 256)], True),
    (16, 128, 128, 0, [(0, 256)] + [(500, 1)] * 60, True), (16, 128, 128, 0, [(0, 256)] + [(20, 1)] * 60, False), (16, 128, 128, 0, [(500, 8)] * 32, True),
    (16, 64, 64, 0, [(200, 4)] * 64, True), (4, 128, 128, 0, [(0, 100)] * 8, True), (16, 128, 128, 0, [(0, 300), (9, 0)], True)])
def test_which_form_latent_attention_takes(heads, dim, vdim, window, requests, tcgen05):
    assert K.latent_tc_pays([r for _, r in requests], [p for p, _ in requests], heads, dim, vdim, window, 148) == tcgen05
