"""Row kernels around the recurrent mixers at the edges of their vector forms: against the plain formulas in 64 bits, and their order of sums."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


@pytest.mark.parametrize("rows,H", [(3, 4), (5, 1020), (2, 1024), (9, 2048), (4, 2052), (3, 8192), (2, 8196), (3, 77)])
def test_rmsnorm_add(rows, H):
    from cajeta_llm_b200.csrc import kernels as K
    hs, y, w = rnd(rows, H, seed=1), rnd(rows, H, seed=2), rnd(H, seed=3)
    want = hs.double() + y.double() / torch.sqrt((y.double() ** 2).mean(-1, keepdim=True) + 1e-6) * w.double()
    got = hs.clone()
    K.rmsnorm_add(got, y, w, 1e-6)
    assert torch.allclose(got.double(), want, atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("taps", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("channels,offset,lengths", [(512, 4, [1, 2, 200]), (516, 0, [127, 3, 17, 1]), (1028, 8, [130]), (510, 0, [140]), (512, 3, [128]),
                                                      (64, 0, [5, 9])])
@pytest.mark.parametrize("dtype,activate", [(torch.float32, True), (torch.bfloat16, False)])
def test_short_conv_of_many_rows_equals_token_by_token(taps, channels, offset, lengths, dtype, activate):
    from types import SimpleNamespace
    from cajeta_llm_b200.csrc import kernels as K
    R, T = len(lengths), sum(lengths)
    x, w, b = rnd(T, channels + 12, seed=4), rnd(channels, taps, seed=5), rnd(channels, seed=6)
    slots = torch.randperm(R + 1, generator=torch.Generator().manual_seed(7))[:R].int().to(DEV)
    starts = [sum(lengths[:i]) for i in range(R + 1)]
    req = torch.cat([torch.full((n,), i) for i, n in enumerate(lengths)]).int().to(DEV)
    first = rnd(R + 1, (taps - 1) * channels + 5, seed=8)
    results = []
    for single in (False, True):
        state, out = first.clone(), torch.empty(T, channels, device=DEV, dtype=dtype)

        def conv(rows, row_req, req_start, slot, all_single):
            part = torch.empty(len(rows), channels, device=DEV, dtype=dtype)
            ctx = SimpleNamespace(row_req=row_req, req_start=torch.tensor(req_start, dtype=torch.int32, device=DEV), req_slot=slot,
                                  n_requests=slot.numel(), all_single=all_single)
            K.short_conv_moved(x[rows].contiguous(), offset, channels, taps, w, b, state, ctx, part, activate=activate, state_offset=5)
            out[rows] = part

        if single:
            for t in range(max(lengths)):                                    # a step of every request that has a token t
                live = [r for r in range(R) if t < lengths[r]]
                conv([starts[r] + t for r in live], torch.arange(len(live), dtype=torch.int32, device=DEV), list(range(len(live) + 1)),
                     slots[live].contiguous(), True)
        else:
            conv(list(range(T)), req, starts, slots, False)
        results.append((out, state))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
    if taps > 1:                                                             # and the formula, for the last request
        r = R - 1
        padded = torch.cat([first[slots[r], 5:5 + (taps - 1) * channels].view(taps - 1, channels), x[starts[r]:starts[r + 1], offset:offset + channels]]).double()
        want = sum(w.double()[:, j] * padded[j:j + lengths[r]] for j in range(taps)) + b.double()
        want = want * torch.sigmoid(want) if activate else want
        tol = dict(atol=1e-5, rtol=1e-5) if dtype == torch.float32 else dict(atol=2e-2, rtol=1e-2)
        assert torch.allclose(results[0][0][starts[r]:].double(), want, **tol)


@pytest.mark.parametrize("n,part,w_len,z_offset", [(512, 128, 128, 4), (1024, 256, 1024, 0), (1024, 512, 1024, 8), (2048, 1024, 1024, 0), (768, 384, 768, 0),
                                                    (512, 128, 128, 3)])
@pytest.mark.parametrize("gate_first,sigmoid", [(True, False), (False, False), (False, True)])
def test_gated_group_norm(n, part, w_len, z_offset, gate_first, sigmoid):
    from cajeta_llm_b200.csrc import kernels as K
    y, z, w = rnd(5, n, seed=9), rnd(5, n + 12, seed=10), rnd(w_len, seed=11)
    out = torch.empty(5, n, device=DEV)
    K.gated_group_norm(y, part, z, z_offset, w, 1e-6, gate_first, out, sigmoid_gate=sigmoid)
    zz = z[:, z_offset:z_offset + n].double()
    gate = torch.sigmoid(zz) * (1.0 if sigmoid else zz)
    v = (y.double() * gate if gate_first else y.double()).view(5, n // part, part)
    v = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-6)).reshape(5, n) * w.double().repeat(n // w_len)
    assert torch.allclose(out.double(), v if gate_first else v * gate, atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("rows,H", [(2, 100), (2, 512), (3, 2048), (2, 4100), (2, 8192), (2, 9000)])
def test_rmsnorm_add_sums_a_row_in_one_order(rows, H):
    """A thread's entries one after the other (every 128th, 256th or 512th of the row, by its width), a warp's threads in pairs 16, 8, 4, 2
    and 1 apart, then the warps: the same bits whichever kernel ran."""
    from cajeta_llm_b200.csrc import kernels as K
    f, wide = np.float32, np.longdouble                      # (a product of two float32 is exact in the wide type)
    hs, y, w = rnd(rows, H, seed=12), rnd(rows, H, seed=13), rnd(H, seed=14)
    threads = 512 if H >= 2048 else 256 if H >= 512 else 128
    want = []
    for h, v in zip(hs.cpu().numpy(), y.cpu().numpy()):
        part = np.zeros(threads, f)
        for i in range(0, H, threads):
            e = v[i:i + threads].astype(wide)
            part[:len(e)] = (e * e + part[:len(e)]).astype(f)
        part = part.reshape(-1, 32)
        for o in (16, 8, 4, 2, 1):
            part = part + part[:, np.arange(32) ^ o]
        total = f(0.0)
        for p in part[:, 0]:
            total = f(total + p)
        scale = f(1.0) / np.sqrt(f(f(total / f(H)) + f(1e-6)))
        want.append(((v * scale).astype(wide) * w.cpu().numpy() + h).astype(f))
    got = hs.clone()
    K.rmsnorm_add(got, y, w, 1e-6)
    assert np.array_equal(got.cpu().numpy(), np.stack(want))


@pytest.mark.parametrize("part", [128, 256, 512, 1024])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("gate_first,sigmoid", [(True, False), (False, True)])
def test_gated_group_norm_gives_the_same_bits_for_any_weight_length(part, dtype, gate_first, sigmoid):
    from cajeta_llm_b200.csrc import kernels as K
    y, z, w = rnd(7, part, seed=15), rnd(7, part, seed=16), rnd(part + 32, seed=17)
    outs = [torch.empty(7, part, device=DEV, dtype=dtype) for _ in range(2)]
    K.gated_group_norm(y, part, z, 0, w, 1e-6, gate_first, outs[0], sigmoid_gate=sigmoid)          # a weight of another length: entry by entry
    K.gated_group_norm(y, part, z, 0, w[:part].clone(), 1e-6, gate_first, outs[1], sigmoid_gate=sigmoid)
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("rows", [1, 5])
def test_a_normed_mixers_output_product_is_one_sum(monkeypatch, rows):
    """Where a norm follows at once, the output product of a state mixer is one sum over K for few rows as for many, not partial sums."""
    from cajeta_llm_b200 import bench_design as B
    from cajeta_llm_b200.config import parse_config_dict
    from cajeta_llm_b200.csrc import kernels as K
    from cajeta_llm_b200.engine.model import random_model
    from cajeta_llm_b200.engine.step import ModelRunner, StepEntry
    from cajeta_llm_b200.parts.base import Runtime
    config = B.balalorn_config(dict(width=512, layers=4, heads=4, rank=128, experts=4, top=2, eff=128, ff=256, state=64))
    config["vocab"], config["layers"] = 300, [dict(c, mlp=None) for c in config["layers"][1:3]]
    r = ModelRunner(random_model(parse_config_dict(config), Runtime("bfloat16"), 5), max_seqs=rows, max_tokens_per_seq=64, cuda_graphs=False)
    cuts, plain = [], K.gemm_tc
    monkeypatch.setattr(K, "gemm_tc", lambda *a, **k: (cuts.append(k.get("k_splits", 1)), plain(*a, **k)))
    r.step([StepEntry(r.admit(), [i], [0]) for i in range(rows)])
    assert cuts and set(cuts) == {1}


def test_single_tokens_convolution_of_more_channels_than_a_grid_has_threads():
    from types import SimpleNamespace
    from cajeta_llm_b200.csrc import kernels as K
    C, taps = 65535 * 128 + 5, 2
    x, w, state = rnd(1, C, seed=18), rnd(C, taps, seed=19), rnd(1, C, seed=20)
    at = torch.zeros(1, dtype=torch.int32, device=DEV)
    want, out = w[:, 0] * state[0] + w[:, 1] * x[0], torch.empty(1, C, device=DEV)
    K.short_conv_moved(x, 0, C, taps, w, None, state, SimpleNamespace(row_req=at, req_slot=at, all_single=True), out, activate=False)
    assert torch.allclose(out[0], want, atol=1e-5, rtol=1e-5) and torch.equal(state, x)


@pytest.mark.parametrize("rows,n", [(1, 1), (3, 100), (2, 1023), (4, 2048), (2, 2049), (3, 5000)])
def test_row_norms_whose_first_entries_stay_in_registers(rows, n):
    """Widths around what the threads hold (latent_q_norm 1,024 and 2,048, gated_row_norm 512 to 2,048), and past it."""
    from cajeta_llm_b200.csrc import kernels as K
    x, z, w = rnd(rows, n + 3, seed=31), rnd(rows, n + 5, seed=32), rnd(n, seed=33)
    v = x[:, 2:2 + n].double()
    want = v / torch.sqrt((v ** 2).mean(-1, keepdim=True) + 1e-6) * w.double()
    out = torch.empty(rows, n, device=DEV)
    K.latent_q_norm(x, 2, n, w, 1e-6, out)
    assert torch.allclose(out.double(), want, atol=1e-5, rtol=1e-5)
    K.gated_row_norm(x[:, 2:2 + n].contiguous(), z, 4, w, 1e-6, out)
    assert torch.allclose(out.double(), want * torch.sigmoid(z[:, 4:4 + n].double()), atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("H", [8, 20, 264, 2048, 2056])
def test_embedding_rows_in_pieces_of_eight(H):
    """Rows of whole 16-byte pieces and not, a scale, and an id out of range."""
    from cajeta_llm_b200.csrc import kernels as K
    table = rnd(7, H, seed=41).bfloat16()
    ids = torch.tensor([6, 0, 3, 9, -1], dtype=torch.int32, device=DEV)
    for scale in (0.0, 1.75):
        out = torch.empty(5, H, device=DEV)
        K.embed_gather(out, table, ids, scale)
        want = torch.cat([table[[6, 0, 3]].float() * (scale or 1.0), torch.zeros(2, H, device=DEV)])
        assert torch.equal(out, want)


@pytest.mark.parametrize("rows,H", [(1, 4), (3, 7), (5, 1028), (2, 2048), (3, 4096), (2, 4100)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_two_normed_rows_mixed_and_cast(rows, H, accumulate):
    from cajeta_llm_b200.csrc import kernels as K
    a, b, wa, wb, out = rnd(rows, H, seed=42), rnd(rows, H, seed=43), rnd(H, seed=44), rnd(H, seed=45), rnd(rows, H, seed=46)

    def normed(t, w):
        return t.double() / torch.sqrt((t.double() ** 2).mean(-1, keepdim=True) + 1e-6) * w.double()

    want = 0.5 * (normed(a, wa) + normed(b, wb)) + (out.double() if accumulate else 0.0)
    K.rmsnorm_mix2(a, wa, b, wb, 1e-6, 0.5, out, accumulate=accumulate)
    assert torch.allclose(out.double(), want, atol=1e-5, rtol=1e-5)
    for dtype in (torch.float32, torch.bfloat16):
        cast = torch.empty(rows, H, device=DEV, dtype=dtype)
        K.cast_rows(out, cast)
        assert torch.equal(cast, out.to(dtype))


@pytest.mark.parametrize("H", [248, 256, 508, 512, 516])
def test_rows_on_both_sides_of_the_widths_that_go_in_pieces(H):
    from cajeta_llm_b200.csrc import kernels as K
    a, b, wa, wb, out = rnd(3, H, seed=51), rnd(3, H, seed=52), rnd(H, seed=53), rnd(H, seed=54), torch.empty(3, H, device=DEV)
    K.rmsnorm_mix2(a, wa, b, wb, 1e-6, 0.5, out)
    x, y = (t.double() / torch.sqrt((t.double() ** 2).mean(-1, keepdim=True) + 1e-6) * w.double() for t, w in ((a, wa), (b, wb)))
    assert torch.allclose(out.double(), 0.5 * (x + y), atol=1e-5, rtol=1e-5)
    table, ids = rnd(7, H, seed=55).bfloat16(), torch.tensor([6, 0, -1], dtype=torch.int32, device=DEV)
    K.embed_gather(out, table, ids, 0.0)
    assert torch.equal(out, torch.cat([table[[6, 0]].float(), torch.zeros(1, H, device=DEV)]))
