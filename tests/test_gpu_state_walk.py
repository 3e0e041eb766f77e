"""The scans of steps with many tokens a request (several columns and tokens at a time) and of single tokens give the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("heads,groups,rows,cols,lengths", [
    (64, 8, 128, 64, [4, 37]), (16, 8, 128, 128, [32, 1, 70]), (8, 8, 128, 256, [33, 8]), (8, 4, 128, 100, [65]),
    (32, 8, 64, 64, [9, 31]), (64, 64, 64, 72, [40]), (4, 4, 128, 30, [29])])
def test_walked_and_single_tokens_agree(mode, heads, groups, rows, cols, lengths):
    from cajeta_llm_b200.csrc import kernels as K
    g = torch.Generator().manual_seed(11)
    if mode >= 2:
        groups = heads
    R, T = len(lengths), sum(lengths)
    off_dt, off_beta = 1, 2 + heads
    A, bias, skip = (torch.randn(heads, generator=g).to(DEV) * 0.3 for _ in range(3))
    n = K.state_scan_floats(heads, rows, cols, mode)
    slots = torch.randperm(R + 1, generator=g)[:R].int().to(DEV)
    starts = [sum(lengths[:i]) for i in range(R + 1)]
    states = [torch.zeros(R + 1, n + 3, device=DEV) for _ in range(2)]
    for step in range(2):                                                    # from empty states, then from those the first step left
        x = torch.randn(T, 2 * groups * rows + heads * cols + 7, generator=g).to(DEV)
        raw = torch.randn(T, heads * (rows if mode == 2 else 1) + heads + 3, generator=g).to(DEV)
        outs = []
        for single, state in zip((False, True), states):
            out = torch.zeros(T, heads * cols, device=DEV)

            def scan(lo, hi, slot, req_start):
                K.state_scan(mode, x[lo:hi], 3, 3 + groups * rows, 3 + 2 * groups * rows, raw[lo:hi], off_dt, off_beta, A, bias, skip, state, 3,
                             torch.tensor(req_start, dtype=torch.int32, device=DEV), slot, out[lo:hi], slot.numel(), heads, groups, rows, cols,
                             q_scale=0.125, c0=5.0 if mode == 3 else 0.25, c1=1e-6)

            if single:
                for r in range(R):
                    for t in range(starts[r], starts[r + 1]):
                        scan(t, t + 1, slots[r:r + 1].contiguous(), [0, 1])
            else:
                scan(0, T, slots, starts)
            outs.append(out)
        assert bool(outs[0].abs().sum() > 0) and bool(states[0][slots.long()].abs().sum(1).min() > 0)
        assert torch.equal(outs[0], outs[1]) and torch.equal(states[0], states[1])


def test_raw_rows_that_end_with_the_requests():
    """x may have rows behind the requests' (of another step's length, say) that raw has not: the same bits."""
    from cajeta_llm_b200.csrc import kernels as K
    heads, rows, cols, T, more = 4, 128, 64, 40, 24
    g = torch.Generator().manual_seed(12)
    x, raw = torch.randn(T + more, heads * (2 * rows + cols), generator=g).to(DEV), torch.randn(T, heads * rows, generator=g).to(DEV)
    start, slot = torch.tensor([0, T], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    outs = []
    for n in (T, T + more):
        state, out = torch.zeros(1, K.state_scan_floats(heads, rows, cols, K.SCAN_GLA), device=DEV), torch.zeros(n, heads * cols, device=DEV)
        K.state_scan(K.SCAN_GLA, x[:n], 0, heads * rows, 2 * heads * rows, raw, 0, 0, None, None, None, state, 0, start, slot, out, 1, heads, heads,
                     rows, cols, q_scale=0.125, c0=0.25)
        outs.append((out[:T], state))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
