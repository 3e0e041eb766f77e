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
    x = torch.randn(T, 2 * groups * rows + heads * cols + 7, generator=g).to(DEV)
    raw = torch.randn(T, heads * (rows if mode == 2 else 1) + heads + 3, generator=g).to(DEV)
    off_dt, off_beta = 1, 2 + heads
    A, bias, skip = (torch.randn(heads, generator=g).to(DEV) * 0.3 for _ in range(3))
    n = K.state_scan_floats(heads, rows, cols, mode)
    slots = torch.randperm(R + 1, generator=g)[:R].int().to(DEV)
    starts = [sum(lengths[:i]) for i in range(R + 1)]
    results = []
    for single in (False, True):
        state, out = torch.zeros(R + 1, n + 3, device=DEV), torch.zeros(T, heads * cols, device=DEV)

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
        results.append((state, out))
    assert bool(results[0][1].abs().sum() > 0)
    assert torch.equal(results[0][1], results[1][1]) and torch.equal(results[0][0], results[1][0])
