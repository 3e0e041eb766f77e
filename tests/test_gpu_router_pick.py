"""Picks of equal scores, of scores of zero and of rows that are not numbers: the largest score, of equal ones the first expert."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("sigmoid", [False, True])
@pytest.mark.parametrize("E,k", [(1, 1), (2, 2), (33, 5), (60, 4), (64, 64), (513, 40), (1024, 8)])
def test_equal_scores_fall_to_the_first_expert(E, k, sigmoid):
    from cajeta_llm_b200.csrc import kernels as K
    g = torch.Generator().manual_seed(E)
    T = 40
    logits = torch.randint(-6, 7, (T, E), generator=g).float() / 2          # many equal ones; others apart by 1/2 and more
    logits[1:9][torch.rand(8, E, generator=g) < 0.5] = -float("inf")         # a score of exactly zero
    logits[1:9, 0] = 1.0
    logits[9] = float("nan")
    for rows in (T, 8):
        sel, w = torch.full((rows, k), -7, dtype=torch.int32, device=DEV), torch.empty(rows, k, device=DEV)
        gap = torch.empty(rows, device=DEV)
        K.router_select(logits[None, :rows].contiguous().to(DEV), E, k, False, sel, w, None, gap=gap, sigmoid_scores=sigmoid)
        real = logits[:rows].double()
        scores = torch.sigmoid(real) if sigmoid else torch.softmax(real, 1)
        want = torch.sort(-scores, dim=1, stable=True).indices[:, :k]
        ok = ~torch.isnan(real).any(1)
        assert torch.equal(sel.cpu().long()[ok], want[ok])
        # float32 exponentials, a sum of E of them and a division: a few units in the last place
        torch.testing.assert_close(w.cpu().double()[ok], torch.gather(scores, 1, want)[ok], rtol=3e-6, atol=0)
        bad = ~ok
        assert torch.equal(sel.cpu().long()[bad], torch.arange(k).expand(int(bad.sum()), k)) and bool(torch.isnan(w.cpu()[bad]).all())
