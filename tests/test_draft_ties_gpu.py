"""Draft levels whose rows' best entries crowd into one vocabulary segment of 2048 or tie at the threshold: what a segment does not list is
then looked for in its logits (draft_tree.cu).  Bit-exact against a stable sort of the log-probabilities, which are taken from the kernel where
an fp32 sum in another order may round one of them elsewhere (so the logits here have few distinct values: every lp of a row shifts alike)."""
import numpy as np
import pytest
import torch

from test_kernels_gpu import C, dev, run_gpu_tree

pytestmark = pytest.mark.gpu


def rows_of(kind, n, V, k, g):
    x = torch.zeros(n, V)
    if kind == "flat":                      # every entry ties
        return x
    if kind == "one segment":               # the k + 5 best in the last segment, ties among them
        first = (V - 1) // 2048 * 2048
        for r in range(n):
            at = first + torch.randperm(V - first, generator=g)[:k + 5]
            x[r, at] = 8.0 + (torch.arange(len(at)) // 3 % 3).float()
        return x
    if kind == "two levels":                # fewer than k above, the rest tie in many segments
        for r in range(n):
            x[r, torch.randperm(V, generator=g)[:max(k // 2, 1)]] = 9.0
            x[r, torch.randperm(V, generator=g)[:4 * k]] += 3.0
        return x
    x += torch.randint(0, 3, (n, V), generator=g) * 2.0   # a third of the row ties at the top
    return x


@pytest.mark.parametrize("kind", ["flat", "one segment", "two levels", "thirds"])
@pytest.mark.parametrize("V,k", [(2049, 10), (4100, 32), (5000, 4), (73448, 10), (32768, 1)])
def test_ties(kind, V, k):
    c = C()
    n_iter, T = 2, min(16, k + 1)
    g = torch.Generator().manual_seed(V + k)
    logits = rows_of(kind, 1 + (n_iter - 1) * k, V, k, g).to(torch.bfloat16)
    *_, tv, tp, _ = run_gpu_tree(c, dev(logits), k, n_iter, T, 100)
    x = logits.float().numpy()
    want = [np.argsort(-row, kind="stable")[:k] for row in x]
    assert np.array_equal(tp[:k], want[0])
    assert np.array_equal(tp[k:].reshape(k, k), np.stack(want[1:1 + k]))
    # an lp below its row's first by the logits' difference: one bf16 step of the larger magnitude (under 32)
    lp = tv[:k] - tv[0] - (x[0][want[0]] - x[0][want[0][0]])
    assert np.abs(lp).max() <= 0.125
