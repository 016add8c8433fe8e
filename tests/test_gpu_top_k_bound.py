"""Top-k sampling where the bound in front of the selection is loose, empty or tied: all logits equal, a handful of values, the
kept ones all in one block's share, in the last ids, blocks with fewer threads at work than the bound counts, and logits that
leave more keys above the bound than block 0 holds.  The token's slice of the float64 distribution over the kept ids contains
the row's uniform number."""
import numpy as np
import pytest
import torch

import plain_llama as pl

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("vocab", [8192, 8200, 32000, 128256])
@pytest.mark.parametrize("top_k", [1, 2, 7, 8, 9, 40, 200, 513, 1024])
def test_kept_ids(vocab, top_k):
    from cpp_minilamma_b200.csrc import kernels as K
    gen = torch.Generator().manual_seed(vocab + top_k)
    rows = [torch.zeros(vocab), torch.randint(0, 4, (vocab,), generator=gen).float(), torch.arange(vocab).float() / vocab,
            -torch.arange(vocab).float() / vocab, torch.randn(vocab, generator=gen), torch.full((vocab,), -3.0)]
    rows[5][:top_k] = 1.0 + 0.1 * torch.rand(top_k, generator=gen)
    rows.append(rows[4].clone())
    rows[6][vocab - 5:] = 9.0
    logits = torch.stack(rows)
    n = len(rows)
    ints = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    tokens, status = ints([-1] * n), ints([-1] * n)
    for step in range(3):
        K.sample(logits.to(DEV), 0.7, top_k, 5, ints(list(range(n))), ints([step] * n), tokens, status)
        assert status.cpu().tolist() == [0] * n
        for r in range(n):
            x = logits[r].double().numpy()
            kept = np.lexsort((np.arange(vocab), -x))[:top_k]
            w = np.exp((x[kept] - x[kept].max()) / 0.7)
            cdf = np.cumsum(w) / w.sum()
            at = np.nonzero(kept == int(tokens[r]))[0]
            assert len(at) == 1, (r, int(tokens[r]))
            u = float(pl.uniform_from_counter(5, r, step))
            slack = 64 * 2.0 ** -24  # float32 sums taken as a tree
            assert (cdf[at[0] - 1] if at[0] else 0.0) - slack <= u <= cdf[at[0]] + slack, (r, step)
