"""fp32 rows without Top-K that a thread-block cluster finishes: every cluster size (the batch size chooses it), every
way a sum can end (in the head, inside a literal group, never), and the shapes the clusters leave to single CTAs.
Tokens and probability bits are compared with the oracle, so no tolerance applies."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(rng, vocab):
    normal = rng.standard_normal(vocab).astype(np.float32)
    spiked = 3.0 * normal
    spiked[rng.choice(vocab, 16, replace=False)] += rng.uniform(4.0, 12.0, 16)
    rows = [3.0 * normal, spiked, 2.0 * normal, 0.02 * normal]
    rows.append(rng.uniform(-6.0, 6.0, vocab))                          # flat histogram, long sums
    rows.append(-np.abs(3.0 * normal) - 50.0)                           # everything negative
    rows.append(1000.0 + 3.0 * normal)                                  # coarse logits: many exact ties
    rows.append(np.round(3.0 * normal * 4096.0) / 4096.0)               # quantised: ties, a few per group
    rows.append(np.round(3.0 * normal * 8.0) / 8.0)                     # thousands per value: left to single CTAs
    masked = 3.0 * normal
    masked[rng.random(vocab) < 0.5] = -np.inf
    rows.append(masked)
    return np.stack(rows).astype(np.float32)


@pytest.mark.parametrize("copies", [1, 2, 4, 9, 20])
@pytest.mark.parametrize("vocab", [40001, 151936])
def test_rows_finished_by_clusters(pkg, parity, copies, vocab):
    if copies == 20 and vocab == 151936:
        vocab = 65537
    rng = np.random.default_rng(1000 * copies + vocab)
    logits = np.concatenate([_rows(rng, vocab) for _ in range(copies)])
    if copies == 1:
        logits = logits[:3]
    count = logits.shape[0]
    params = pkg.make_row_params(count, seed=copies, top_k=0,
                                 temperature=rng.choice(np.array([0.6, 0.9, 1.0, 1.5, 3.0], dtype=np.float32), count),
                                 top_p=rng.choice(np.array([0.5, 0.85, 0.95, 0.999, 1.0], dtype=np.float32), count),
                                 min_p=rng.choice(np.array([0.0, 0.0, 1e-5, 0.001, 0.05], dtype=np.float32), count))
    for step in range(3):
        params["step"] = step
        parity.check(logits, params)
