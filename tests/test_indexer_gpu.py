"""GPU parity of moe_indexer_topk against the CPU oracle's statement of the latent-attention indexer selection
(src/kernels/cpu_latent_attention.cpp:414-423 of the reference: std::partial_sort with scored_index_precedes).

Bar: the selected index lists equal the oracle's, position by position (integer work: bit-exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(sampler, checker, torch, scores, top_k, count=None):
    rows, stride = scores.shape
    count = stride if count is None else count
    device = torch.from_numpy(scores).cuda()
    indices, values = sampler.indexer_topk(device, top_k, count=count, with_scores=True)
    torch.cuda.synchronize()
    indices = indices.cpu().numpy()
    values = values.cpu().numpy()
    selected = min(top_k, count)
    for r in range(rows):
        want = checker.indexer_topk(scores[r, :count], top_k)
        np.testing.assert_array_equal(indices[r, :selected].view(np.uint32), want, err_msg=f"row {r}")
        np.testing.assert_array_equal(values[r, :selected].view(np.uint32), scores[r, want].view(np.uint32))
        assert np.all(indices[r, selected:] == -1)


def test_reference_shaped_scores(sampler, checker, torch_cuda):
    # the scores of select_compressed_indices are sums of relu(dot) * weight: many exact zeros, a few large values
    rng = np.random.default_rng(41)
    for count, top_k in ((513, 512), (4096, 512), (40000, 2048), (131072, 2048), (9000, 8192)):
        scores = np.maximum(0.0, rng.standard_normal((3, count))).astype(np.float32) * rng.random((3, count)).astype(np.float32)
        check(sampler, checker, torch_cuda, scores, top_k)


def test_ties_small_and_ragged(sampler, checker, torch_cuda):
    rng = np.random.default_rng(42)
    for count, top_k in ((1, 1), (2, 1), (7, 7), (33, 5), (100, 64), (1000, 1), (257, 300), (5000, 4095)):
        scores = (np.round(rng.standard_normal((4, count)) * 2) / 2).astype(np.float32)     # coarse grid: the selection cuts through ties
        scores[0] = 1.0                                                                        # one row all equal: lowest indices win
        scores[1, ::3] = -0.0                                                                  # -0 == +0 in the comparator
        check(sampler, checker, torch_cuda, scores, top_k)
    # a strided view: only the first `count` entries of every row take part
    padded = rng.standard_normal((5, 3000)).astype(np.float32)
    check(sampler, checker, torch_cuda, padded, 128, count=2500)


def test_limits(sampler, pkg, torch_cuda):
    torch = torch_cuda
    scores = torch.zeros((1, 10), device="cuda")
    with pytest.raises(pkg.MoeError):
        sampler.indexer_topk(scores, 0)
    with pytest.raises(pkg.MoeError):
        sampler.indexer_topk(scores, 8193)
    indices = sampler.indexer_topk(scores, 16)          # more than there are entries
    torch.cuda.synchronize()
    assert indices.cpu().numpy()[0].tolist() == list(range(10)) + [-1] * 6


@pytest.mark.parametrize("count,top_k", [(1025, 1024), (2049, 2047), (5000, 2500), (10001, 5000), (40448, 512), (40449, 2048), (50001, 8192)])
def test_boundaries_of_the_selection(sampler, checker, torch_cuda, count, top_k):
    """Every way the k-th key can be found (few keys share its leading digit, only zeros do, many equal or nearly equal
    ones do) and every way the selection is put in order (buckets, the network for piled-up keys), at the sizes where
    the row stops fitting shared memory and the lists change their length; rows of every 16-byte phase."""
    rng = np.random.default_rng(count)
    rows = np.empty((9, count + 3), dtype=np.float32)                                   # odd stride: every phase
    normal = rng.standard_normal((9, count + 3)).astype(np.float32)
    rows[0] = normal[0]
    rows[1] = np.maximum(normal[1], 0.0)                                                # half zeros
    rows[2] = np.where(rng.random(count + 3) < 0.02, normal[2], 0.0)                    # the boundary lies among the zeros
    rows[3] = np.where(normal[3] > 0.0, normal[3] * 1e-41, 0.0)                         # denormals share the zeros' digit
    rows[4] = np.round(normal[4] * 2.0) / 2.0                                           # a few values
    rows[5] = 1.0 + 1e-6 * normal[5]                                                    # nearly equal: the later digits decide
    rows[6] = np.where(rng.random(count + 3) < 0.5, -0.0, -np.abs(normal[6]))           # zeros on top, negative rest
    rows[7] = 7.25                                                                      # all equal
    rows[8] = normal[8]
    rows[8, rng.choice(count, 40, replace=False)] = np.inf
    rows[8, rng.choice(count, 40, replace=False)] = -np.inf
    check(sampler, checker, torch_cuda, rows, top_k, count=count)


@pytest.mark.parametrize("count", [1, 2, 31, 32, 33, 63, 64, 65, 127, 129, 255, 257, 511, 513, 1023, 1024])
@pytest.mark.parametrize("top_k", [1, 32, 100, 1024, 2000])
def test_short_rows(sampler, checker, torch_cuda, count, top_k):
    """Rows of one record per thread, around every number of threads: all of the row is put in order."""
    rng = np.random.default_rng(count)
    rows = np.empty((6, count + 1), dtype=np.float32)
    normal = rng.standard_normal((6, count + 1)).astype(np.float32)
    rows[0] = normal[0]
    rows[1] = np.maximum(normal[1], 0.0)
    rows[2] = np.round(normal[2] * 2.0) / 2.0
    rows[3] = np.where(normal[3] > 0.0, normal[3] * 1e-41, -0.0)
    rows[4] = 7.25
    rows[5] = normal[5]
    rows[5, rng.integers(count)] = np.inf
    rows[5, rng.integers(count)] = -np.inf
    check(sampler, checker, torch_cuda, rows, top_k, count=count)


@pytest.mark.parametrize("count,top_k", [(1025, 64), (2049, 1024), (2300, 2048), (9001, 2048), (11264, 512), (11265, 512), (11264, 2048), (3000, 3000)])
def test_more_rows_than_sms(sampler, checker, torch_cuda, count, top_k):
    """Two CTAs share an SM while the row and the lists of both fit (11264 scores), one takes it otherwise."""
    rng = np.random.default_rng(count)
    rows = rng.standard_normal((320, count)).astype(np.float32)
    rows[1::4] = np.maximum(rows[1::4], 0.0)
    rows[2::4] = np.round(rows[2::4] * 4.0) / 4.0
    rows[3::4] = 1.0 + 1e-6 * rows[3::4]
    check(sampler, checker, torch_cuda, rows, top_k)
