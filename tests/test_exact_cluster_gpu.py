"""fp32 rows without Top-K that a thread-block cluster finishes: every cluster size (fixed, and chosen from the batch size),
every way a sum can end (in the head, inside a literal group, never), sums that are repeated, and the rows the clusters
leave to single CTAs.  A row that is left has the same result, so the tests also look at what the clusters counted.
Tokens and probability bits are compared with the oracle, so no tolerance applies."""
import ctypes as C

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


class Clusters:
    """The cluster size of a handle, and what its clusters have done since the last look."""

    def __init__(self, pkg, torch, sampler, size):
        self.library, self.torch, self.sampler = pkg.library(), torch, sampler
        assert self.library.moe_internal_set_cluster_ctas(sampler._handle, size) == 0

    def counts(self):
        words = (C.c_uint32 * 4)()
        assert self.library.moe_internal_cluster_counts(self.sampler._handle, C.c_void_p(self.torch.cuda.current_stream().cuda_stream), words) == 0
        return dict(zip(("rows", "left", "repeats", "refinements"), words))

    def __enter__(self):
        self.counts()
        return self

    def __exit__(self, *_):
        assert self.library.moe_internal_set_cluster_ctas(self.sampler._handle, 0) == 0


@pytest.mark.parametrize("size", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("vocab", [2600, 40001, 151936])
def test_ordinary_rows_are_finished_by_their_cluster(pkg, parity, torch_cuda, size, vocab):
    """Ordinary rows with whole vocabularies alive (top_p = 0.5: the bound is the end of a binade): none is left."""
    rng = np.random.default_rng(vocab)
    rows = []
    for _ in range(2):
        normal = rng.standard_normal(vocab).astype(np.float32)
        rows += [normal, 2.0 * normal, rng.uniform(-4.0, 4.0, vocab), 1000.0 + 3.0 * normal, -np.abs(normal) - 50.0]
    logits = np.stack(rows).astype(np.float32)
    params = pkg.make_row_params(len(rows), seed=size, top_k=0, temperature=3.0, top_p=np.array([0.5, 0.25, 0.95, 1.0, 0.999] * 2, dtype=np.float32))
    with Clusters(pkg, torch_cuda, parity.sampler, size) as clusters:
        for step in range(2):
            params["step"] = step
            parity.check(logits, params)
        counts = clusters.counts()
    assert counts["rows"] == 2 * len(rows) and counts["left"] == 0


@pytest.mark.parametrize("size", [1, 2, 4, 8, 16])
def test_sums_that_are_repeated(pkg, parity, torch_cuda, size):
    """top_p = 1: the nucleus sum ends within ulps of its bound, where groups are literal in large numbers (a guess is refined)
    and ties move the accumulator off the scanned one (the sum is repeated with the correction).  Both happen here."""
    rng = np.random.default_rng(2)
    vocab = 40001
    logits = np.stack([-np.abs(3.0 * rng.standard_normal(vocab)) - 50.0 for _ in range(16)] +
                      [-rng.exponential(2.0, vocab) for _ in range(16)]).astype(np.float32)
    params = pkg.make_row_params(len(logits), seed=3, top_k=0, top_p=1.0)
    with Clusters(pkg, torch_cuda, parity.sampler, size) as clusters:
        for step in range(2):
            params["step"] = step
            parity.check(logits, params)
        counts = clusters.counts()
    assert counts["rows"] + counts["left"] == 2 * len(logits) and counts["rows"] > len(logits)
    assert counts["repeats"] > 0 and counts["refinements"] > 0


@pytest.mark.parametrize("size", [1, 2, 4, 8, 16])
def test_rows_that_are_dense_at_the_top(pkg, parity, torch_cuda, size):
    """The head fills within the first four groups, before which there is no accumulator to guess an exponent from."""
    rng = np.random.default_rng(12)
    vocab = 120000
    logits = np.stack([-rng.exponential(scale, vocab) for scale in (1.5, 2.0, 3.0, 4.0)]).astype(np.float32)
    with Clusters(pkg, torch_cuda, parity.sampler, size) as clusters:
        for top_p in (0.9, 0.999):
            parity.check(logits, pkg.make_row_params(4, seed=size, top_k=0, top_p=top_p))
        counts = clusters.counts()
    assert counts["rows"] == 8 and counts["left"] == 0


@pytest.mark.parametrize("size", [1, 4, 16])
def test_rows_that_are_left(pkg, parity, torch_cuda, size):
    """Rows of bf16 values, rows with more equal logits than a group holds, and rows with a Top-K above the streaming limit
    are left to the one-CTA kernel; ordinary rows of the same batch are not."""
    rng = np.random.default_rng(9)
    vocab = 40001
    normal = (3.0 * rng.standard_normal((4, vocab))).astype(np.float32)
    widened = ((normal[1].view(np.uint32) >> 16) << 16).view(np.float32)
    filled = normal[2].copy()
    filled[-4000:] = np.float32(0.1)
    logits = np.stack([normal[0], widened, filled, normal[3]])
    params = pkg.make_row_params(4, seed=1, top_k=np.array([0, 0, 0, 1500], dtype=np.uint32), temperature=1.5, top_p=0.99)
    with Clusters(pkg, torch_cuda, parity.sampler, size) as clusters:
        parity.check(logits, params)
        counts = clusters.counts()
    assert counts["rows"] == 1 and counts["left"] == 3


@pytest.mark.parametrize("size", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("equal,most_left", [(119, 0), (121, 0), (255, 0), (257, 0), (1000, 5), (3000, 10), (3073, 20), (40000, 20)])
def test_equal_logits_share_a_group(pkg, parity, torch_cuda, size, equal, most_left):
    """Equal logits, as the padding of a vocabulary has them, wherever they lie: deep in the tail, where the bound or the draw may
    fall among them, and in the head.  A group takes as many as the list of literal items, the head 512 candidates."""
    rng = np.random.default_rng(equal)
    vocab = 50021
    rows = []
    for value in (-12.0, -6.0, 0.0, 3.0, 9.0):
        row = (3.0 * rng.standard_normal(vocab)).astype(np.float32)
        row[rng.choice(vocab, equal, replace=False)] = np.float32(value + 1.0 / 1024.0)
        rows.append(row)
    logits = np.stack(rows)
    with Clusters(pkg, torch_cuda, parity.sampler, size) as clusters:
        for top_p in (0.6, 0.9, 0.999, 1.0):
            params = pkg.make_row_params(len(rows), seed=equal + size, top_k=0, temperature=1.5, top_p=top_p, step=int(1000 * top_p))
            parity.check(logits, params)
        counts = clusters.counts()
    assert counts["rows"] + counts["left"] == 4 * len(rows)
    assert counts["left"] <= most_left
    if equal > 3072:
        assert counts["rows"] == 0


@pytest.mark.parametrize("size", [1, 2, 16])
def test_rows_of_odd_strides(pkg, parity, torch_cuda, size):
    """Rows that begin at every 16-byte phase: slices that are read by vectors and slices that are not."""
    rng = np.random.default_rng(6)
    vocab, rows = 20003, 8
    logits = (2.0 * rng.standard_normal((rows, vocab))).astype(np.float32)
    wide = torch_cuda.zeros((rows, vocab + 2), device="cuda")   # a stride of 20005 logits
    wide[:, :vocab] = torch_cuda.from_numpy(logits)
    params = pkg.make_row_params(rows, seed=5, top_k=0, temperature=2.0, top_p=0.98)
    with Clusters(pkg, torch_cuda, parity.sampler, size) as clusters:
        out = parity.sampler.sample_batch(wide, params, vocab=vocab)
        counts = clusters.counts()
    assert counts["rows"] == rows and counts["left"] == 0
    want = parity.checker.sample_batch(logits, params["temperature"], params["top_k"], params["top_p"], params["min_p"], parity.uniforms(params))
    np.testing.assert_array_equal(out["token"].cpu().numpy(), want["token"])


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


@pytest.mark.parametrize("stored", ["bf16", "widened"])
@pytest.mark.parametrize("vocab", [33000, 129280])
def test_rows_of_bf16_values_in_either_type(pkg, workloads, parity, stored, vocab):
    """Rows of bf16 values, stored as bf16 or widened to fp32 (the clusters leave those to the value-run path): both give
    the oracle's result, whatever the number of distinct values and the place where a sum ends."""
    rng = np.random.default_rng(vocab)
    rows = 40
    values = rng.standard_normal((rows, vocab)).astype(np.float32) * rng.choice(np.array([0.3, 1.0, 2.0, 3.0, 5.0], dtype=np.float32), (rows, 1))
    values[:10] += 8.0 * (rng.random((10, vocab)) < 0.0005)
    values[10:14] = np.round(values[10:14] * 4.0) / 4.0
    values[14:16] += 300.0
    bits = workloads.to_bf16_bits(values)
    logits = bits if stored == "bf16" else (bits.astype(np.uint32) << 16).view(np.float32)
    params = pkg.make_row_params(rows, seed=vocab, top_k=0, temperature=rng.choice(np.array([0.7, 1.0, 1.3, 2.0], dtype=np.float32), rows),
                                 top_p=rng.choice(np.array([0.6, 0.95, 1.0, 1.0], dtype=np.float32), rows),
                                 min_p=rng.choice(np.array([0.0, 0.0, 1e-4], dtype=np.float32), rows))
    for step in range(4):
        params["step"] = step
        parity.check(logits, params)


def test_infinities_and_nans(pkg, parity):
    """NaNs of any payload are skipped (one whose payload lies in the low half must not become an infinity in a row of
    bf16 values), -inf is never chosen, +inf anywhere is the reference's error; a peak that overflows in the division by
    the temperature gives an invalid distribution."""
    rng = np.random.default_rng(5)
    vocab = 40007
    plain = (3.0 * rng.standard_normal(vocab)).astype(np.float32)
    widened = ((plain.view(np.uint32) >> 16) << 16).view(np.float32)
    rows = []
    for base in (plain, widened):
        quiet = base.copy(); quiet[rng.choice(vocab, 300, replace=False)] = np.nan; rows.append(quiet)
        signalling = base.copy(); signalling.view(np.uint32)[rng.choice(vocab, 300, replace=False)] = 0x7F800001; rows.append(signalling)
        masked = base.copy(); masked[rng.random(vocab) < 0.3] = -np.inf; rows.append(masked)
        infinite = base.copy(); infinite[vocab - 1] = np.inf; rows.append(infinite)
        huge = base.copy(); huge[:] = np.float32(3.0e38) - np.abs(base) * np.float32(1.0e32); rows.append(huge)
    logits = np.stack(rows)
    for temperature in (1.0, 0.5):
        params = pkg.make_row_params(len(rows), seed=9, top_k=0, temperature=temperature, top_p=0.97)
        parity.check(logits, params)


@pytest.mark.parametrize("stored", ["fp32", "bf16"])
def test_scratch_of_the_first_batch_without_top_k(pkg, torch_cuda, stored):
    """The first batch with a row without Top-K allocates 16 bytes per vocabulary entry and slot, whatever its logits' type."""
    torch = torch_cuda
    rows, vocab = 148, 201088
    slots = min(rows, torch.cuda.get_device_properties(0).multi_processor_count)
    logits = (3.0 * torch.randn((1, vocab), device="cuda")).to(torch.float32 if stored == "fp32" else torch.bfloat16)
    warm = pkg.Sampler(max_rows=1, max_vocab=vocab)   # the kernels are loaded and have their stacks
    warm.sample_batch(logits, pkg.make_row_params(1, seed=1, top_k=0))
    torch.cuda.synchronize()
    warm.close()
    sampler = pkg.Sampler(max_rows=rows, max_vocab=vocab)
    try:
        out = sampler.sample_batch(logits, pkg.make_row_params(1, seed=1, top_k=50))
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        sampler.sample_batch(logits, pkg.make_row_params(1, seed=1, top_k=0), out=out)
        torch.cuda.synchronize()
        taken = before - torch.cuda.mem_get_info()[0]
        assert 16 * vocab * slots <= taken <= 16 * vocab * slots + (8 << 20)
    finally:
        sampler.close()


@pytest.mark.parametrize("vocab", [33, 4099, 20480])
def test_handle_no_larger_than_the_row(pkg, parity, torch_cuda, vocab):
    """Rows as long as the handle allows, every slot in use at once: neighbouring slots must not see each other's items."""
    rng = np.random.default_rng(vocab)
    rows = 160
    logits = rng.uniform(-6.0, 6.0, (rows, vocab)).astype(np.float32)
    params = pkg.make_row_params(rows, seed=4, top_k=0, temperature=rng.choice(np.array([1.0, 3.0], dtype=np.float32), rows), top_p=0.999)
    sampler = pkg.Sampler(max_rows=rows, max_vocab=vocab)
    try:
        out = sampler.sample_batch(torch_cuda.from_numpy(logits).cuda(), params)
        torch_cuda.cuda.synchronize()
        want = parity.checker.sample_batch(logits, params["temperature"], params["top_k"], params["top_p"], params["min_p"], parity.uniforms(params))
        np.testing.assert_array_equal(out["token"].cpu().numpy(), want["token"])
    finally:
        sampler.close()


def _compare_divisions(test_kernels, seed, a_exponents, b_exponents):
    mismatches, largest = C.c_ulonglong(), C.c_float()
    code = test_kernels.test_compare_divisions(C.c_uint64(seed), C.c_uint32(1184), C.c_uint32(1024), *[C.c_int(e) for e in (*a_exponents, *b_exponents)],
                                               C.byref(mismatches), C.byref(largest))
    assert code == 0
    return mismatches.value, largest.value


@pytest.mark.parametrize("a_exponents,b_exponents", [((-27, 0), (0, 17)), ((-45, 0), (-18, 0)), ((-100, 1), (-24, 24)), ((-100, -90), (20, 24))])
def test_division_by_a_reciprocal(torch_cuda, test_kernels, a_exponents, b_exponents):
    """The item passes divide by the two normalisers with a reciprocal and two corrections: every quotient of seeded pairs (a
    quarter of the mantissas next to a power of two or to the middle) is the division's, over the operands of ordinary rows (the
    first two) and over the whole range the function is stated for."""
    assert _compare_divisions(test_kernels, 1 - a_exponents[0], a_exponents, b_exponents)[0] == 0


def test_division_of_numerators_below_the_range(torch_cuda, test_kernels):
    """Numerators below 2^-100, zero and denormal ones among them, give finite quotients below 2^-70: no step in any accumulator."""
    _, largest = _compare_divisions(test_kernels, 5, (-127, -101), (-24, 24))
    assert largest < 2.0 ** -70


def test_peaks_far_above_the_temperature(pkg, parity):
    """A peak of 1e6 to 1e8 temperatures: the logits lie on a coarse grid, the live window is wider and holds numerators that
    are tiny or zero."""
    rng = np.random.default_rng(17)
    vocab = 60001
    rows = []
    for scale in (1.0e6, 1.0e7, 1.0e8):
        base = np.float32(scale)
        rows.append(base - np.abs(rng.standard_normal(vocab)).astype(np.float32) * np.float32(40.0 + scale * 2.0e-6))
        rows.append(base - rng.uniform(0.0, 3.0e-6 * scale, vocab).astype(np.float32))
    logits = np.stack(rows).astype(np.float32)
    for temperature, min_p in ((1.0, 0.0), (4.0, 1e-30), (0.5, 1e-4)):
        params = pkg.make_row_params(len(rows), seed=6, top_k=0, temperature=temperature, top_p=0.9999, min_p=min_p)
        for step in range(2):
            params["step"] = step
            parity.check(logits, params)
