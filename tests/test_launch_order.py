"""The order of the library's kernels on a stream.  They are launched behind the running kernel (programmatic stream
serialization) and wait for it on the device, so a call sees what the kernel before it wrote, whatever that kernel is and
whenever it lets its successors start."""
import ctypes as C
import re
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "ncnn-moe-runtime_b200" / "csrc"


def test_kernels_do_not_read_through_the_read_only_path():
    """ld.global.nc and __ldg are defined for data that nobody writes while the kernel runs.  The library's kernels may be
    resident while the kernel before them still writes their input."""
    for path in sorted(CSRC.iterdir()):
        code = re.sub(r"//[^\n]*", "", path.read_text())
        assert "ld.global.nc" not in code and "__ldg(" not in code and "__restrict__" not in code, path.name


def test_the_device_code_of_the_tests_compiles(test_kernels):
    assert hasattr(test_kernels, "test_produce_late")


def produce_late(test_kernels, torch, source, target, stream=None):
    """target = source on the stream, by a kernel that lets the next one start about 50 us before it writes."""
    handle = torch.cuda.current_stream().cuda_stream if stream is None else stream
    code = test_kernels.test_produce_late(C.c_void_p(handle), C.c_void_p(source.data_ptr()), C.c_void_p(target.data_ptr()),
                                          C.c_size_t(source.numel() * source.element_size() // 4), C.c_longlong(100000))
    assert code == 0


@pytest.mark.gpu
@pytest.mark.parametrize("stored", ["fp32", "bf16"])
@pytest.mark.parametrize("top_k", [0, 40])
def test_logits_of_a_producer_that_lets_the_sampler_start_early(pkg, torch_cuda, test_kernels, stored, top_k):
    torch = torch_cuda
    rows, vocab = 24, 50000
    dtype = torch.float32 if stored == "fp32" else torch.bfloat16
    generator = torch.Generator(device="cuda").manual_seed(top_k)
    versions = [(3.0 * torch.randn((rows, vocab), generator=generator, device="cuda")).to(dtype) for _ in range(4)]
    params = pkg.make_row_params(rows, seed=8, top_k=top_k, top_p=0.95)
    sampler = pkg.Sampler(max_rows=rows, max_vocab=vocab)
    try:
        want = []
        for logits in versions:
            want.append({k: v.clone() for k, v in sampler.sample_batch(logits, params).items() if v is not None})
        torch.cuda.synchronize()
        current = versions[0].clone()
        out = sampler.sample_batch(current, params)
        for version in (1, 2, 3, 0):
            produce_late(test_kernels, torch, versions[version], current)
            sampler.sample_batch(current, None, out=out)      # resident parameters: no copy between the two kernels
            torch.cuda.synchronize()
            assert torch.equal(current, versions[version])
            for name in ("token", "probability", "flags", "status"):
                assert torch.equal(out[name], want[version][name]), name
    finally:
        sampler.close()


@pytest.mark.gpu
def test_other_kernels_behind_a_producer_that_lets_them_start_early(pkg, torch_cuda, test_kernels, sampler):
    torch = torch_cuda
    generator = torch.Generator(device="cuda").manual_seed(3)

    def versions(*shape):
        return [torch.randn(shape, generator=generator, device="cuda") for _ in range(3)]

    def check(inputs, call):
        want = [[t.clone() for t in call(x)] for x in inputs]
        torch.cuda.synchronize()
        current = inputs[0].clone()
        call(current)
        for version in (1, 2, 0):
            produce_late(test_kernels, torch, inputs[version], current)
            got = call(current)
            torch.cuda.synchronize()
            for g, w in zip(got, want[version]):
                assert torch.equal(g, w)

    ids = torch.randint(64, (700,), generator=generator, device="cuda", dtype=torch.int32)
    check(versions(64, 2048), lambda x: [sampler.regroup_gather(x, ids)])
    check(versions(8, 50000), lambda x: sampler.indexer_topk(x, 1024, with_scores=True))
    check(versions(8, 40001), lambda x: [sampler.local_candidates(x, 128, 64)])
    for tokens in (32, 600):
        def dispatch(x):
            plan = sampler.router_dispatch(x, 4)
            return [plan.expert_offsets, plan.route_token, plan.route_rank, plan.route_weight, plan.status]
        check(versions(tokens, 96), dispatch)
