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


class Captured:
    """The launches of `call` on a stream of its own as a graph: how many kernels, and another run of them."""

    def __init__(self, torch, call):
        from cuda.bindings import runtime
        self.runtime, self.torch, self.stream = runtime, torch, torch.cuda.Stream()
        self.check(runtime.cudaStreamBeginCapture(self.stream.cuda_stream, runtime.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal))
        try:
            call(self.stream.cuda_stream)
        finally:
            self.graph = self.check(runtime.cudaStreamEndCapture(self.stream.cuda_stream))
        count = self.check(runtime.cudaGraphGetNodes(self.graph, 0))[1]
        nodes = self.check(runtime.cudaGraphGetNodes(self.graph, count))[0]
        kinds = [self.check(runtime.cudaGraphNodeGetType(node)) for node in nodes]
        self.kernels = sum(kind == runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel for kind in kinds)
        self.nodes = len(kinds)
        self.executable = self.check(runtime.cudaGraphInstantiate(self.graph, 0))

    def check(self, result):
        assert int(result[0]) == 0, result[0]
        return result[1] if len(result) == 2 else result[1:]

    def run(self):
        self.check(self.runtime.cudaGraphLaunch(self.executable, self.stream.cuda_stream))
        self.torch.cuda.synchronize()

    def close(self):
        self.runtime.cudaGraphExecDestroy(self.executable)
        self.runtime.cudaGraphDestroy(self.graph)


@pytest.mark.gpu
@pytest.mark.parametrize("tokens,experts,top_k,launches", [(32, 128, 4, 1), (128, 1024, 16, 1), (129, 64, 4, 4), (4, 1025, 2, 4), (4, 64, 17, 4)])
def test_static_router_launches_what_it_needs(pkg, sampler, torch_cuda, tokens, experts, top_k, launches):
    """One launch for a few tokens; the three launches over the fixed scratch follow a reset of its counters."""
    torch = torch_cuda
    generator = torch.Generator(device="cuda").manual_seed(tokens)
    logits = torch.randn((tokens, experts), generator=generator, device="cuda")
    want = sampler.router_dispatch(logits, top_k)
    torch.cuda.synchronize()
    got = pkg.DispatchPlan(*[torch.empty_like(t) for t in (want.expert_offsets, want.route_token, want.route_rank, want.route_weight, want.status)])
    options = pkg.RouterOptions(experts, top_k, pkg.ROUTER_SOFTMAX, 1, 1.0, pkg.ROUTER_FLAG_NORMALIZE_TOPK, None, None)

    def dispatch(stream):
        message = C.create_string_buffer(256)
        pointers = [C.c_void_p(t.data_ptr()) for t in (logits, got.expert_offsets, got.route_token, got.route_rank, got.route_weight, got.status)]
        code = pkg.library().moe_router_dispatch_static(C.c_void_p(stream), pointers[0], tokens, C.byref(options), *pointers[1:], message, 256)
        assert code == 0, message.value

    dispatch(torch.cuda.current_stream().cuda_stream)   # the scratch's address is looked up
    torch.cuda.synchronize()
    captured = Captured(torch, dispatch)
    try:
        assert captured.nodes == captured.kernels == launches
        for _ in range(2):
            for t in (got.expert_offsets, got.route_token, got.route_rank):
                t.fill_(-1)
            torch.cuda.synchronize()
            captured.run()
            for g, w in zip((got.expert_offsets, got.route_token, got.route_rank, got.route_weight, got.status),
                            (want.expert_offsets, want.route_token, want.route_rank, want.route_weight, want.status)):
                assert torch.equal(g, w)
    finally:
        captured.close()
