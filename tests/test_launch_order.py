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
@pytest.mark.parametrize("tokens,experts,top_k,score,launches", [(32, 128, 4, 0, 1), (128, 768, 16, 0, 1), (128, 1024, 16, 0, 4), (129, 64, 4, 0, 4), (4, 1025, 2, 0, 4), (4, 64, 17, 0, 4),
                                                                 (128, 384, 8, 1, 1), (128, 385, 8, 1, 4), (128, 384, 8, 2, 1), (49, 1004, 8, 2, 4)])
def test_static_router_launches_what_it_needs(pkg, sampler, torch_cuda, tokens, experts, top_k, score, launches):
    """One launch for a few tokens; the three launches over the fixed scratch follow a reset of its counters."""
    torch = torch_cuda
    generator = torch.Generator(device="cuda").manual_seed(tokens)
    logits = torch.randn((tokens, experts), generator=generator, device="cuda")
    want = sampler.router_dispatch(logits, top_k, score_function=score)
    torch.cuda.synchronize()
    got = pkg.DispatchPlan(*[torch.empty_like(t) for t in (want.expert_offsets, want.route_token, want.route_rank, want.route_weight, want.status)])
    options = pkg.RouterOptions(experts, top_k, score, 1, 1.0, pkg.ROUTER_FLAG_NORMALIZE_TOPK, None, None)

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


class Calls:
    """One call of every device-buffer entry point with resident parameters, into outputs of its own: kernels per call, the call,
    and the tensors it writes."""

    def __init__(self, pkg, torch, overlap=False):
        generator = torch.Generator(device="cuda").manual_seed(11)

        def normal(*shape):
            return torch.randn(shape, generator=generator, device="cuda")

        self.handles = {}
        self.entries = {}

        def sampling(name, launches, logits, **options):
            rows, vocab = logits.shape
            handle = self.handles[name] = pkg.Sampler(max_rows=rows, max_vocab=vocab)
            handle.set_overlap(overlap)
            out = handle.sample_batch(logits, pkg.make_row_params(rows, seed=5, **options))
            self.entries[name] = (launches, lambda stream: handle.sample_batch(logits, None, stream=stream, out=out), [v for v in out.values() if v is not None])

        sampling("top_k", 1, 3.0 * normal(20, 60000), top_k=40, top_p=0.9)
        sampling("clusters", 3, 3.0 * normal(20, 60000), top_p=0.97)
        sampling("value_runs", 2, (3.0 * normal(20, 60000)).bfloat16(), top_p=0.97)
        rest = self.handles["rest"] = pkg.Sampler(max_rows=64, max_vocab=40000)
        rest.set_overlap(overlap)
        shard = normal(12, 40000)
        candidates = rest.local_candidates(shard, 1000, 32)
        merged = rest.merge_candidates(candidates.view(1, 12, 32), pkg.make_row_params(12, seed=6, top_k=32), 32)

        def shards(stream):
            rest.local_candidates(shard, 1000, 32, stream=stream, out=candidates)
            rest.merge_candidates(candidates.view(1, 12, 32), None, 32, stream=stream, out=merged)
        self.entries["shards"] = (2, shards, [candidates] + [v for v in merged.values() if v is not None])
        for tokens, launches in ((32, 1), (400, 3)):
            scores = normal(tokens, 96)
            plan = rest.router_dispatch(scores, 4)
            self.entries[f"router_{tokens}"] = (launches, lambda stream, scores=scores, plan=plan: rest.router_dispatch(scores, 4, stream=stream, out=plan),
                                                [plan.expert_offsets, plan.route_token, plan.route_rank, plan.route_weight, plan.status])
        hidden, ids = normal(64, 1536), torch.randint(64, (300,), generator=generator, device="cuda", dtype=torch.int32)
        gathered = torch.empty((300, 1536), device="cuda")
        library = pkg.library()

        def gather(stream):
            assert library.moe_regroup_gather(rest._handle, C.c_void_p(stream), C.c_void_p(hidden.data_ptr()), 64, 1536, C.c_void_p(ids.data_ptr()), 300,
                                              C.c_void_p(gathered.data_ptr())) == 0
        self.entries["gather"] = (1, gather, [gathered])
        history = normal(6, 30000)
        chosen = torch.empty((6, 512), dtype=torch.int32, device="cuda")

        def index(stream):
            assert library.moe_indexer_topk(rest._handle, C.c_void_p(stream), C.c_void_p(history.data_ptr()), 6, 30000, C.c_size_t(30000), 512,
                                            C.c_void_p(chosen.data_ptr()), None) == 0
        self.entries["indexer"] = (1, index, [chosen])
        torch.cuda.synchronize()
        self.torch = torch
        for _, call, _ in self.entries.values():
            call(torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        self.want = {name: [t.clone() for t in outputs] for name, (_, _, outputs) in self.entries.items()}
        self.clear()

    def clear(self):
        for _, _, outputs in self.entries.values():
            for t in outputs:
                t.fill_(0)
        self.torch.cuda.synchronize()

    def compare(self):
        self.torch.cuda.synchronize()
        for name, (_, _, outputs) in self.entries.items():
            for got, want in zip(outputs, self.want[name]):
                assert self.torch.equal(got, want), name
        self.clear()

    def close(self):
        for handle in self.handles.values():
            handle.close()


@pytest.mark.gpu
@pytest.mark.parametrize("overlap", [False, True])
def test_all_kernels_after_one_another_on_one_stream(pkg, torch_cuda, overlap):
    """Every kernel of the library behind every other, three times over and nothing waited for in between, on the default stream
    and on a stream of the caller's; the same with overlapping sampler launches (no input depends on an earlier call)."""
    torch = torch_cuda
    calls = Calls(pkg, torch, overlap)
    try:
        names = list(calls.entries)
        streams = [torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream(priority=-1)]
        for stream in streams:
            for shift in range(len(names)):
                for _ in range(3):
                    for i in range(len(names)):
                        calls.entries[names[(i * (shift + 1)) % len(names)]][1](stream.cuda_stream)
                for name in names:
                    calls.entries[name][1](stream.cuda_stream)
                calls.compare()
    finally:
        calls.close()


@pytest.mark.gpu
def test_every_call_can_be_captured(pkg, torch_cuda):
    """Each call with resident parameters becomes a graph of exactly its kernels, alone and all of them in one graph."""
    torch = torch_cuda
    calls = Calls(pkg, torch)
    graphs = []
    try:
        for name, (launches, call, _) in calls.entries.items():
            graphs.append(Captured(torch, call))
            assert (graphs[-1].nodes, graphs[-1].kernels) == (launches, launches), name
        for _ in range(2):
            for graph in graphs:
                graph.run()
            calls.compare()
        together = Captured(torch, lambda stream: [call(stream) for _, call, _ in calls.entries.values()])
        graphs.append(together)
        assert together.kernels == sum(launches for launches, _, _ in calls.entries.values())
        for _ in range(2):
            together.run()
            calls.compare()
    finally:
        for graph in graphs:
            graph.close()
        calls.close()


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 16, 64, 65, 200])
@pytest.mark.parametrize("overlap", [False, True])
def test_calls_with_and_without_rows_for_the_exact_kernels(pkg, torch_cuda, rows, overlap):
    """Batches that finish on chip, batches that do not and batches some of whose rows the clusters leave, one after the other
    and nothing waited for: the exact kernels of each find the list of their own call."""
    torch = torch_cuda
    vocab = 30011
    generator = torch.Generator(device="cuda").manual_seed(rows)
    peaked = 12.0 * torch.randn((rows, vocab), generator=generator, device="cuda")
    alive = 2.0 * torch.randn((rows, vocab), generator=generator, device="cuda")
    mixed = torch.where(torch.arange(rows, device="cuda")[:, None] % 3 == 0, peaked, alive)
    mixed[1::3] = mixed[1::3].bfloat16().float()          # left to the one-CTA kernel
    sampler = pkg.Sampler(max_rows=rows, max_vocab=vocab)
    try:
        params = pkg.make_row_params(rows, seed=4, temperature=0.8, top_p=0.97)
        kinds = (peaked, alive, mixed)
        want = []
        for logits in kinds:
            want.append(sampler.sample_batch(logits, params))
            torch.cuda.synchronize()
        sampler.set_overlap(overlap)
        order = [0, 0, 1, 0, 2, 2, 1, 1, 0, 2, 0, 1, 2, 0]
        got = [{k: torch.empty_like(v) if v is not None else None for k, v in want[0].items()} for _ in order]
        torch.cuda.synchronize()
        for kind, out in zip(order, got):
            sampler.sample_batch(kinds[kind], None, out=out)
        torch.cuda.synchronize()
        for kind, out in zip(order, got):
            for name in ("token", "probability", "flags", "status"):
                assert torch.equal(out[name], want[kind][name]), (kind, name)
    finally:
        sampler.close()
