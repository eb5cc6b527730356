"""Launches that overlap the end of the kernel before them: every read and write still happens in stream order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


FORMS = [dict(cta_group=1), dict(cta_group=1, tile_cols=64), dict(cta_group=1, tile_cols=128, split_k=2), dict(cta_group=1, tile_cols=128, split_k=4),
         dict(cta_group=2, tile_cols=256), dict(cta_group=2, tile_cols=96), dict(cta_group=2, tile_cols=512)]


@pytest.mark.parametrize("M", [128, 512])
@pytest.mark.parametrize("form", FORMS, ids=lambda f: "-".join(str(v) for v in f.values()))
def test_chains_of_dependent_calls(native_lib, M, form):
    """Each call reads what the one before it wrote, another kernel overwrites an input right after the call that
    read it, and results are read by another kernel right after the call that wrote them."""
    from tileccl_b200.ops.gemm import GemmPlan
    torch.manual_seed(M)
    K = 512
    form = dict(form, ragged_m=form["cta_group"] == 2 and M % 256 != 0)
    w = [torch.randn(K, K, device="cuda", dtype=torch.bfloat16) * K ** -0.5 for _ in range(2)]
    x0 = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)

    def chain(sync):
        x, y = x0.clone(), torch.empty_like(x0)
        there, back = GemmPlan(x, w[0], out=y, timeout_ms=1000, **form), GemmPlan(y, w[1], out=x, timeout_ms=1000, **form)
        seen = []
        for i in range(40):
            there()
            sync()
            back()                       # reads y, overwrites x, which the call before read
            sync()
            if i % 3 == 0:
                seen.append(x.clone())   # an ordinary kernel that reads the result
                x.mul_(0.5)              # and one that overwrites it ahead of the next call
                sync()
        torch.cuda.synchronize()
        there.check()
        back.check()
        return seen + [x]

    want = chain(torch.cuda.synchronize)
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            torch.cuda.synchronize()
            got = chain(lambda: None)
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("tokens,hidden,ffn", [(256, 512, 640), (768, 512, 1024)])
def test_chain_of_the_fused_pair(native_lib, tokens, hidden, ffn):
    """All-gather GEMM with the SiLU epilogue, then GEMM + reduce-scatter, its result copied into the next call's input:
    eager, and from a graph whose kernels count the calls themselves."""
    from tileccl_b200.models.tp_mlp import TpMlp
    from tileccl_b200.parallel.heap import SymmetricHeap
    torch.manual_seed(tokens)
    x0 = torch.randn(tokens, hidden, device="cuda", dtype=torch.bfloat16)
    heap = SymmetricHeap(64 << 20)
    try:
        eager, graph = (TpMlp(heap, tokens, hidden, ffn, seed=3, init_std=0.05, graph=g) for g in (False, True))
        graph.capture()

        def chain(call, block, sync):
            block.x_shard.copy_(x0)
            seen = []
            for _ in range(30):
                y = call()
                sync()
                seen.append(y.clone())
                # behind the call that reads it, ahead of the one that needs it; bounded, so that the feedback cannot grow
                block.x_shard.copy_(torch.tanh(y) + x0)
                sync()
            torch.cuda.synchronize()
            block.check()
            return torch.stack(seen)

        want = chain(eager, eager, torch.cuda.synchronize)
        assert torch.isfinite(want).all()
        assert torch.equal(chain(eager, eager, lambda: None), want)
        assert torch.equal(chain(graph.replay, graph, lambda: None), want)
    finally:
        heap.close()


@pytest.mark.parametrize("cta_group", [1, 2])
def test_capped_calls_leave_the_other_sms_alone(native_lib, cta_group):
    """Calls with a grid cap, back to back on one stream, hold no more SMs than the cap: a call on another stream that
    fits in the rest runs beside the first of them, it does not wait for the last."""
    from tileccl_b200.ops.gemm import GemmPlan
    cap = torch.cuda.get_device_properties(0).multi_processor_count // 4 * 2 - 2
    a, b = (torch.randn(4096, 8192, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    long = GemmPlan(a, b, cta_group=cta_group, num_ctas=cap, timeout_ms=1000)           # some 400 us a call
    short = GemmPlan(a[:1024, :1024], b[:1024, :1024], cta_group=cta_group, num_ctas=cap, timeout_ms=1000)
    streams = torch.cuda.Stream(), torch.cuda.Stream()
    for s, plan in zip(streams, (long, short)):
        s.wait_stream(torch.cuda.current_stream())
        plan(s)                                                                          # loaded and warm
    torch.cuda.synchronize()
    begun, ended, beside = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    under_way = torch.cuda.Event()
    calls = 10
    with torch.cuda.stream(streams[0]):
        begun.record()
        long()
        under_way.record()
        for _ in range(calls - 1):
            long()
        ended.record()
    with torch.cuda.stream(streams[1]):
        streams[1].wait_event(under_way)
        short()
        beside.record()
    torch.cuda.synchronize()
    long.check()
    short.check()
    # beside the second call: over before that one is.  Behind calls that hold SMs ahead of their turn it ends with the third.
    assert begun.elapsed_time(beside) < 2 * begun.elapsed_time(ended) / calls
