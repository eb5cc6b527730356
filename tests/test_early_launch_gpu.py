"""Launches that overlap the end of the kernel before them: every read and write still happens in stream order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [128, 512])
def test_chains_of_dependent_calls(native_lib, M):
    """Each call reads what the one before it wrote, another kernel overwrites an input right after the call that
    read it, and results are read by another kernel right after the call that wrote them."""
    from tileccl_b200.ops.gemm import GemmPlan
    torch.manual_seed(M)
    K = 512
    w = [torch.randn(K, K, device="cuda", dtype=torch.bfloat16) * K ** -0.5 for _ in range(2)]
    x0 = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)

    def chain(sync):
        x, y = x0.clone(), torch.empty_like(x0)
        there, back = GemmPlan(x, w[0], out=y, cta_group=1, timeout_ms=1000), GemmPlan(y, w[1], out=x, cta_group=1, timeout_ms=1000)
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
