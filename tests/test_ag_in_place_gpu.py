"""torch.ops.tileccl.ag_gemm on one rank: which shards the GEMM reads where they are, and which are copied first."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["dense", "pitched", "transposed", "misaligned", "fp32", "result"])
def test_ag_gemm_takes_every_shard(native_lib, form):
    import tileccl_b200 as tc
    from tileccl_b200.ops import torch_ops
    torch.manual_seed(3)
    M, K = 384, 256
    w = torch.randn(K, K, device="cuda", dtype=torch.bfloat16) * 0.1        # N = K: a result can be the next input
    x = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    tc.init(64 << 20)
    try:
        first = torch.ops.tileccl.ag_gemm(x, w)
        a = {"dense": lambda: x,
             "pitched": lambda: torch.zeros(M, 2 * K, device="cuda", dtype=torch.bfloat16)[:, :K].copy_(x),
             "transposed": lambda: x.t().contiguous().t(),
             "misaligned": lambda: torch.zeros(M * K + 8, device="cuda", dtype=torch.bfloat16)[4:M * K + 4].view(M, K).copy_(x),
             "fp32": lambda: x.float(),
             "result": lambda: first}[form]()
        assert torch_ops._reads_in_place(1, a, K, first) == (form == "dense")
        want, amax = a.double() @ w.double().t(), float(a.abs().max())
        got = torch.ops.tileccl.ag_gemm(a, w)
        tc.check_all()
        # half a bf16 step, and K fp32 additions
        tol = want.abs() * 2.0 ** -8 + K * 2.0 ** -23 * amax * float(w.abs().max())
        assert ((got.double() - want).abs() <= tol).all()
    finally:
        tc.shutdown()
