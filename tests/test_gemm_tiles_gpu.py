"""Tile widths of the GEMM kernel: every width and both CTA forms give the bits of the 256-column tile."""
import pytest
import torch

pytestmark = pytest.mark.gpu

WIDTHS = [32, 64, 96, 128, 160, 192, 224]


def _operands(M, N, K, seed=0):
    torch.manual_seed(M + N + K + seed)
    return torch.randn(M, K, device="cuda", dtype=torch.bfloat16), torch.randn(N, K, device="cuda", dtype=torch.bfloat16) * 0.1


def _same_as_reference(out, A, Bt):
    ref = A.double() @ Bt.double().t()
    # half a bf16 step, and K fp32 additions of terms of at most max|a| max|b|
    tol = ref.abs() * 2.0 ** -8 + A.shape[1] * 2.0 ** -23 * float(A.abs().max()) * float(Bt.abs().max())
    assert ((out.double() - ref).abs() <= tol).all()


@pytest.mark.parametrize("cta_group", [1, 2])
@pytest.mark.parametrize("width", WIDTHS)
@pytest.mark.parametrize("store", ["st16", "st256"])
def test_every_width_gives_the_same_bits(native_lib, cta_group, width, store):
    from tileccl_b200.ops.gemm import GemmPlan
    A, Bt = _operands(768, 1792, 1000)             # a K remainder, and a last tile that hangs over N for most widths
    want = GemmPlan(A, Bt, cta_group=cta_group, tile_cols=256, timeout_ms=1000)
    _same_as_reference(want(), A, Bt)
    out = torch.full((769, 1792), 7.0, device="cuda", dtype=torch.bfloat16)
    plan = GemmPlan(A, Bt, out=out[:768], cta_group=cta_group, tile_cols=width, store=store, timeout_ms=1000, num_ctas=10)
    plan()
    plan.check()
    assert torch.equal(out[:768], want.out)
    assert (out[768] == 7.0).all()


@pytest.mark.parametrize("K", [64, 128, 256, 328, 512, 576, 1000])      # 1 to 16 k-blocks around the skew of 4
@pytest.mark.parametrize("N", [256, 512, 768, 1792])                     # with and without a last single half
@pytest.mark.parametrize("num_ctas", [2, 8, 10, 0])
def test_wide_tiles_give_the_same_bits(native_lib, K, N, num_ctas):
    from tileccl_b200.ops.gemm import GemmPlan
    A, Bt = _operands(1152, N, K)
    want = GemmPlan(A, Bt, cta_group=2, ragged_m=True, tile_cols=256, timeout_ms=1000)()
    _same_as_reference(want, A, Bt)
    out = torch.full((1153, N), 7.0, device="cuda", dtype=torch.bfloat16)
    plan = GemmPlan(A, Bt, out=out[:1152], cta_group=2, ragged_m=True, tile_cols=512, timeout_ms=1000, num_ctas=num_ctas)
    for _ in range(2):
        plan()
        plan.check()
    assert torch.equal(out[:1152], want)
    assert (out[1152] == 7.0).all()


@pytest.mark.parametrize("num_ctas", [2, 6, 0])
def test_wide_gate_up_tiles(native_lib, num_ctas):
    from tileccl_b200.ops.gemm import GemmPlan
    x, w = _operands(768, 2 * 896, 520)
    want = GemmPlan(x, w, cta_group=2, epi="silu_mul", tile_cols=256, timeout_ms=1000)()
    plan = GemmPlan(x, w, cta_group=2, epi="silu_mul", tile_cols=512, timeout_ms=1000, num_ctas=num_ctas)
    got = plan()
    plan.check()
    assert torch.equal(got, want)


@pytest.mark.parametrize("split,width", [(2, 64), (2, 192), (2, 256), (4, 128), (4, 256)])
@pytest.mark.parametrize("M,N,K", [(128, 256, 256), (256, 768, 328), (128, 1792, 1000), (384, 512, 8192)])
def test_split_k(native_lib, split, width, M, N, K):
    from tileccl_b200.ops.gemm import GemmPlan
    A, Bt = _operands(M, N, K)
    out = torch.full((M + 1, N), 7.0, device="cuda", dtype=torch.bfloat16)
    plan = GemmPlan(A, Bt, out=out[:M], cta_group=1, tile_cols=width, split_k=split, timeout_ms=1000)
    assert native_lib.tcl_gemm_plan_split(plan.handle) == split
    plan()
    plan.check()
    _same_as_reference(out[:M], A, Bt)
    assert (out[M] == 7.0).all()
    first = out.clone()
    for _ in range(3):
        plan()
    plan.check()
    assert torch.equal(out, first)


@pytest.mark.parametrize("M", [128, 512])
@pytest.mark.parametrize("N", [256, 1024, 2048])
def test_split_k_alone_finds_its_width(native_lib, M, N):
    """split_k without tile_cols: refused only where no width fits; and a plan has the width and split that the rule names."""
    from tileccl_b200.ops.gemm import GemmPlan
    A, Bt = _operands(M, N, 4096)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for split in (2, 4):
        assert M // 128 * -(-N // 256) * split <= sms
        plan = GemmPlan(A, Bt, cta_group=1, split_k=split, timeout_ms=1000)
        assert native_lib.tcl_gemm_plan_split(plan.handle) == split
        _same_as_reference(plan(), A, Bt)
        plan.check()
    plan = GemmPlan(A, Bt, cta_group=1)
    assert native_lib.tcl_gemm_plan_tile_cols(plan.handle) == native_lib.tcl_gemm_pick_tile(M, N, 4096, 1, sms, 0)
    assert native_lib.tcl_gemm_plan_split(plan.handle) == native_lib.tcl_gemm_pick_split(M, N, 4096, sms)


def test_split_k_refuses_what_it_cannot_do(native_lib):
    from tileccl_b200.ops.gemm import GemmPlan
    A, Bt = _operands(512, 8192, 256)
    for kw in (dict(cta_group=2, split_k=2), dict(cta_group=1, split_k=3), dict(cta_group=1, split_k=4, tile_cols=64),
               dict(cta_group=1, split_k=2, tile_cols=128), dict(cta_group=1, split_k=2, tile_cols=256, num_ctas=64),
               dict(cta_group=1, split_k=2, tile_cols=256, epi="silu_mul")):
        with pytest.raises(ValueError):
            GemmPlan(A, Bt, **kw)


@pytest.mark.parametrize("M", [128, 384, 1152])
@pytest.mark.parametrize("width", [32, 160, 256])
def test_pair_with_a_half_empty_last_tile(native_lib, M, width):
    from tileccl_b200.ops.gemm import GemmPlan
    A, Bt = _operands(M, 512, 328)
    with pytest.raises(ValueError):
        GemmPlan(A, Bt, cta_group=2)               # still refused unless asked for
    out = torch.full((M + 256, 512), 7.0, device="cuda", dtype=torch.bfloat16)
    plan = GemmPlan(A, Bt, out=out[:M], cta_group=2, ragged_m=True, tile_cols=width, timeout_ms=1000)
    plan()
    plan.check()
    _same_as_reference(out[:M], A, Bt)
    assert (out[M:] == 7.0).all()


@pytest.mark.parametrize("cta_group", [1, 2])
@pytest.mark.parametrize("width", WIDTHS)
def test_gate_up_tiles_of_every_width(native_lib, cta_group, width):
    from tileccl_b200.ops.gemm import GemmPlan
    x, w = _operands(512, 2 * 640, 328)            # 640 features: a remainder for most widths
    want = GemmPlan(x, w, cta_group=cta_group, epi="silu_mul", tile_cols=256, timeout_ms=1000)()
    plan = GemmPlan(x, w, cta_group=cta_group, epi="silu_mul", tile_cols=width, timeout_ms=1000, num_ctas=6)
    got = plan()
    plan.check()
    assert torch.equal(got, want)


@pytest.mark.parametrize("op", ["gemm", "gemm_rs", "ag_gemm"])
@pytest.mark.parametrize("shape", [(128, 256, 64), (128, 2048, 520), (384, 768, 72), (640, 256, 8192), (2176, 3584, 256)])
def test_ops_take_odd_multiples_of_128_rows(native_lib, op, shape):
    import tileccl_b200 as tc
    A, Bt = _operands(*shape)
    tc.init(128 << 20)
    try:
        _same_as_reference(getattr(torch.ops.tileccl, op)(A, Bt), A, Bt)
        tc.check_all()
    finally:
        tc.shutdown()


@pytest.mark.parametrize("cta_group", [1, 2])
def test_stores_of_the_epilogue_experiment_run_one_kernel_form(native_lib, cta_group):
    """At a shape whose default one-CTA plan splits K: with comm_form every store has the same tiles and the same bits."""
    from tileccl_b200.ops.gemm import GemmPlan
    A, Bt = _operands(512, 1024, 8192)
    if cta_group == 1:
        assert native_lib.tcl_gemm_plan_split(GemmPlan(A, Bt, cta_group=1).handle) > 1
    plans = [GemmPlan(A, Bt, cta_group=cta_group, store=s, comm_form=True, timeout_ms=1000) for s in ("st16", "st256", "tma")]
    for p in plans:
        assert (native_lib.tcl_gemm_plan_split(p.handle), native_lib.tcl_gemm_plan_tile_cols(p.handle)) == (1, 256)
        p()
        p.check()
        assert torch.equal(p.out, plans[0].out)
    _same_as_reference(plans[0].out, A, Bt)
    with pytest.raises(ValueError):
        GemmPlan(A, Bt, cta_group=cta_group, tile_cols=128, comm_form=True)
    with pytest.raises(ValueError):
        GemmPlan(A, Bt, cta_group=cta_group, split_k=2, comm_form=True)


@pytest.mark.parametrize("args,checks", [
    ("exp3_epilogue_remote --cta-group 1 --epi st16,st256,tma --sizes 512x1024x8192", 2),
    ("exp2_ag_gemm_granularity --cta-group 1 --m 512 --n 1024 --k 8192 --modes fused,ce --gather-rows 256,512", 4),
])
def test_experiments_verify_where_the_default_plan_splits_k(args, checks):
    import os
    import subprocess
    import sys
    module, *flags = args.split()
    r = subprocess.run([sys.executable, "-m", f"tileccl_b200.bench.{module}", *flags, "--verify", "--iters", "2", "--warmup", "1"],
                       capture_output=True, text=True, timeout=300, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert r.stdout.count("| ok") == checks and "FAIL" not in r.stdout, r.stdout


@pytest.mark.parametrize("cta_group", [1, 2])
def test_base_ctrl_and_fused_of_the_reduce_scatter_experiment_run_the_same_tiles(native_lib, cta_group):
    """Also on one rank, at a shape where a plan left to itself takes other tiles (one CTA: K split, pair: narrower)."""
    from tileccl_b200.ops.gemm import GemmPlan
    from tileccl_b200.ops.gemm_rs import GemmRs
    from tileccl_b200.parallel.heap import SymmetricHeap
    A, Bt = _operands(512, 1024, 8192)

    def form(handle):
        return native_lib.tcl_gemm_plan_split(handle), native_lib.tcl_gemm_plan_tile_cols(handle)

    assert form(GemmPlan(A, Bt, cta_group=cta_group).handle) != (1, 256)
    heap = SymmetricHeap(128 << 20)
    try:
        ops = [GemmRs(heap, A, Bt, cta_group=cta_group, comm_form=True, timeout_ms=1000, **kw) for kw in ({}, {"comm_enabled": False}, {"force_staged": True})]
        base = GemmPlan(A, Bt, cta_group=cta_group, comm_form=True, timeout_ms=1000)
        assert {form(base.handle), *(form(op.plan.handle) for op in ops)} == {(1, 256)}
        want = base()
        for op in (ops[0], ops[2]):          # ctrl leaves its result in the staging buffer
            assert torch.equal(op(), want)
            op.check()
    finally:
        heap.close()


@pytest.mark.parametrize("cta_group,K", [(1, 8192), (2, 512)])
def test_routed_outputs_take_the_form_measured_at_peers(native_lib, cta_group, K):
    from tileccl_b200.ops.gemm import GemmPlan
    A, Bt = _operands(512, 1024, K)
    parts = [torch.full((128 * cta_group, 1024), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(4 // cta_group)]
    plan = GemmPlan(A, Bt, cta_group=cta_group, seg_rows=128 * cta_group, dst_ptrs=[t.data_ptr() for t in parts], timeout_ms=1000)
    assert (native_lib.tcl_gemm_plan_split(plan.handle), native_lib.tcl_gemm_plan_tile_cols(plan.handle)) == (1, 256)
    plan()
    plan.check()
    _same_as_reference(torch.cat(parts), A, Bt)


@pytest.mark.parametrize("kw", [dict(cta_group=1, tile_cols=96), dict(cta_group=1, tile_cols=128, split_k=2), dict(cta_group=1, tile_cols=256, split_k=4),
                                dict(cta_group=2, tile_cols=160), dict(cta_group=2, tile_cols=512), dict(cta_group=2, tile_cols=512, num_ctas=6)])
@pytest.mark.parametrize("segments", [2, 4])
def test_row_segments_on_every_form(native_lib, kw, segments):
    """Segments routed to separate buffers in shuffled order, on the forms that find segment and row offset by themselves."""
    from tileccl_b200.ops.gemm import GemmPlan
    M, N = 1024, 768
    A, Bt = _operands(M, N, 1000)
    rows = M // segments
    parts = [torch.full((rows + 1, N), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(segments)]
    order = list(range(1, segments)) + [0]
    plan = GemmPlan(A, Bt, seg_rows=rows, dst_ptrs=[parts[i].data_ptr() for i in order], comm_form=False, timeout_ms=1000, **kw)
    plan()
    plan.check()
    _same_as_reference(torch.cat([parts[i][:rows] for i in order]), A, Bt)
    assert all((t[rows] == 7.0).all() for t in parts)
    # and through the row offsets of one output
    out = torch.full((M + 1, N), 7.0, device="cuda", dtype=torch.bfloat16)
    plan = GemmPlan(A, Bt, out=out[:M], seg_rows=rows, timeout_ms=1000, **kw)
    plan()
    plan.check()
    assert torch.equal(out[:M], torch.cat([parts[i][:rows] for i in order])) and (out[M] == 7.0).all()
