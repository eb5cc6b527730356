"""``torch.ops.tileccl.*``: the thin PyTorch op layer.

    import tileccl_b200 as tc
    tc.init(heap_bytes=4 << 30)                      # once per process, after torch.distributed is up
    y_shard = torch.ops.tileccl.gemm_rs(a, w_t)      # a [M, K/tp], w_t [N, K/tp]  ->  [M/tp, N]
    y       = torch.ops.tileccl.ag_gemm(x_shard, w_t)  # x_shard [M/tp, K], w_t [N/tp, K]  ->  [M, N/tp]
    c       = torch.ops.tileccl.gemm(a, b_t)         # plain tcgen05 GEMM, a @ b_t.T
    h       = torch.ops.tileccl.silu_mul(gate_up)
    torch.ops.tileccl.barrier()                      # device barrier over all ranks, on the current stream

Plans (tensor maps, staging buffers, counters) are built on first use for a given operand *layout* (shapes,
row pitches) and are cached; the operands' addresses are not part of the key.  Every call launches the cached
plan on the tensors it was given (a host-side encoding of two tensor maps) and keeps no reference to them,
so a loop that allocates fresh activations every step reuses one plan and one set of staging buffers, and
every rank builds the same plans in the same order whatever addresses its allocator hands out.  Results live
in buffers owned by the cached plan: a result is valid until the next call with operands of the same layout.
Across ranks the AG shard must be peer-visible: it is copied into the plan's slot of the symmetric heap when
it is not already there.  On one rank it is read where it is, if TMA can (dense bf16 on a 16-byte boundary, not
overlapping the result).  Building a fused plan allocates from the symmetric heap and is collective: all
ranks must make the same sequence of first calls.

A plan repeats its bits exactly, call after call.  On one rank they may depend on the number of rows: problems with few
tiles split K over two or four CTAs, which add their fp32 partial sums in a fixed order, but another one than an unsplit
plan (N = K = 4096: M = 128 and 256 split, M = 384 does not).  ``GemmPlan(..., split_k=1)`` and all plans in the pair form
(``cta_group=2``) add every row's products in the same order whatever M, N and the tile width are.

The reference stops at C++ programs; this layer is what the north star adds.
"""
from __future__ import annotations

import torch

from .. import _native
from ..parallel.heap import SymmetricHeap
from . import elementwise as ew
from .ag_gemm import AgGemm
from .gemm import GemmPlan
from .gemm_rs import GemmRs

_ctx: dict = {"heap": None, "plans": {}, "barrier": None, "cta_group": 2}


def init(heap_bytes: int = 2 << 30, backend: str = "ipc", multicast: bool = False, cta_group: int = 2) -> SymmetricHeap:
    """Creates the process-wide symmetric heap (collective: every rank calls it with the same size)."""
    if _ctx["heap"] is None:
        _ctx["heap"] = SymmetricHeap(heap_bytes, backend=backend, multicast=multicast)
        _ctx["cta_group"] = cta_group
    return _ctx["heap"]


def heap() -> SymmetricHeap:
    if _ctx["heap"] is None:
        raise RuntimeError("call tileccl_b200.init(heap_bytes) first (collectively on every rank)")
    return _ctx["heap"]


def shutdown() -> None:
    _ctx["plans"].clear()
    _ctx["barrier"] = None
    if _ctx["heap"] is not None:
        _ctx["heap"].close()
        _ctx["heap"] = None


def symm_empty(shape, dtype=torch.bfloat16) -> torch.Tensor:
    """A tensor in the symmetric heap (same offset on every rank; collective)."""
    return heap().empty(shape, dtype)


def _key(kind, *tensors, extra=()):
    """Cache key: the operands' layout and device only (never their addresses)."""
    return (kind, extra, *((t.shape, t.stride(), t.dtype, t.get_device()) for t in tensors))


def check_all() -> None:
    """Synchronises and raises if any cached plan recorded a time-out."""
    for p in _ctx["plans"].values():
        p.check() if hasattr(p, "check") else None


_lib = torch.library.Library("tileccl", "DEF")
_lib.define("gemm(Tensor a, Tensor b_t) -> Tensor")
_lib.define("gemm_rs(Tensor a, Tensor b_t) -> Tensor")
_lib.define("ag_gemm(Tensor a_shard, Tensor b_t, int gather_rows=512) -> Tensor")
_lib.define("silu_mul(Tensor gate_up) -> Tensor")
_lib.define("barrier() -> ()")


def _form(m: int, b_t: torch.Tensor, world: int) -> dict:
    """CTA form of a plan whose rank holds ``m`` rows.  One rank: whichever is estimated to be faster, the pair
    also for an odd multiple of 128 rows (last tile half empty).  Several: the pair where its 256-row tiles fit.
    Operands that no form takes are left to the plan, which says what is wrong with them."""
    if _ctx["cta_group"] != 2 or m % 128 or b_t.dim() != 2:
        return {"cta_group": 1}
    if world > 1:
        return {"cta_group": 2 if m % 256 == 0 else 1}
    sms = torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
    if _native.lib().tcl_gemm_pick_form(m, *b_t.shape, sms) == 1:
        return {"cta_group": 1}
    return {"cta_group": 2, "ragged_m": m % 256 != 0}


def _gemm(a: torch.Tensor, b_t: torch.Tensor) -> torch.Tensor:
    k = _key("gemm", a, b_t)
    plan = _ctx["plans"].get(k)
    if plan is None:
        plan = _ctx["plans"][k] = GemmPlan(a, b_t, hold_operands=False, **_form(a.shape[0], b_t, world=1))
        return plan()
    plan.run_on(a.data_ptr(), b_t.data_ptr())       # the key has checked everything but the addresses
    return plan.out


def _gemm_rs(a: torch.Tensor, b_t: torch.Tensor) -> torch.Tensor:
    k = _key("gemm_rs", a, b_t)
    op = _ctx["plans"].get(k)
    if op is None:
        h = heap()
        op = _ctx["plans"][k] = GemmRs(h, a, b_t, hold_operands=False, **_form(a.shape[0] // h.world, b_t, world=h.world))
        return op()
    op.plan.run_on(a.data_ptr(), b_t.data_ptr())
    return op.out


def _reads_in_place(world: int, a: torch.Tensor, k: int, out: torch.Tensor) -> bool:
    """On one rank nobody else reads the shard, so the GEMM can take it where it is, if TMA can: the plan's dense bf16
    rows on a 16-byte boundary.  Not when it overlaps the result (the result of a call may be the next one's input).
    The copy it saves cost 12 us of 119 for 2048 x 8192."""
    if world != 1 or a.dtype != torch.bfloat16 or a.stride() != (k, 1) or a.get_device() != out.get_device():
        return False
    ptr, o = a.data_ptr(), out.data_ptr()
    return ptr % 16 == 0 and (ptr + a.numel() * 2 <= o or o + out.numel() * 2 <= ptr)


def _ag_gemm(a_shard: torch.Tensor, b_t: torch.Tensor, gather_rows: int = 512) -> torch.Tensor:
    h = heap()
    M, K = a_shard.shape[0] * h.world, a_shard.shape[1]
    k = _key("ag_gemm", b_t, extra=(M, K, gather_rows))
    op = _ctx["plans"].get(k)
    if op is None:
        op = _ctx["plans"][k] = AgGemm(h, M, K, b_t, gather_rows=gather_rows, hold_operands=False, **_form(a_shard.shape[0], b_t, world=h.world))
    a_ptr = a_shard.data_ptr()
    if a_ptr != op.a_shard.data_ptr():
        if not _reads_in_place(h.world, a_shard, K, op.out):
            op.a_shard.copy_(a_shard)
            a_ptr = op.a_full.data_ptr()
    else:
        a_ptr = op.a_full.data_ptr()
    op.plan.run_on(a_ptr, b_t.data_ptr())
    return op.out


def _barrier() -> None:
    if _ctx["barrier"] is None:
        _ctx["barrier"] = ew.DeviceBarrier(heap())
    _ctx["barrier"]()


_lib.impl("gemm", _gemm, "CUDA")
_lib.impl("gemm_rs", _gemm_rs, "CUDA")
_lib.impl("ag_gemm", _ag_gemm, "CUDA")
_lib.impl("silu_mul", lambda gu: ew.silu_mul(gu), "CUDA")
_lib.impl("barrier", _barrier, "CompositeExplicitAutograd")
