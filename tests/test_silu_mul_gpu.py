"""Edges of the SiLU*mul kernel: chunk widths, partial blocks, alignment, the ends of the gate's range."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(out, gu):
    f = gu.shape[1] // 2
    g, u = gu[:, :f].double(), gu[:, f:].double()
    ref = g * torch.sigmoid(g) * u
    # half a bf16 step of the exact value (8 significant bits: spacing 2^-7 in [1, 2), so 2^-8 at most) and some fp32 steps; below 1e-37 bf16 itself has no relative accuracy
    assert ((out.double() - ref).abs() <= ref.abs() * 2.0 ** -8 * 1.01 + 1e-37).all()


@pytest.mark.parametrize("rows,ffn", [(1, 8), (1, 16), (3, 24), (16, 256), (33, 520), (511, 16), (7, 4104), (2049, 3584)])
@pytest.mark.parametrize("offset", [0, 8])          # 8 elements: 16-byte but not 32-byte aligned
def test_silu_mul_edges(native_lib, rows, ffn, offset):
    from tileccl_b200.ops import elementwise as ew
    torch.manual_seed(rows + ffn)
    store = torch.randn(rows * 2 * ffn + offset, device="cuda", dtype=torch.bfloat16)
    gu = store[offset:].view(rows, 2 * ffn)
    guard = torch.full((rows * ffn + 64,), 7.0, device="cuda", dtype=torch.bfloat16)
    out = ew.silu_mul(gu, guard[:rows * ffn].view(rows, ffn))
    _check(out, gu)
    assert (guard[rows * ffn:] == 7.0).all()


def test_silu_mul_every_gate_value(native_lib):
    from tileccl_b200.ops import elementwise as ew
    gate = torch.arange(65536, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16).view(128, 512)
    out = ew.silu_mul(torch.cat([gate, torch.ones_like(gate)], 1).contiguous())
    finite = torch.isfinite(gate)
    assert torch.equal(torch.isnan(out), torch.isnan(gate) | (gate == float("-inf")))
    assert (out[gate == float("inf")] == float("inf")).all()
    ref = gate.double() * torch.sigmoid(gate.double())
    err = (out.double() - ref).abs()
    # exp(-|g|) carries up to 2 + 1.2 |g| fp32 steps (its documented bound): far inside a bf16 half step.  From -87.4 down it is
    # subnormal and less precise, but these results are below 4e-36 times up = 1; a large up shows them, in the next test
    assert (err[finite] <= (ref.abs() * (2.0 ** -8 + 2.0 ** -16) + 2e-37)[finite]).all()


def test_silu_mul_gates_whose_exponential_is_subnormal(native_lib):
    from tileccl_b200.ops import elementwise as ew
    gate = torch.arange(-104, -80, 0.5, device="cuda").bfloat16().repeat(8, 2)[:, :96].contiguous()
    up = torch.full_like(gate, 1e36)
    out = ew.silu_mul(torch.cat([gate, up], 1).contiguous())
    g, u = gate.double(), up.double()
    ref = g * torch.sigmoid(g) * u
    # exp(-|g|) to its documented 2 + 1.173 |g| fp32 steps or to one subnormal quantum, its product with the gate to half a
    # quantum, and half a bf16 step
    tol = ref.abs() * (2.0 ** -8 * 1.01 + 130 * 2.0 ** -23) + (g.abs() + 0.5) * 2.0 ** -149 * u
    assert ((out.double() - ref).abs() <= tol).all()
    assert (out[gate > -100] != 0).all()


def test_silu_mul_rounds_like_a_correctly_rounded_divide(native_lib):
    """fp32 errors show in bf16 results where the exact value lies next to a midpoint.  A chain with a correctly rounded
    divide picks the wrong neighbour for 56 of these results, one with a divide of two fp32 steps for 228."""
    from tileccl_b200.ops import elementwise as ew
    gen = torch.Generator(device="cuda").manual_seed(0)
    gu = torch.empty(16384, 2 * 3584, device="cuda", dtype=torch.bfloat16).normal_(generator=gen)
    out = ew.silu_mul(gu)
    wrong = 0
    for rows in range(0, gu.shape[0], 2048):
        g, u = gu[rows:rows + 2048].double().split(3584, dim=1)
        wrong += int((out[rows:rows + 2048] != (g * torch.sigmoid(g) * u).bfloat16()).sum())
    assert wrong <= 100


def test_silu_mul_keeps_the_sign_of_zero(native_lib):
    from tileccl_b200.ops import elementwise as ew
    gate = torch.tensor([0.0, -0.0, -200.0, 0.0] * 4, device="cuda").bfloat16()
    up = torch.tensor([1.0, 1.0, 1.0, -1.0] * 4, device="cuda").bfloat16()
    out = ew.silu_mul(torch.cat([gate, up])[None])
    assert torch.equal(torch.signbit(out)[0], torch.tensor([False, True, True, True] * 4, device="cuda")) and (out == 0).all()
