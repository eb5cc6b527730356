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
    # exp(-|g|) carries up to 2 + 1.2 |g| fp32 steps (its documented bound), which stays inside a bf16 half step up to |g| = 100
    assert (err[finite] <= (ref.abs() * (2.0 ** -8 + 2.0 ** -16) + 2e-37)[finite]).all()
