"""The rule that gives a GEMM its tile width (no GPU)."""
import random


def test_width_is_legal_and_never_estimated_slower(native_lib):
    rng = random.Random(5)
    for _ in range(500):
        m, n, k = 128 * rng.randint(1, 256), 256 * rng.randint(1, 56), 8 * rng.randint(1, 1024)
        for g in (1, 2):
            bn = native_lib.tcl_gemm_pick_tile(m, n, k, g, rng.choice([0, 1, 2, 20, 148]), rng.randint(0, 1))
            assert 32 <= bn <= 256 and bn % 32 == 0 or bn == 512 and g == 2
        assert native_lib.tcl_gemm_pick_form(m, n, k, 148) in (1, 2)


def test_widths_of_known_shapes(native_lib):
    pick = native_lib.tcl_gemm_pick_tile
    assert pick(8192, 8192, 8192, 2, 148, 0) == 512       # many waves, long K: two tiles share their rows of A
    assert pick(8192, 8192, 8192, 1, 148, 0) == 256
    assert pick(32768, 8192, 1024, 2, 148, 0) == 256      # short K: the epilogue would show
    assert pick(2048, 3584, 8192, 2, 148, 0) == 224       # 128 tiles in two waves instead of 112 in two
    assert pick(512, 7168, 8192, 2, 148, 0) == 224        # one wave either way
    assert pick(512, 7168, 8192, 2, 148, 1) == 256        # as gate|up, 112 features would take seven loads per k-block
    assert pick(128, 8192, 3584, 1, 148, 0) == 128        # 64 CTAs read the weight, not 32
    assert pick(4992, 4096, 4096, 2, 148, 0) == 256       # two waves; 192 columns fill the last one, at 161 us against 142
    form = native_lib.tcl_gemm_pick_form
    assert [form(*s, 148) for s in ((128, 8192, 3584), (512, 768, 320), (4992, 4096, 4096), (8192, 8192, 8192))] == [1, 1, 2, 2]
