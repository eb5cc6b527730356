"""The rule that gives a GEMM its tile width, split and form (no GPU)."""
import random


def test_every_pick_is_legal(native_lib):
    rng = random.Random(5)
    for _ in range(2000):
        m, n, k = 128 * rng.randint(1, 256), 256 * rng.randint(1, 56), 8 * rng.randint(1, 1024)
        for g in (1, 2):
            ctas, gate_up = rng.choice([0, 1, 2, 20, 148]), rng.randint(0, 1)
            bn = native_lib.tcl_gemm_pick_tile(m, n, k, g, ctas, gate_up)
            assert 32 <= bn <= 256 and bn % 32 == 0 or bn == 512 and g == 2
            split = native_lib.tcl_gemm_pick_split(m, n, k, ctas)
            assert split in (1, 2, 4)
            if g == 1 and not gate_up and split > 1:       # the width that the split was picked with
                assert bn % (32 * split) == 0
                assert m // 128 * -(-n // bn) * split <= ctas       # one tile to a cluster, all side by side
                assert -(-k // 64) >= 4 * split
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


def test_splits_of_known_shapes(native_lib):
    pick, split = native_lib.tcl_gemm_pick_tile, native_lib.tcl_gemm_pick_split
    for shape, want in {(128, 8192, 3584): (2, 128), (128, 3584, 8192): (4, 128), (512, 1024, 8192): (4, 128), (256, 4096, 4096): (2, 128),
                        (128, 256, 1968): (4, 128), (256, 4096, 1024): (1, 128), (512, 768, 320): (1, 128), (384, 4096, 4096): (1, 128)}.items():
        assert (split(*shape, 148), pick(*shape, 1, 148, 0)) == want, shape
        assert split(*shape, 1) == 1
