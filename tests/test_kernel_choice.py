"""Which kernel serves a product of a few or of some tens of rows, by the shapes of the three model sizes (no GPU: the
choice is host arithmetic).  The figures behind the rules were measured on a B200, in a chain of the product alone
and then in the decode step."""
import pytest
import torch

from qwen_engine_b200 import ops

BF = torch.bfloat16
# (hidden, intermediate, q heads, kv heads) with head size 128
SIZES = {"0.6b": (1024, 3072, 16, 8), "1.7b": (2048, 6144, 16, 8), "4b": (2560, 9728, 32, 8)}


def _products(name):
    H, I, Hq, Hkv = SIZES[name]
    return {"qkv": ((Hq + 2 * Hkv) * 128, H), "o": (H, Hq * 128), "gate_up": (2 * I, H), "down": (H, I)}


@pytest.mark.parametrize("name", list(SIZES))
def test_up_to_eight_rows_stream_the_weights(name):
    """... but for the one product whose K is so long and whose weight rows are so awkward a number (2 560: 160 CTAs of
    16 rows for 148 SMs) that clusters sharing K are faster at any number of rows: Qwen3-4B's down projection."""
    for what, (N, K) in _products(name).items():
        for M in (1, 4, 8):
            assert ops.splitk_splits(M, N, K, BF) == (4 if (name, what) == ("4b", "down") else 0)


def test_nine_to_sixteen_rows_share_k_only_where_the_streaming_kernel_is_at_its_worst():
    for name in ("0.6b", "1.7b"):
        for N, K in _products(name).values():
            assert ops.splitk_splits(12, N, K, BF) == 0, (name, N, K)
    p = _products("4b")
    assert ops.splitk_splits(9, *p["o"], BF) == 4 and ops.splitk_splits(16, *p["down"], BF) == 4
    assert ops.splitk_splits(16, *p["qkv"], BF) == 0 and ops.splitk_splits(16, *p["gate_up"], BF) == 0


def test_some_tens_of_rows_share_k_in_clusters_that_find_room():
    # 1 024 weight rows: 8 clusters of 8 CTAs; 2 048 and 2 560: 16 and 20 clusters, of 4
    assert ops.splitk_splits(32, *_products("0.6b")["o"], BF) == 8 and ops.splitk_splits(64, *_products("0.6b")["down"], BF) == 8
    assert ops.splitk_splits(32, *_products("1.7b")["o"], BF) == 4 and ops.splitk_splits(32, *_products("1.7b")["down"], BF) == 4
    assert ops.splitk_splits(32, *_products("4b")["o"], BF) == 4
    # many weight rows: fewer CTAs a cluster, or none (the swapped kernel or the streaming one serves)
    assert ops.splitk_splits(32, *_products("0.6b")["qkv"], BF) == 4 and ops.splitk_splits(32, *_products("0.6b")["gate_up"], BF) == 2
    assert ops.splitk_splits(32, *_products("4b")["gate_up"], BF) == 0
    for s in (2, 4, 8):        # whatever is chosen fits the GPU at once and leaves every CTA two blocks of K at least
        for name in SIZES:
            for N, K in _products(name).values():
                got = ops.splitk_splits(40, N, K, BF)
                assert got == 0 or (-(-N // 128) * got <= ops.SPLITK_MAX_CTAS and -(-K // 64) >= 2 * got)


def test_other_types_and_many_rows_are_not_for_that_kernel():
    assert ops.splitk_splits(32, 1024, 2048, torch.float32) == 0
    assert ops.splitk_splits(65, 1024, 2048, BF) == 0
    assert ops.splitk_splits(32, 1024, 2052, BF) == 0          # K must be a multiple of 8


def test_very_many_weight_rows_go_64_to_a_cta():
    for K in (1024, 2048, 2560):
        assert all(ops.stream_applies(M, 151936, K, BF) for M in (1, 8, 16, 32)) and not ops.stream_applies(33, 151936, K, BF)
    assert not ops.stream_applies(8, 32768, 1024, BF) and ops.stream_applies(9, 32768, 1024, BF) and not ops.stream_applies(17, 32768, 1024, BF)
    assert not ops.stream_applies(8, 16384, 200, BF) and ops.stream_applies(9, 16384, 200, BF) and ops.stream_applies(8, 65536, 200, BF)
    assert not ops.stream_applies(8, 151936, 1024, torch.float32) and not ops.stream_applies(8, 151936, 1020, BF)
    assert not any(ops.stream_applies(M, N, K, BF) for M in (1, 16, 32) for name in ("0.6b", "1.7b") for N, K in _products(name).values())
    glu = lambda M, name: ops.swiglu_stream_applies(M, SIZES[name][1], SIZES[name][0], BF)
    assert all(glu(M, "4b") and glu(M, "1.7b") for M in (1, 8, 16, 17, 64)) and not glu(65, "4b")
    assert not glu(8, "0.6b") and not glu(16, "0.6b") and glu(17, "0.6b") and glu(64, "0.6b")
    assert not ops.swiglu_stream_applies(28, 3072, 4096, BF), "K too long for a CTA alone"


def test_rows_beyond_what_a_form_serves_are_refused():
    """64 weight rows a CTA: up to 32 rows as they are, up to 64 with the activation (refused before anything is launched)."""
    import ctypes
    at = ctypes.c_void_p(1 << 20)
    call = lambda M, form: ops.lib().qe_linear_tcgen05_swap(at, at, at, M, 128, 64, 0, form, 0, ctypes.c_void_p(0))
    for M, form, most in ((33, 1, b"32"), (64, 1, b"32"), (65, 2, b"64"), (257, 0, b"256")):
        assert call(M, form) == 1 and b"above " + most in ops.lib().qe_last_error()
    assert call(8, 3) == 1 and ops.STREAM_MAX_M == 32 and ops.STREAM_GLU_MAX_M == 64


def test_few_rows_share_k_where_the_streaming_kernel_takes_a_second_round_or_two_tiles_of_tokens():
    got = lambda M, N, K: ops.few_rows_splits(M, N, K, BF)
    assert got(9, 2432, 1536) == got(16, 4096, 4096) == 4 and got(9, 4096, 1024) == 0 and got(9, 2368, 2048) == 0
    assert got(9, 4736, 2048) == 0 and got(16, 6144, 2560) == 2 and got(16, 6144, 2048) == 0 and got(9, 7168, 1024) == 2
    assert got(8, 8192, 1536) == got(1, 6144, 4096) == 2 and got(8, 9216, 1024) == got(8, 5120, 4096) == got(8, 6144, 2560) == 0
    assert got(17, 6144, 2560) == got(8, 9600, 2560) == got(9, 12288, 2048) == 0          # (more than 74 clusters of 2)
    assert ops.few_rows_splits(9, 6144, 2560, torch.float32) == 0 and got(9, 6144, 2564) == 0 and got(9, 6146, 2560) == 0
    for M in (1, 8, 9, 16):
        for N in range(16, 20000, 52):
            for K in (512, 1024, 1536, 2048, 4096, 9728):
                s = got(M, N, K)
                assert s == 0 or (-(-N // 128) * s <= ops.SPLITK_MAX_CTAS and -(-K // 64) >= 2 * s)


def test_the_scan_of_a_long_prompt_stays_with_the_kernel_that_stages_ahead():
    """... alone and beside requests of few tokens, whatever their number of CTAs; prompts of like lengths, short ones, 256 key channels
    and more go through the ring of asynchronous copies."""
    def ring(lens, H=8, dk=64, dv=128, dtype=1):
        return bool(ops.lib().qe_linear_attention_scan_streams(len(lens), max(lens), sum(lens), H, dk, dv, dtype))
    assert ops._DT[BF] == 1 and ops._DT[torch.float32] == 0
    for dtype in (0, 1):
        for alone in ([2048], [512], [130]):
            assert not ring(alone, dtype=dtype)
        for beside in ([512] + [1] * 3, [2048] + [1] * 3, [2048] + [1] * 15, [1024, 64], [1000] + [30] * 8):
            assert not ring(beside, dtype=dtype)
        assert not ring([2048] + [1] * 3, H=16, dtype=dtype) and not ring([2048] + [1] * 15, H=16, dtype=dtype)
        assert not ring([2048] + [1] * 15, H=4, dk=128, dtype=dtype) and not ring([512] + [1] * 3, H=8, dk=128, dv=256, dtype=dtype)
        for many in ([256] * 8, [512, 512], [700, 500, 300], [1024, 200, 100], [512] + [1] * 63, [64] * 32, [9], [100], [128], [1, 2]):
            assert ring(many, dtype=dtype)
        assert ring([2048], H=2, dk=256, dv=64, dtype=dtype) and ring([512] + [1] * 15, H=1, dk=512, dv=64, dtype=dtype)
        assert not ring([1]) and not ring([1] * 64), "single tokens have a form of their own"
    assert ring([512] + [1] * 15, H=8, dk=128, dv=256) and not ring([512] + [1] * 15, H=8, dk=128, dv=256, dtype=0)
    assert not ring([9], dk=16, dtype=1) and ring([9], dk=16, dtype=0), "a thread's channels are not whole pieces"
    assert not ring([9], dk=72) and not ring([9], dv=132)
