"""How the float32 product cuts K for the tensor cores (csrc/gemm_f32.cu), on the CPU."""
import ctypes


def test_pieces_of_k_are_three_stages_and_more():
    """The kernel hands the rows' maxima from its converting to its adding warps in two slots without a way back, which holds for items of three stages of 64."""
    from mini_inference_b200.ops import load_library
    pieces, length = load_library().mi_gemm_f32_pieces, ctypes.c_int()
    taken = 0
    for N in (128, 300, 600, 896, 1024, 1152, 1500, 2048, 2304, 2560, 4096, 6144, 19456, 151936):
        for K in [*range(512, 6200, 4), *range(9000, 10500, 4), 16384, 25600]:
            n = pieces(N, K, ctypes.byref(length))
            if n == 0:
                continue
            taken += 1
            last = K - (n - 1) * length.value
            assert length.value % 64 == 0 and 1 <= n <= 8 and (n == 1 or length.value >= 512)
            assert -(-last // 64) >= 3 and last <= length.value + 128, (N, K)
    assert taken > 15000
