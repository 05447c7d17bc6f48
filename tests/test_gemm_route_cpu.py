"""Which kernel a plain product takes below 1024 tokens, against what the two were measured to take (one B200, weights from HBM, slices as
dis_k_gemm_pick_split gives them; microseconds in one CTA per tile / in pairs of CTAs)."""
import pytest

from distributed_inference_server_b200 import binding as B

MEASURED = [  # N, K, T, slices, one CTA per tile, pairs
    (1024, 5120, 129, 16, 10.45, 11.38), (1024, 5120, 512, 9, 11.88, 12.47), (1024, 5120, 1000, 4, 15.96, 15.66),
    (4096, 1024, 200, 4, 9.99, 11.07), (4096, 1024, 400, 2, 11.33, 11.94), (4096, 1024, 640, 1, 13.30, 12.09),
    (2048, 2048, 200, 8, 9.91, 11.01), (2048, 2048, 512, 4, 11.27, 11.97), (1024, 4096, 129, 16, 9.86, 10.85),
    (512, 2048, 1000, 8, 9.69, 10.64), (512, 512, 1000, 2, 7.88, 8.24), (1024, 1024, 1000, 4, 9.56, 10.34),
    (6176, 1024, 640, 1, 15.30, 17.25), (6176, 1024, 1000, 1, 27.06, 17.48), (3072, 1024, 200, 4, 9.59, 8.88),
    (2560, 2048, 512, 3, 12.36, 11.79), (4096, 2048, 640, 1, 18.61, 16.26), (4096, 4096, 320, 3, 17.74, 20.49),
    (4096, 4096, 400, 2, 21.77, 20.70), (4096, 14336, 200, 4, 36.59, 31.49), (4096, 14336, 320, 3, 41.78, 48.24),
    (10240, 8192, 320, 1, 63.82, 72.22), (10240, 8192, 512, 1, 110.99, 73.73), (12288, 1024, 129, 1, 14.81, 12.47),
    (8192, 28672, 640, 1, 363.60, 255.68),
]


@pytest.mark.parametrize("N,K,T,split,single,pairs", MEASURED)
def test_the_faster_kernel_is_taken(N, K, T, split, single, pairs):
    lib = B.load()
    assert lib.dis_k_gemm_pick_split(T, N, K) == split
    taken = pairs if lib.dis_k_gemm_in_pairs(T, N, K, split) else single
    assert taken <= 1.03 * min(single, pairs)


@pytest.mark.parametrize("N,K", [(512, 512), (1024, 5120), (8192, 8192)])
def test_the_ends_of_the_range(N, K):
    lib = B.load()
    for T in (1, 128):
        assert lib.dis_k_gemm_in_pairs(T, N, K, 1) == 0
    for T in (1024, 5000):
        assert lib.dis_k_gemm_in_pairs(T, N, K, lib.dis_k_gemm_pick_split(T, N, K)) == 1
