"""What the benchmark reads from committed profiles belongs to the kernel that it times. No GPU is needed."""
import bench

HEADLINE = (4096, 7168, 2048)


def test_traffic_is_that_of_the_kernel_that_the_headline_shape_takes():
    name = "bs_gemm_dense_M{}_N{}_K{}.md".format(*HEADLINE)
    kernel = bench.dense_kernel(*HEADLINE, sms=148)
    M, N, K = HEADLINE
    traffic = bench.profile_traffic(name, kernel)
    assert 0.9 * (M * K + N * K) < traffic < 2 * (M * K + N * K + 2 * M * N)
    for other in {"bs_gemm_kernel", "bs_gemm_decode_kernel", "bs_pair_kernel"} - {kernel}:
        assert bench.profile_traffic(name, other) is None
    assert bench.profile_traffic("no_such_profile.md", kernel) is None
