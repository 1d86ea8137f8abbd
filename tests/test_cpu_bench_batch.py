"""The batched bench line names and counts the kernels that its sizes and its
autotuned configuration launch."""
import pytest


@pytest.mark.parametrize("sizes,threads,kernels", [
    ([32, 81, 512], 256, ["k_batch_big", "k_batch_qz"]),
    ([32, 80], 256, ["k_batch_qz"]),
    ([81, 512], 256, ["k_batch_big"]),
    ([32, 81, 512], 128, ["k_batch_qz"]),
])
def test_batch_kernels(sizes, threads, kernels):
    import bench
    assert bench.batch_kernels(sizes, threads) == kernels
