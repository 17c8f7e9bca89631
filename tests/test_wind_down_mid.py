"""gemm_mid_kernel winds down like the other tensor-core kernels (test_wind_down.py): either of its two copy warps waits for its copies,
the MMA warp for its MMAs, before the block's last barrier and before the tensor memory goes back."""
from test_cluster_order import kernel_body


def test_block_winds_down():
    body = kernel_body("llm.cu_b200/csrc/gemm_mid.cu", "gemm_mid_kernel")
    copies, mma = body.index("else if (warp == 0 || warp == 10)"), body.index("else if (warp == 1)")
    after_copies = body[body.rindex("tma_load", copies, mma):mma]
    assert "if (!ok && lane == 0) drain_copies(" in after_copies
    rest = body[mma:]
    assert rest.rindex("umma_f16") < rest.index("wind_down_mma(") < rest.rindex("__syncthreads()") < rest.index("tcgen05.dealloc")
