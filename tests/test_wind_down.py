"""A block whose wait gave up may not leave while a copy into its shared memory or an MMA on its tensor memory is under way.  A
wait that gives up there cannot be provoked without a fault, so the kernels' text is read: after its loop, the thread that
requests copies and the one that issues MMAs wait again (bounded) for what they have started, before the barrier behind which
tensor memory is freed, and so does an epilogue that gave up on its accumulator."""
import pytest

from test_cluster_order import kernel_body


@pytest.mark.parametrize("path,name,copies,mma", [
    ("gemm_tc.cu", "gemm_tc_kernel", "if (warp == 0)", "else if (warp == 1)"), ("gemm_smallm.cu", "gemm_smallm_kernel", "if (warp == 0)", "else if (warp == 1)"),
    ("gemm_wide.cu", "gemm_wide_kernel", "else if (warp == 0)", "else if (warp == 1)"),
    ("attn_prefill.cu", "attn_prefill_kernel", "else if (warp == 8)", "else if (warp == 9)")])
def test_blocks_wind_down(path, name, copies, mma):
    body = kernel_body("llm.cu_b200/csrc/" + path, name)
    role, rest = body[body.index(copies):body.index(mma)], body[body.index(mma):]
    after_copies = role[role.rindex("tma_load"):]
    assert "if (!ok)" in after_copies and ("drain_copies(" in after_copies or "mbar_wait(&k_full" in after_copies)
    assert rest.rindex("umma_f16") < rest.index("wind_down_mma(") < rest.rindex("__syncthreads()") < rest.index("tcgen05.dealloc")
    assert ", nullptr, 0)" in rest[rest.index("wind_down_mma("):]
