"""The split length of the batched attention is the caller's where a caller has set one, also for short sequences; only the engine's own
choice keeps sequences of up to 256 rows in one piece.  Seen through the per-CTA stamps (2 = first tile landed): as many CTAs have
one as there are shares of Q tiles, Q as in test_attn_partition.py, times KV heads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def working_ctas(pkg, launch):
    stamps = torch.zeros(148 * 32 * 8, dtype=torch.int64, device="cuda")  # no more than 32 CTAs reside on an SM
    pkg.lib.llmb_attn_decode_trace(stamps.data_ptr())
    launch()
    torch.cuda.synchronize()
    pkg.lib.llmb_attn_decode_trace(None)
    return int((stamps.view(-1, 8)[:, 2] != 0).sum())


@pytest.mark.parametrize("rows,split_len,shares", [(200, 32, 8), (200, 64, 8), (200, 128, 4), (200, 256, 2), (256, 128, 4), (65, 64, 4), (64, 64, 2), (257, 128, 5)])
def test_entry_point(pkg, rows, split_len, shares):
    nq, nkv, hd, n_splits = 32, 8, 128, -(-rows // split_len)
    q = torch.randn(2, nq * hd, device="cuda").half()
    k, v = (torch.randn(2, rows, nkv * hd, device="cuda").half() for _ in range(2))
    pos = torch.full((2,), rows - 1, dtype=torch.int32, device="cuda")
    out = torch.zeros(2, nq * hd, dtype=torch.float16, device="cuda")
    scratch = torch.zeros(pkg.lib.llmb_attn_decode_batch_scratch_bytes(2, nq, nkv, hd, n_splits), dtype=torch.uint8, device="cuda")

    def launch():
        assert pkg.lib.llmb_attn_decode_batch(q.data_ptr(), k.data_ptr(), v.data_ptr(), pos.data_ptr(), 2, rows, nq, nkv, hd, n_splits, split_len,
                                              out.data_ptr(), scratch.data_ptr(), 0, None) == 0
    assert working_ctas(pkg, launch) == shares * nkv


@pytest.mark.parametrize("split_len,shares", [(None, 2), (64, 8), (128, 4), (256, 2)])
def test_engine(pkg, oracle, split_len, shares):
    cfg = pkg.CONFIGS["tiny"]
    model = pkg.Model.synthetic(cfg, seed=0, max_seq=256)
    cache = pkg.Cache(model)
    cache.batch_init(2)
    if split_len:
        cache.batch_set_split_len(split_len)
    cache.set_options(use_graph=0)  # the stamps' address travels with the launch
    cache.batch_prefill(np.stack([oracle.synth_tokens(b, 200, cfg.vocab) for b in range(2)]))
    assert working_ctas(pkg, lambda: cache.batch_step(None)) == shares * cfg.n_kv_heads
    cache.close()
    model.close()
