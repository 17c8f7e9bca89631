"""Attention of the whole-step kernel at the edges of its work split: 16-row tiles, 16 row slots per CTA (8 at head_dim 128),
up to 128 rows in one split, splits of 128 rows and more beyond, up to eight query heads per KV head.  Teacher-forced steps behind
prompts of every such length against the block path, whose attention is another kernel; 2-layer models, logits within 4e-3
(FP32 summation orders only, the bound of the prefix test in test_gpu_prefill.py)."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("nq,nkv,hd,lens", [
    (4, 2, 64, (30, 33, 255, 256, 257, 511, 513, 700, 4607, 9300)), (8, 1, 128, (31, 127, 128, 129, 256, 257, 300, 1000, 2500)),
    (8, 2, 128, (17, 240, 256, 257, 1025, 5000)), (6, 1, 64, (40, 257, 1300)), (3, 1, 128, (20, 255, 700)), (32, 8, 128, (128, 4200, 4800))])
def test_step_attention_matches_the_block_path(pkg, oracle, nq, nkv, hd, lens):
    cfg = dataclasses.replace(pkg.CONFIGS["tiny"], name="attn", n_q_heads=nq, n_kv_heads=nkv, head_dim=hd, vocab=512)
    model = pkg.Model.synthetic(cfg, seed=1, max_seq=max(lens) + 8)
    a, b = pkg.Cache(model), pkg.Cache(model)
    for n in lens:
        ids = oracle.synth_tokens(n, n + 3, cfg.vocab).tolist()
        a.reset()
        a.infer(ids[:n])
        for i in range(1, 4):
            a.infer(ids[:n + i])                 # one decode step each
            b.reset()
            b.infer(ids[:n + i])                 # the same rows as one block
            d = np.abs(oracle.f16(a.logits()) - oracle.f16(b.logits())).max()
            assert d <= 4e-3, (n, i, d)
    a.close(); b.close(); model.close()
