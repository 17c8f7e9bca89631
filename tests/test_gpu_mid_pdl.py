"""Prompt blocks at the 8B layer shape whose projections take the one-wave kernel (gemm_mid.cu) with K in two slices, the two CTAs of a
tile a cluster, and without: launched ahead of the previous kernel's end, as the engine does, and behind it the logits are the same bits;
also where the block is the short prompts of a batch.  The batch's logits are those of its sequences one by one within 2e-2, as everywhere."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def model(pkg):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    m = pkg.Model.synthetic(pkg.CONFIGS["llama3_8b_l2"], seed=0, max_seq=512)
    yield m
    m.close()


def ids(pkg, oracle, stream, n):
    cfg = pkg.CONFIGS["llama3_8b_l2"]
    return oracle.synth_tokens(stream, n, cfg.embed_rows or cfg.vocab)


@pytest.mark.parametrize("n", [129, 201, 225, 384, 449])
def test_prompt(pkg, oracle, model, n):
    got, seq = [], ids(pkg, oracle, n, n).tolist()
    for use_pdl in (1, 0, 1):
        cache = pkg.Cache(model)
        cache.set_options(use_pdl=use_pdl)
        cache.infer(seq)
        got.append(cache.logits())
        cache.close()
    assert (got[0] == got[1]).all() and (got[0] == got[2]).all()


@pytest.mark.parametrize("n_seqs,n", [(3, 60), (5, 80)])
def test_batch_of_short_prompts(pkg, oracle, model, n_seqs, n):
    got, prompts = [], np.stack([ids(pkg, oracle, 10 + b, n) for b in range(n_seqs)])
    for use_pdl in (1, 0):
        cache = pkg.Cache(model)
        cache.set_options(use_pdl=use_pdl)
        cache.batch_init(n_seqs)
        cache.batch_prefill(prompts)
        got.append(cache.batch_step(None)[1].view(np.float16).astype(np.float32))
        cache.close()
    assert (got[0] == got[1]).all()
    cache = pkg.Cache(model)
    for b in range(n_seqs):
        cache.reset()
        cache.infer(prompts[b].tolist())
        assert np.abs(cache.logits().view(np.float16).astype(np.float32) - got[0][b]).max() <= 2e-2
    cache.close()
