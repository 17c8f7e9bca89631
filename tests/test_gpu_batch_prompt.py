"""New prompts of a batch share blocks of rows (cache_batch_prefill): a sequence's next-step logits must not depend on
which sequences share its block or where the block ends.  Each is compared with a single-sequence run of the same prompt on
the same model: other tile positions and split counts change FP32 summation orders only, 4e-3 as in
test_gpu_prefill.py's prefix test."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("n_seqs,n_prompt", [(1, 2), (3, 2), (5, 37), (7, 129), (128, 40), (3, 1500), (2, 4300), (2, 1)])
def test_batch_prompt_equals_single_prompts(pkg, oracle, n_seqs, n_prompt):
    cfg = pkg.CONFIGS["tiny"]
    prompts = np.stack([oracle.synth_tokens(300 + b, n_prompt, cfg.vocab) for b in range(n_seqs)])
    model = pkg.Model.synthetic(cfg, seed=0, max_seq=n_prompt + 8)
    cache = pkg.Cache(model)
    cache.batch_init(n_seqs)
    cache.batch_prefill(prompts[::-1].copy())  # a longer past of other rows in the same cache
    cache.batch_prefill(prompts)
    first, logits = cache.batch_step(None)
    second, logits2 = cache.batch_step(first)
    one = pkg.Cache(model)
    for b in sorted({0, 1 % n_seqs, n_seqs // 2, n_seqs - 1}):
        one.reset()
        seq = prompts[b].tolist()
        assert np.abs(oracle.f16(logits[b]) - (one.infer(seq), oracle.f16(one.logits()))[1]).max() <= 4e-3, b
        seq.append(int(first[b]))
        assert np.abs(oracle.f16(logits2[b]) - (one.infer(seq), oracle.f16(one.logits()))[1]).max() <= 4e-3, b
    one.close()
    cache.close()
    model.close()
