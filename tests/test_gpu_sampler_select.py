"""The device sampler's selection at its edges (llmb_sample_logits): vocabularies around the 1024 summation classes, one
that keeps its t_i in the caller's scratch, orders decided by the index alone (every logit equal, so that the radix select
refines down to the last index bits), top_k from 1 to 1024, prefixes that run past top_k.  The token is the oracle's; at
top_p = 1 either side of the FP32 ulp at which the prefix ends (see test_gpu_sampler.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from gpu_util import dev  # noqa: E402
from test_gpu_sampler import chain_f32, device_sample  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("vocab,kind", [(1, "normal"), (2, "equal"), (1023, "normal"), (1024, "normal"), (1025, "normal"), (2049, "equal"),
                                        (5000, "two"), (128256, "equal"), (128256, "two"), (400001, "normal")])
def test_selection_edges(pkg, oracle, vocab, kind):
    logits = oracle.synth_fp16(77 + vocab, 9, vocab, std=1.5).copy()
    if kind == "equal":
        logits[:] = np.float16(0.5).view(np.uint16)
    if kind == "two":  # a few hundred equal heads among equal rest: both bins have to be refined by index
        logits[:] = np.float16(-2.0).view(np.uint16)
        logits[np.random.default_rng(1).choice(vocab, 300, replace=False)] = np.float16(4.0).view(np.uint16)
    d = dev(logits)
    scratch = torch.zeros(pkg.lib.llmb_sample_scratch_bytes(vocab), dtype=torch.uint8, device="cuda")
    tok = torch.zeros(1, dtype=torch.int32, device="cuda")
    checked = 0
    for temperature, top_k, top_p in [(0.7, 50, 0.9), (1.3, 1024, 0.95), (0.9, 1000, 0.5), (1.0, 1, 1.0), (0.8, 333, 1.0), (0.6, 300, 0.999)]:
        for draw in range(3):
            rc, got, result = device_sample(pkg, d, vocab, scratch, tok, temperature, top_k, top_p, 5, draw)
            assert rc == 0, pkg.lib.llmb_last_error()
            u = float(oracle.lib().oracle_sampler_uniform(5, draw))
            if result == 2:  # past 1024 entries: reported; only where rounding can carry the prefix past the first top_k
                assert got == -1 and top_p >= 0.99 and vocab > 1024
                continue
            accept = {int(oracle.lib().oracle_sample(logits.ctypes.data, vocab, temperature, top_k, top_p, u))}
            if top_p >= 0.99:
                accept |= {chain_f32(logits, temperature, top_k, top_p, u, slack) for slack in (-4, 4)}
            if kind != "normal" and got not in accept:
                # equal entries: u may lie within FP32 ulps of the boundary between two of them; neighbours in the order
                order = np.lexsort((np.arange(vocab), -logits.view(np.float16).astype(np.float32)))
                where = {int(t): i for i, t in enumerate(order[:1100])}
                assert min(abs(where[got] - where[a]) for a in accept) <= 1
                accept.add(got)
            assert result == 0 and got in accept, (temperature, top_k, top_p, draw, got, accept)
            checked += 1
    assert checked >= 9
