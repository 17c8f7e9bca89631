"""The device sampler's floor from the largest entry of each of the 1024 summation classes: all large entries in one class or two (the
floor then lies in the bulk and the general selection takes over), many more entries above the floor than the list takes, exactly as
many as it takes, large entries that differ by one FP16 step, probabilities that the division by the total joins, as many classes as
wanted entries and fewer.  The token is the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from gpu_util import dev  # noqa: E402
from test_gpu_sampler import device_sample  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("vocab,kind,top_k", [(128256, "one class", 100), (128256, "two classes", 50), (128256, "above cap", 50), (128256, "at cap", 64),
                                              (128256, "past cap", 64), (32768, "steps", 200), (128256, "tiny", 50), (1000, "normal", 900), (1024, "normal", 1024),
                                              (4096, "normal", 1), (128256, "normal", 50), (128256, "normal", 200)])
def test_floor(pkg, oracle, vocab, kind, top_k):
    rng = np.random.default_rng(vocab + top_k)
    x = (rng.standard_normal(vocab) * 1.3).astype(np.float16)
    if kind == "one class":
        x[5::1024] = (6 + rng.random(len(x[5::1024]))).astype(np.float16)
    elif kind == "two classes":
        x[[5 + 1024 * i for i in range(60)] + [700 + 1024 * i for i in range(60)]] = (7 + rng.random(120)).astype(np.float16)
    elif kind in ("above cap", "at cap", "past cap"):
        n = {"above cap": 5000, "at cap": 2048, "past cap": 2049}[kind]
        x[rng.choice(vocab, n, replace=False)] = (5 + 0.001 * rng.random(n)).astype(np.float16)
    elif kind == "steps":
        x[rng.choice(vocab, 400, replace=False)] = (np.float16(6).view(np.uint16) + np.arange(400) % 7).astype(np.uint16).view(np.float16)
    elif kind == "tiny":  # every probability within a few steps of another, total far from one
        x[:] = (-20 + 0.01 * rng.integers(0, 8, vocab)).astype(np.float16)
    bits = x.view(np.uint16).copy()
    d = dev(bits)
    scratch = torch.zeros(pkg.lib.llmb_sample_scratch_bytes(vocab), dtype=torch.uint8, device="cuda")
    tok = torch.zeros(1, dtype=torch.int32, device="cuda")
    order = np.lexsort((np.arange(vocab), -x.astype(np.float32)))
    where = {int(t): i for i, t in enumerate(order[:1100])}
    for temperature, top_p in [(0.7, 0.9), (1.3, 0.6), (0.5, 0.98)]:
        for draw in range(4):
            rc, got, result = device_sample(pkg, d, vocab, scratch, tok, temperature, top_k, top_p, 9, draw)
            assert rc == 0 and result == 0, (rc, result)
            u = float(oracle.lib().oracle_sampler_uniform(9, draw))
            want = int(oracle.lib().oracle_sample(bits.ctypes.data, vocab, temperature, top_k, top_p, u))
            # u may lie within FP32 ulps of the boundary between two entries: neighbours in the order
            assert got == want or (kind != "normal" and abs(where[got] - where[want]) <= 1), (temperature, top_p, draw, got, want)
