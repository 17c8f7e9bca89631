"""The device sampler's floor from the largest entry of each of the 1024 summation classes.  The kernel says how many entries it ordered and
whether the classes led to them; both are what the host finds from the same t_i, so that each case takes the path it is there for: all
large entries in one class or two, exactly as many above the floor as the list takes, one less and one more, nearly all classes above it (the
list is not tried), logits of any scale and at any temperature, equal logits, large entries that differ by one FP16 step, a floor that is
exactly a wanted entry, the most wanted entries that go by classes and one more, the smallest vocabulary that does.  The token is
the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from gpu_util import dev  # noqa: E402
from test_gpu_sampler import device_sample  # noqa: E402

CAP, LISTED = 2048, 880


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def tree_total(t):
    """The kernel's sum: 1024 classes in index order, 32 classes by a butterfly, 32 warps by another."""
    classes = np.zeros(1024, dtype=np.float32)
    for row in range(0, len(t), 1024):
        part = t[row:row + 1024]
        classes[:len(part)] += part
    warps = classes.reshape(32, 32)
    for _ in range(2):
        for m in (16, 8, 4, 2, 1):
            warps = warps + warps[:, np.arange(32) ^ m]
        warps = np.tile(warps[:, 0], (32, 1))
    return warps[0, 0]


def expected(t, want):
    """(entries ordered, 1 if by classes) for the t_i; entries None where the radix select chooses."""
    if want > 512 or len(t) < 32768:
        return None, 0
    most = np.array([t[c::1024].max() for c in range(1024)], dtype=np.float32)

    def down_to(bits):
        return ((np.sort(most)[-want].view(np.uint32) >> bits) << bits).view(np.float32)
    floor = down_to(19)
    if floor > 0 and (most >= floor).sum() > (220 if want <= 200 else 400 if want <= 390 else 640):
        floor = down_to(9)
    if (most >= floor).sum() > LISTED:
        return None, 0
    total = tree_total(t)
    n = int((t / total >= floor / total).sum())
    return (n, 1) if n <= CAP else (None, 0)


def exps(bits, temperature):
    x = torch.from_numpy(bits.view(np.float16).astype(np.float32)).cuda()
    return torch.exp(x / torch.full_like(x, temperature)).cpu().numpy()


def order_of(bits):
    return np.lexsort((np.arange(len(bits)), -bits.view(np.float16).astype(np.float32)))


def draws(pkg, oracle, bits, temperature, top_k, top_p, exact, seed=9):
    """Four draws checked against the oracle; returns (entries ordered, by classes) of the kernel."""
    vocab, d = len(bits), dev(bits)
    scratch = torch.zeros(pkg.lib.llmb_sample_scratch_bytes(vocab), dtype=torch.uint8, device="cuda")
    tok = torch.zeros(1, dtype=torch.int32, device="cuda")
    where = {int(t): i for i, t in enumerate(order_of(bits)[:1100])}
    for draw in range(4):
        rc, got, result = device_sample(pkg, d, vocab, scratch, tok, temperature, top_k, top_p, seed, draw)
        assert rc == 0 and result == 0, (rc, result)
        u = float(oracle.lib().oracle_sampler_uniform(seed, draw))
        want = int(oracle.lib().oracle_sample(bits.ctypes.data, vocab, temperature, top_k, top_p, u))
        # u may lie within FP32 ulps of the boundary between two entries: neighbours in the order
        assert got == want or (not exact and abs(where[got] - where[want]) <= 1), (temperature, top_p, draw, got, want)
    _, n, by_class = scratch[:12].view(torch.int32).tolist()
    return n, by_class


def logits(vocab, kind, rng, std=1.3):
    x = (rng.standard_normal(vocab) * std).astype(np.float16)
    if kind == "one class":
        x[5::1024] = (6 + rng.random(len(x[5::1024]))).astype(np.float16)
    elif kind == "two classes":
        x[[5 + 1024 * i for i in range(60)] + [700 + 1024 * i for i in range(60)]] = (7 + rng.random(120)).astype(np.float16)
    elif kind == "above cap":  # of all classes
        x[rng.choice(vocab, 5000, replace=False)] = (5 + 0.001 * rng.random(5000)).astype(np.float16)
    elif isinstance(kind, tuple):  # so many equal entries in so many classes, the rest well below
        n, classes = kind
        x = np.minimum(x, np.float16(3.0))
        x[np.arange(classes)] = 5.0
        spare = (np.arange(1, vocab // 1024)[:, None] * 1024 + np.arange(classes)[None]).reshape(-1)
        x[rng.choice(spare, n - classes, replace=False)] = 5.0
    elif kind == "steps":
        x[rng.choice(vocab, 400, replace=False)] = (np.float16(6).view(np.uint16) + np.arange(400) % 7).astype(np.uint16).view(np.float16)
    elif kind == "low":
        x = (-20 + x.astype(np.float32)).astype(np.float16)
    elif kind == "tiny":  # every probability within a few steps of another, total far from one
        x[:] = (-20 + 0.01 * rng.integers(0, 8, vocab)).astype(np.float16)
    elif kind == "equal":
        x[:] = 0.5
    elif kind == "masked":  # a few that are allowed
        x[rng.permutation(vocab)[30:]] = -np.inf
    return x.view(np.uint16).copy()


@pytest.mark.parametrize("vocab,kind,top_k,by_class", [
    (128256, "one class", 100, 1), (128256, "two classes", 50, 1), (128256, "above cap", 50, 0), (32768, "steps", 200, 1), (8192, "steps", 200, 0), (128256, "tiny", 50, 0),
    (128256, "low", 50, 1), (128256, "equal", 50, 0), (128256, "masked", 50, 0), (128256, "masked", 20, 1), (1000, "normal", 900, 0), (1024, "normal", 1024, 0),
    (4096, "normal", 1, 0), (32767, "normal", 50, 0), (32768, "normal", 50, 1), (32768, "normal", 200, 1), (32769, "normal", 512, 1), (32768, "normal", 513, 0), (128256, "normal", 1, 1),
    (128256, "normal", 50, 1), (128256, "normal", 200, 1), (128256, "normal", 201, 1), (128256, "normal", 391, 1), (128256, "normal", 512, 1), (128256, "normal", 513, 0), (400001, "normal", 50, 1)])
def test_floor(pkg, oracle, vocab, kind, top_k, by_class):
    bits = logits(vocab, kind, np.random.default_rng(vocab + top_k))
    for temperature, top_p in [(0.7, 0.9), (1.3, 0.6), (0.5, 0.98)]:
        n, by = draws(pkg, oracle, bits, temperature, top_k, top_p, kind == "normal")
        want_n, want_by = expected(exps(bits, temperature), top_k)
        assert by == want_by == by_class and min(top_k, vocab) <= n <= CAP
        assert n == want_n or not by, (n, want_n)


@pytest.mark.parametrize("n,classes,by_class", [(2047, 600, 1), (2048, 600, 1), (2049, 600, 0), (3000, 600, 0), (880, 880, 1), (881, 881, 0), (1000, 880, 1)])
def test_list_is_full(pkg, oracle, n, classes, by_class):
    bits = logits(128256, (n, classes), np.random.default_rng(n))
    for temperature in (0.7, 1.3):
        assert expected(exps(bits, temperature), 64) == ((n, 1) if by_class else (None, 0))
        got, by = draws(pkg, oracle, bits, temperature, 64, 0.9, False)
        assert by == by_class and (got == n if by_class else 64 <= got <= CAP)


@pytest.mark.parametrize("std,temperature", [(1.3, 0.1), (1.3, 0.2), (2.5, 0.2), (2.5, 0.3), (2.5, 0.7), (0.3, 1.3), (1.3, 5.0), (0.01, 1.0)])
def test_any_scale(pkg, oracle, std, temperature):
    """exp(logit / temperature) from 2^-90 to 2^86: the classes lead to the wanted entries wherever these stand out."""
    bits = logits(128256, "normal", np.random.default_rng(int(std * 100)), std)
    n, by = draws(pkg, oracle, bits, temperature, 50, 0.9, False)
    want_n, want_by = expected(exps(bits, temperature), 50)
    assert by == want_by == 1 and n == want_n, (n, want_n)


def test_floor_on_a_bin_edge(pkg):
    """The wanted entries are exactly 1, the lower end of a bin, and as many are the nearest that an exponential comes to below it: these
    count only where the division by the total gives them the same probability."""
    vocab = 33000
    below = next(k for k in range(1, 64) if exps(np.array([0x8000 + k], dtype=np.uint16), 1.0)[0] < 1)  # FP16 numbers next to -0
    rng = np.random.default_rng(3)
    scratch = torch.zeros(pkg.lib.llmb_sample_scratch_bytes(vocab), dtype=torch.uint8, device="cuda")
    tok = torch.zeros(1, dtype=torch.int32, device="cuda")
    for count in range(20, 32):
        wanted = rng.permutation(1024)[:count] + 1024 * rng.integers(0, 8, count)  # one to a class
        bits = np.full(vocab, np.float16(-np.inf).view(np.uint16), dtype=np.uint16)
        bits[wanted], bits[rng.choice(np.setdiff1d(np.arange(9000), wanted), count, replace=False)] = 0, 0x8000 + below
        t = exps(bits, 1.0)
        total = tree_total(t)
        p = t / total
        n, by = expected(t, count)
        assert by == 1 and n in (count, 2 * count)
        order = np.lexsort((np.arange(vocab), -p))[:count]
        f = np.float32
        pr = p[order] / np.cumsum(p[order], dtype=np.float32)[-1]  # top_k_sampling
        run = np.cumsum(pr, dtype=np.float32)
        cut = int(np.argmax(run >= f(0.9)))
        pr = np.cumsum(pr[:cut + 1] / run[cut], dtype=np.float32)
        for draw in range(6):
            rc, got, result = device_sample(pkg, dev(bits), vocab, scratch, tok, 1.0, count, 0.9, 4, draw)
            assert rc == 0 and result == 0 and scratch[4:12].view(torch.int32).tolist() == [n, 1]
            u = f(pkg.lib.llmb_sampler_uniform(4, draw))
            over = np.nonzero(u < pr)[0]
            assert got == int(order[over[0] if len(over) else 0]), (count, draw)
