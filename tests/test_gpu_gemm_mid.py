"""The one-wave projection kernel of middling blocks (gemm_mid.cu) at its edges: the fewest rows, tiles of 16 columns more or less
than the rows need, the last tile nearly empty, K in two slices (from 2048 on, also of odd lengths), one K step, K steps that do not divide among the accumulators (two and four of them), the
most rows it takes and one more.  Against float64, tolerances as in test_gpu_prefill.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from gpu_util import assert_close_fp16, dev, f16, host_u16  # noqa: E402
from test_gpu_prefill import EPI_RESIDUAL, EPI_ROPE_KV, EPI_STORE, gemm, mats, matmul64, tc_tol  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("m,n,k", [(129, 4096, 64), (129, 4096, 320), (192, 4096, 4096), (193, 6144, 448), (145, 18816, 128), (224, 18944, 192),
                                   (225, 18944, 64), (384, 4736, 1024), (385, 4096, 576), (256, 4096, 2048), (257, 4096, 2112), (448, 4096, 2048), (200, 6144, 2176), (449, 4096, 2048), (517, 4096, 704), (896, 4096, 128), (897, 4096, 128)])
def test_store_and_residual(pkg, oracle, m, n, k):
    a, b = mats(oracle, m, n, k, 50)
    da, db = dev(a), dev(b)
    out = torch.full((m + 3, n), 0x7BFF, dtype=torch.int16, device="cuda")  # rows past m must stay untouched
    gemm(pkg, a=da, b=db, c=out, m=m, n=n, k=k, epilogue=EPI_STORE)
    acc = matmul64(a, b)
    got = host_u16(out).reshape(m + 3, n)
    assert_close_fp16(got[:m], acc, what="store", abs_tol=tc_tol(acc, k))
    assert (got[m:] == 0x7BFF).all()
    res = oracle.synth_fp16(7, 3, m * n, std=1.0).reshape(m, n)
    out = dev(res.copy())
    gemm(pkg, a=da, b=db, c=out, m=m, n=n, k=k, epilogue=EPI_RESIDUAL)
    want = acc.astype(np.float16).astype(np.float64) + f16(res).astype(np.float64)
    # half(acc) may sit one FP16 step (|acc| 2^-10) from the product's rounding, and the sum is rounded once more (|want| 2^-10)
    assert_close_fp16(host_u16(out).reshape(m, n), want, what="residual", max_frac=0.1,
                      abs_tol=(np.abs(acc) + np.abs(want)) * 2.0 ** -10 + tc_tol(acc, k))


@pytest.mark.parametrize("m,nqh,nkvh,hd,k,batched", [(129, 32, 8, 128, 192, False), (200, 32, 8, 128, 2112, False), (210, 28, 6, 128, 2048, True), (300, 32, 8, 128, 64, True), (517, 20, 6, 128, 128, False), (250, 48, 12, 64, 320, False)])
def test_rope_kv(pkg, oracle, m, nqh, nkvh, hd, k, batched):
    """Rows of one sequence, and one row of each of m sequences (row_pos)."""
    n_q, n_kv, pos0, max_pos = nqh * hd, nkvh * hd, 5, (16 if batched else m + 3)   # not batched: the last rows lie past the cache
    n = n_q + 2 * n_kv
    a, b = mats(oracle, m, n, k, 52)
    pos = np.arange(m) % 13 if batched else np.arange(pos0, pos0 + m)
    ang = pos[:, None].astype(np.float32) * np.linspace(1.0, 0.01, hd // 2, dtype=np.float32)[None]
    cs = np.stack([np.cos(ang), np.sin(ang)], axis=-1).astype(np.float32)
    q = torch.zeros((m, n_q), dtype=torch.int16, device="cuda")
    rows = m * max_pos if batched else max_pos
    kc, vc = (torch.zeros((rows + 1, n_kv), dtype=torch.int16, device="cuda") for _ in range(2))
    kw = dict(row_pos=torch.tensor(pos, dtype=torch.int32, device="cuda"), seq_stride=max_pos) if batched else dict(pos0=pos0)
    gemm(pkg, a=dev(a), b=dev(b), c=q, m=m, n=n, k=k, epilogue=EPI_ROPE_KV, n_q=n_q, n_kv=n_kv, head_dim=hd, rope_cs=dev(cs), k_cache=kc,
         v_cache=vc, max_pos=max_pos, **kw)
    y = matmul64(a, b).astype(np.float16).astype(np.float64)
    r = y[:, :n_q + n_kv].reshape(m, -1, hd // 2, 2)
    c, s = cs[:, None, :, 0].astype(np.float64), cs[:, None, :, 1].astype(np.float64)
    want = np.stack([c * r[..., 0] - s * r[..., 1], s * r[..., 0] + c * r[..., 1]], axis=-1).reshape(m, -1)
    tol = np.repeat(np.abs(r).sum(axis=-1).reshape(m, -1), 2, axis=1) * 2.0 ** -10 + tc_tol(y, k)
    tol += np.abs(want) * 2.0 ** -10  # one FP16 step of either input of a pair, and the result's own rounding
    keep = pos < max_pos
    at = (np.arange(m) * max_pos + pos) if batched else pos[keep]
    assert np.all(np.abs(f16(host_u16(q).reshape(m, n_q)).astype(np.float64) - want[:, :n_q]) <= tol[:, :n_q])
    got_k, got_v = (f16(host_u16(t).reshape(rows + 1, n_kv)).astype(np.float64) for t in (kc, vc))
    assert np.all(np.abs(got_k[at] - want[keep, n_q:]) <= tol[keep, n_q:])
    v = y[keep, n_q + n_kv:]
    assert np.all(np.abs(got_v[at] - v) <= np.abs(v) * 2.0 ** -10 + tc_tol(y, k))
    rest = np.setdiff1d(np.arange(rows + 1), at)
    assert (got_k[rest] == 0).all() and (got_v[rest] == 0).all()
