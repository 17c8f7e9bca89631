"""Block attention on the tensor cores (llmb_attn_prefill) against float64 at the edges of its tiles: 128 rows = 128 / G
positions x G query heads, 128 keys, two row tiles per CTA, one head per tile where G does not divide 128.  Scores of
standard deviation sqrt(head_dim) * std^2 reach past the 2^8 growth at which the running maximum moves and O is
rescaled.  The result is one FP16 rounding of FP32 sums with P carried to ~22 bits: one FP16 step, plus 2e-3 absolute where
terms of magnitude up to ~4 cancel (the same bound as test_gpu_prefill.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from gpu_util import dev, host_u16  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("hd,nqh,nkvh,m,pos0,std", [
    (128, 8, 2, 32, 96, 1.0), (128, 8, 2, 33, 96, 1.0), (128, 4, 1, 64, 64, 1.0), (128, 4, 1, 65, 63, 3.0), (128, 8, 1, 300, 77, 1.0),
    (64, 6, 2, 129, 0, 1.0), (128, 3, 1, 257, 255, 1.0), (64, 8, 1, 17, 640, 3.0), (128, 2, 2, 128, 0, 3.0), (128, 8, 4, 1, 0, 1.0),
    (64, 4, 2, 500, 13, 2.0)])
def test_attn_prefill_tile_edges(pkg, oracle, hd, nqh, nkvh, m, pos0, std):
    total, n_q, n_kv = pos0 + m, nqh * hd, nkvh * hd
    q = oracle.synth_fp16(31, 1, m * n_q, std=std).reshape(m, n_q)
    kc = oracle.synth_fp16(31, 2, (total + 130) * n_kv, std=std).reshape(-1, n_kv)
    vc = oracle.synth_fp16(31, 3, (total + 130) * n_kv, std=1.0).reshape(-1, n_kv)
    kc[total:] = vc[total:] = 0x7E00  # NaN past the last row
    out = torch.full((m + 1, n_q), 0x5555, dtype=torch.int16, device="cuda")
    dq, dk, dv = dev(q), dev(kc), dev(vc)
    assert pkg.lib.llmb_attn_prefill(dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), m, pos0, nqh, nkvh, hd, out.data_ptr(), None) == 0, \
        pkg.lib.llmb_last_error()
    got = host_u16(out).reshape(m + 1, n_q)
    assert (got[m] == 0x5555).all(), "wrote past the last row"
    f = lambda a: torch.from_numpy(a.view(np.float16).astype(np.float64)).cuda()
    qf, kf, vf = f(q).view(m, nqh, hd), f(kc[:total]).view(total, nkvh, hd), f(vc[:total]).view(total, nkvh, hd)
    rep = lambda x: x.repeat_interleave(nqh // nkvh, dim=1)
    s = torch.einsum("mhd,thd->hmt", qf, rep(kf)) / np.sqrt(float(hd))
    mask = torch.arange(total, device="cuda")[None, :] > pos0 + torch.arange(m, device="cuda")[:, None]
    p = torch.softmax(s.masked_fill(mask[None], float("-inf")), dim=-1)
    want = torch.einsum("hmt,thd->mhd", p, rep(vf)).reshape(m, n_q).cpu().numpy()
    g = got[:m].view(np.float16).astype(np.float64)
    assert np.isfinite(g).all()
    err = np.abs(g - want)
    assert (err <= np.maximum(np.abs(want) * 2.0 ** -10, 2e-3)).all(), err.max()
    assert (err > np.maximum(np.abs(want) * 2.0 ** -11 * 1.01, 2.0 ** -24)).mean() < 0.05  # nearly always the nearest FP16
