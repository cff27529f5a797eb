"""Dense attention: what is summed or kept in float32 is so to float32's precision, also in long rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _dense(q, k, v):
    from self_trainable_or_free_attn_b200 import _native as N, backends
    K = backends.kernels(backends.resolve("auto", DEV))
    L, H, _ = q.shape
    out, lse = torch.empty_like(q), torch.empty(-(-L // 128) * 128, H, device=DEV)
    K.dense_attention(q, k, v, out, lse)
    assert N.device_status() == 0
    return out


@pytest.mark.parametrize("L", [32760, 65536, 119056])
def test_row_sums_have_no_bias_that_grows_with_the_row(L):
    """V is zero but for the first 128 keys, so the weighted sum is short and what is left is the divisor, a sum of L rounded P. The mean
    signed error over 16,384 rows x 128 columns: the output's rounding (1.66e-3 rms) leaves 1.1e-6 of it, the rounding of 128 P a
    row (1.66e-3 / sqrt(128) rms) 1.1e-6, float32 sums rounded at random far less: 6e-6 is four times the whole. A sum
    whose adds are cut off instead of rounded is short by 2^-25 to 2^-24 each: 1e-5 and more."""
    n = 16384
    g = torch.Generator(device=DEV).manual_seed(L)
    q, k, v = (torch.randn(L, 1, 128, device=DEV, generator=g).to(torch.bfloat16) for _ in range(3))
    v = torch.zeros_like(v)
    v[:128] = 1.0 + torch.rand(128, 1, 128, device=DEV, generator=g)
    out = _dense(q, k, v)[:n, 0].double()
    kd, vd, bias = k[:, 0].double().t().contiguous(), v[:128, 0].double(), 0.0
    for r in range(0, n, 1024):
        s = (q[r:r + 1024, 0].double() @ kd) / 128 ** 0.5
        ref = torch.exp(s[:, :128] - s.logsumexp(1, keepdim=True)) @ vd
        bias += float((out[r:r + 1024] / ref - 1.0).sum()) / (n * 128)
    assert abs(bias) <= 6e-6


@pytest.mark.parametrize("L,key", [(4096, 647), (9360, 5000)])
def test_the_largest_term_above_the_sample_is_exact_however_small_its_share(L, key):
    """V is zero but at one key, whose logit is every row's largest and in no sampled column: its share is 1 / 1000 or less. The outputs are
    that term alone, rounded once to bf16: 1.66e-3 rms of the value; with a P rounded to bf16 as well 2.3e-3."""
    g = torch.Generator(device=DEV).manual_seed(L)
    k, v = (torch.zeros(L, 1, 128, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    k[key, 0, 0] = 1.0
    v[key, 0] = 1.0 + torch.rand(128, device=DEV, generator=g)
    q = torch.zeros(L, 1, 128, device=DEV, dtype=torch.bfloat16)
    q[:, 0, 0] = (0.2 + 1.1 * torch.rand(L, device=DEV, generator=g)) * 128 ** 0.5
    out = _dense(q, k, v)[:, 0].double()
    p = torch.exp(q[:, 0, :1].double() / 128 ** 0.5)
    ref = p * v[key].double() / (p + (L - 1))
    assert float((out / ref - 1.0).square().mean().sqrt()) <= 1.9e-3
