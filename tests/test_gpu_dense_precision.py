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
