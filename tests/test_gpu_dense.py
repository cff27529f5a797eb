"""es_dense_attention: online softmax over every block with offsets from a sample of the columns, against the fp32 oracle at
ragged lengths, with and without rows for which the sample does not do."""
import pytest
import torch

from oracle import echosparse_ref as R

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 4: one block; 130: a second, ragged tile; 1000: an odd number of blocks; 4288 and 8256: samples of one and of two iterations
@pytest.mark.parametrize("L,H,far", [(4, 1, False), (130, 2, False), (1000, 3, True), (4288, 2, True), (8256, 1, False)])
def test_dense_attention_with_sampled_offsets(L, H, far):
    """`far`: in head 0 a key outside the sample (the first 128 columns at these lengths) has logits more than 2^60 above the
    sample's maximum, in head 1 a value of 1e38 meets a P above 4, so that the unnormalised output overflows: both make their
    tiles start again. Tolerance: P and the output are rounded to bf16 (2^-9 each): 1e-2 of the 2-norm, 3e-2 of a head's
    largest value in a single one; the LSE is fp32 with logits up to a few hundred: 1e-4 of those."""
    from self_trainable_or_free_attn_b200 import _native, backends
    K = backends.kernels(backends.resolve("auto", DEV))
    g = torch.Generator().manual_seed(L)
    pos = torch.arange(L, dtype=torch.float32)[:, None, None] / 300.0
    q, k, v = [(torch.sin(pos * torch.randn(1, H, 128, generator=g) + torch.randn(1, H, 128, generator=g)) * 3.0
                + 0.05 * torch.randn(L, H, 128, generator=g)).to(torch.bfloat16).to(DEV) for _ in range(3)]
    if far:
        k[L - 100, 0] = 90.0 * q[L // 2, 0] / q[L // 2, 0].float().norm()
        k[L - 90, 1] = 30.0 * q[L // 3, 1] / q[L // 3, 1].float().norm()
        v[L - 90, 1] = 1e38
    nq = R.cdiv(L, 128)
    out, lse = torch.full_like(q, 7.0), torch.zeros(nq * 128, H, device=DEV)
    K.dense_attention(q, k, v, out, lse)
    ref, ref_lse = R.dense_attention(q, k, v)
    if far:
        sample = (q[:, 0].float() @ k[:128, 0].float().t()).amax(1) * (R.LOG2E / 128 ** 0.5)
        assert ((ref_lse[:, 0] - sample) > 60).any() and torch.isfinite(ref).all()
    scale = ref.abs().amax((0, 2), keepdim=True)
    got, want = out.float() / scale, ref / scale
    assert (got - want).norm() <= 1e-2 * want.norm() and (got - want).abs().max() <= 3e-2
    assert (lse[:L] - ref_lse).abs().max() <= 1e-4 * max(1.0, float(ref_lse.abs().max()) / 100)
    assert (lse[L:] == 1e30).all()
    assert _native.device_status() == 0


@pytest.mark.parametrize("L", [4, 64, 128, 129, 200, 256])
def test_short_sequences_repeat_their_bits(L):
    """One or two iterations per tile: the two warps that share a row have the least between their reading of the row maximum
    and their writing of the row sums. 200 launches give the same bits, and those of the oracle (tolerances as above)."""
    from self_trainable_or_free_attn_b200 import _native, backends
    K = backends.kernels(backends.resolve("auto", DEV))
    g = torch.Generator().manual_seed(L)
    H = 160
    q, k, v = [(2.0 * torch.randn(L, H, 128, generator=g)).to(torch.bfloat16).to(DEV) for _ in range(3)]
    out, lse = torch.empty_like(q), torch.empty(R.cdiv(L, 128) * 128, H, device=DEV)
    K.dense_attention(q, k, v, out, lse)
    ref, ref_lse = R.dense_attention(q, k, v)
    assert (out.float() - ref).norm() <= 1e-2 * ref.norm() and (lse[:L] - ref_lse).abs().max() <= 1e-4
    again, lse2 = torch.empty_like(out), torch.empty_like(lse)
    for _ in range(200):
        K.dense_attention(q, k, v, again, lse2)
        assert torch.equal(again, out) and torch.equal(lse2, lse)
    assert _native.device_status() == 0


def test_wrong_shapes_are_refused():
    """What the kernel would read or write out of range is refused on the host."""
    from self_trainable_or_free_attn_b200 import backends
    K = backends.kernels(backends.resolve("auto", DEV))
    q = torch.zeros(130, 2, 128, device=DEV, dtype=torch.bfloat16)
    lse = torch.empty(256, 2, device=DEV)
    for bad in (dict(k=q[:129]), dict(v=q[:, :1].contiguous()), dict(out=q[:100]), dict(lse=lse[:130]), dict(lse=lse.double()),
                dict(lse=torch.empty(2, 256, device=DEV).t())):
        with pytest.raises(AssertionError):
            K.dense_attention(**{**dict(q=q, k=q, v=q, out=torch.empty_like(q), lse=lse), **bad})


def _rows_fp64(q, k, v, h, rows):
    s = q[rows, h].double() @ k[:, h].double().t() / 128 ** 0.5
    return torch.softmax(s, 1) @ v[:, h].double(), torch.logsumexp(s, 1) * R.LOG2E


@pytest.mark.parametrize("L", [2240, 4680, 9360])
def test_no_less_precise_than_two_sweeps(L):
    """Peaked rows (a few keys hold most of a row), far more keys than the sample has: the error against fp64 is no larger than
    that of the kernel whose offset is the exact maximum, although most rows have their largest term outside the sample."""
    from self_trainable_or_free_attn_b200 import backends
    K = backends.kernels(backends.resolve("auto", DEV))
    g = torch.Generator(device=DEV).manual_seed(L)
    H = 2
    q, k, v = [(torch.randn(L, H, 128, device=DEV, generator=g) * sc).to(torch.bfloat16) for sc in (1.8, 1.8, 1.0)]
    nq, nb = R.cdiv(L, 128), R.cdiv(L, 64)
    one, lse1, two, lse2 = torch.empty_like(q), torch.empty(nq * 128, H, device=DEV), torch.empty_like(q), torch.empty(nq * 128, H, device=DEV)
    K.dense_attention(q, k, v, one, lse1)
    blocks = torch.arange(nb, device=DEV, dtype=torch.int32).expand(nq, H, nb).contiguous()
    K.exact_fallback(q, k, v, two, torch.full((nq, H), nb, device=DEV, dtype=torch.int32), blocks, lse2,
                     torch.ones(nq, H, device=DEV, dtype=torch.int32))
    err = []
    for out, lse in ((one, lse1), (two, lse2)):
        d = n = 0.0
        for h in range(H):
            ref, ref_lse = _rows_fp64(q, k, v, h, slice(0, L))
            d, n = d + (out[:, h].double() - ref).square().sum(), n + ref.square().sum()
            assert (lse[:L, h] - ref_lse).abs().max() <= 1e-4
        err.append(float((d / n).sqrt()))
    assert err[0] <= err[1], err


@pytest.mark.parametrize("L", [240, 8256, 32760])
def test_tiles_that_start_again(L):
    """A key outside the sample (one pair of blocks in 32, 1 to 8 of them, evenly spread) whose logits pass the sample's maximum by
    more than 2^60 (head 0), or whose value makes the unnormalised output overflow (head 1): two iterations in all, a sample of two,
    a sample of eight. Rows of the tiles in question and some others against fp64; tolerances as above."""
    from self_trainable_or_free_attn_b200 import _native, backends
    K = backends.kernels(backends.resolve("auto", DEV))
    n = R.cdiv(L, 128)
    sample = min(n, min(max(n >> 5, 1), 8))
    columns = torch.cat([torch.arange(128) + 128 * (i * n // sample) for i in range(sample)])
    key = next(c for c in range(L - 60, 0, -1) if not (columns == c).any())
    g = torch.Generator(device=DEV).manual_seed(L)
    q, k, v = [torch.randn(L, 2, 128, device=DEV, generator=g).to(torch.bfloat16) for _ in range(3)]
    far = [L // 2, L // 3]
    k[key, 0] = 80.0 * q[far[0], 0] / q[far[0], 0].float().norm()
    k[key, 1] = 12.0 * q[far[1], 1] / q[far[1], 1].float().norm()
    v[key, 1] = 1e38
    out, lse = torch.full_like(q, 7.0), torch.zeros(n * 128, 2, device=DEV)
    K.dense_attention(q, k, v, out, lse)
    for h in range(2):
        rows = sorted({*range(far[h] // 128 * 128, min(far[h] // 128 * 128 + 128, L)), *range(0, L, 97), L - 1})
        ref, ref_lse = _rows_fp64(q, k, v, h, rows)
        top = (q[far[h], h].float() @ k[columns[columns < L].to(DEV), h].float().t()).max() * (R.LOG2E / 128 ** 0.5)
        gap = float(q[far[h], h].float() @ k[key, h].float()) * R.LOG2E / 128 ** 0.5 - float(top)
        assert gap > (60 if h == 0 else 3), gap
        got = out[rows, h].double()
        assert torch.isfinite(got).all()
        scale = ref.abs().max()
        assert (got / scale - ref / scale).norm() <= 1e-2 * (ref / scale).norm() and (got - ref).abs().max() <= 3e-2 * scale
        assert (lse[rows, h].double() - ref_lse).abs().max() <= 1e-4 * max(1.0, float(ref_lse.abs().max()) / 100)
    assert _native.device_status() == 0
