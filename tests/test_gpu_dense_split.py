"""es_dense_attention_split: tiles cut between CTAs and merged, against the fp32 oracle and against whole tiles."""
import pytest
import torch

from oracle import echosparse_ref as R

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(L, H, seed=0):
    g = torch.Generator().manual_seed(seed + L)
    return [(1.5 * torch.randn(L, H, 128, generator=g)).to(torch.bfloat16).to(DEV) for _ in range(3)]


def _both(q, k, v):
    """(out, lse) of the cut and of the whole tiles."""
    from self_trainable_or_free_attn_b200 import _native as N, backends
    K = backends.kernels(backends.resolve("auto", DEV))
    L, H, _ = q.shape
    res = []
    for cut in (True, False):
        out, lse = torch.full_like(q, 7.0), torch.zeros(R.cdiv(L, 128) * 128, H, device=DEV)
        if cut:
            K.dense_attention(q, k, v, out, lse)
        else:
            N.check(N.load().es_dense_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), L, H,
                                                N.stream_ptr()), "es_dense_attention")
        res.append((out, lse))
    assert N.device_status() == 0
    return res


# on 148 SMs: every iteration a piece of its own, the last with one token (897, 1025); pieces of several iterations, two to eight a
# tile (2111, 4096, 8000 x 1); whole tiles before the cut ones (1560, 2500); cuts inside the tiles of the last two waves (4700 and,
# with whole tiles in front, 8000 x 8)
@pytest.mark.parametrize("L,H", [(897, 1), (1025, 2), (2111, 2), (4096, 1), (8000, 1), (1560, 12), (2500, 8), (4700, 6), (8000, 8)])
def test_cut_tiles_match_the_oracle(L, H):
    """P and the output are rounded to bf16 (2^-9 each): 1e-2 of the 2-norm. Cut and whole differ in the offsets, so in the
    rounding of every P (a random 2^-9 / sqrt(3) of each term, smaller in the sum) and once in the output's."""
    from self_trainable_or_free_attn_b200 import _native as N
    q, k, v = _inputs(L, H)
    assert N.load().es_dense_scratch_bytes(L, H) > 0
    (out, lse), (whole, lse_w) = _both(q, k, v)
    ref, ref_lse = R.dense_attention(q, k, v)
    assert (out.float() - ref).norm() <= 1e-2 * ref.norm() and (out.float() - whole.float()).norm() <= 5e-3 * ref.norm()
    assert (lse[:L] - ref_lse).abs().max() <= 1e-4 and (lse[L:] == 1e30).all()
    again = _both(q, k, v)[0]
    assert torch.equal(again[0], out) and torch.equal(again[1], lse)


def test_pieces_with_far_offsets_and_nonfinite_rows():
    """One piece holds a row's only large logits (its offset is far above the others'), another leaves the range of its sample
    and starts again; a NaN row stays alone, and keys at -inf that fill a piece leave the other pieces' result."""
    L, H = 2048, 1
    q, k, v = _inputs(L, H)
    k[1500, 0] = 60.0 * q[300, 0] / q[300, 0].float().norm()           # iteration 11, not the first of a piece's columns
    k[40, 0] = 40.0 * q[900, 0] / q[900, 0].float().norm()
    (out, lse), (whole, lse_w) = _both(q, k, v)
    ref, ref_lse = R.dense_attention(q, k, v)
    assert (out.float() - ref).norm() <= 1e-2 * ref.norm()
    assert (lse[:L] - ref_lse).abs().max() <= 1e-4 * float(ref_lse.abs().max()) / 100
    q[77] = float("nan")
    (bad, lse_b), _ = _both(q, k, v)
    # a NaN sends its tile's pieces through their second sweep: other offsets for the tile's other rows, same bits elsewhere
    rows = torch.arange(L, device=DEV)
    near, far = (rows < 128) & (rows != 77), rows >= 128
    assert torch.isnan(bad[77]).all() and torch.equal(bad[far], out[far]) and torch.equal(lse_b[:L][far], lse[:L][far])
    assert (bad[near].float() - ref[near]).norm() <= 1e-2 * ref[near].norm()
    q = q.clone()
    q[77] = 0.0
    q[:, 0, 0] = 1.0
    k[256:512, 0, 0] = -float("inf")                                   # iterations 2 and 3
    (out, lse), _ = _both(q, k, v)
    keep = torch.cat([torch.arange(256), torch.arange(512, L)]).to(DEV)
    a = (q[:, 0].float() @ k[keep, 0].float().t()) / 128 ** 0.5
    want = torch.softmax(a, 1) @ v[keep, 0].float()
    assert (out[:, 0].float() - want).norm() <= 1e-2 * want.norm()


def test_scratch_is_checked():
    from self_trainable_or_free_attn_b200 import _native as N
    lib = N.load()
    q, k, v = _inputs(1024, 1)
    out, lse = torch.full_like(q, 7.0), torch.empty(1024, 1, device=DEV)
    size = lib.es_dense_scratch_bytes(1024, 1)
    scratch = torch.empty(size, device=DEV, dtype=torch.uint8)
    call = lambda p, n: lib.es_dense_attention_split(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), p, n,
                                                     1024, 1, N.stream_ptr())
    assert call(scratch.data_ptr(), size - 1) < 0 and "smaller" in N.last_error()
    assert call(scratch.data_ptr() + 4, size) < 0 and "aligned" in N.last_error()
    torch.cuda.synchronize()
    assert (out == 7.0).all()
