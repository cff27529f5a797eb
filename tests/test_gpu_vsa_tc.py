"""The tcgen05 kernels of the VSA2 fine branch at the edges of their list walk: lists of 1 and 2 blocks, of odd
length, around the 32-entry windows the load warp holds, and over every block; ragged blocks, a query block without a list.
Against the CPU restatement in fp64. Tolerance: outputs and gradients are bf16 / fp16 (half a unit in the last place: 2^-9
resp. 2^-12 relative) from products with P and dS rounded to the same type, a few such roundings each: 1e-2 resp. 2e-3 of the
2-norm."""
import pytest
import torch

from oracle import vsa_ref as R

pytestmark = pytest.mark.gpu
LENGTHS = [0, 1, 2, 3, 30, 31, 32, 33, 34, 63, 64, 65, 66, 67]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("split", [False, True])
def test_list_lengths(D, dtype, split):
    from self_trainable_or_free_attn_b200 import vsa as V
    nb = 67
    g = torch.Generator().manual_seed(11)
    cnt = torch.randint(1, 65, (nb,), generator=g, dtype=torch.int32)
    cnt[::3] = 64
    valid = R.token_valid(cnt, nb * 64)[None, None, :, None]
    q, k, v, do = [(torch.randn(1, 1, nb * 64, D, generator=g) * valid).to(dtype) for _ in range(4)]
    mask = torch.zeros(1, 1, nb, nb, dtype=torch.bool)
    for i in range(nb):
        mask[0, 0, i, torch.randperm(nb, generator=g)[:LENGTHS[i % len(LENGTHS)]]] = True
    ref = [x.double().requires_grad_(True) for x in (q, k, v)]
    o_ref, lse_ref = R.fine_attention(*ref, cnt, mask)
    o_ref.backward(do.double())
    dev = [x.cuda().requires_grad_(True) for x in (q, k, v)]
    o, lse = V.fine_block_sparse_attention(*dev, cnt.cuda(), V.mask_to_selection(mask.cuda()),
                                           split_kv=V.SplitKV(chunk=33) if split else None)
    o.backward(do.cuda())
    tol = 1e-2 if dtype == torch.bfloat16 else 2e-3
    for name, got, exp in [("o", o, o_ref)] + [("d" + n, x.grad, y.grad) for n, x, y in zip("qkv", dev, ref)]:
        got = got.detach().double().cpu()
        assert torch.isfinite(got).all(), name
        assert (got - exp).norm() <= tol * exp.norm(), (name, float((got - exp).norm() / exp.norm()))
        assert (got * ~valid == 0).all(), name
    fin = torch.isfinite(lse_ref)
    assert torch.equal(torch.isfinite(lse.cpu()), fin)
    assert (lse.cpu()[fin] - lse_ref[fin]).abs().max() <= 1e-4
