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


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("nb", [1, 63, 64, 65, 130])
def test_coarse_branch(D, nb):
    """The dense attention of the block means, without lists: one tile, full and ragged last tiles; padding gives 0 and -inf."""
    from self_trainable_or_free_attn_b200.vsa import ops
    g = torch.Generator().manual_seed(nb)
    L = -(-nb // 64) * 64
    q, k, v, do = [torch.randn(1, 2, L, D, generator=g).to(torch.bfloat16) for _ in range(4)]
    for x in (q, k, v, do):
        x[:, :, nb:] = 0
    ref = [x[:, :, :nb].double().requires_grad_(True) for x in (q, k, v)]
    s = ref[0] @ ref[1].transpose(-1, -2) / D ** 0.5
    o_ref = torch.softmax(s, -1) @ ref[2]
    o_ref.backward(do[:, :, :nb].double())
    o, lse = ops._coarse_fwd(q.cuda(), k.cuda(), v.cuda(), nb)
    delta = (o.float() * do.cuda().float()).sum(-1)
    grads = ops._coarse_bwd(q.cuda(), k.cuda(), v.cuda(), do.cuda(), lse, delta, nb)
    assert (lse.cpu()[:, :, :nb] - torch.logsumexp(s, -1).detach()).abs().max() <= 1e-4
    assert torch.isneginf(lse[:, :, nb:]).all() and (o[:, :, nb:] == 0).all()
    for got, exp in [(o, o_ref)] + [(x, y.grad) for x, y in zip(grads, ref)]:
        got, exp = got.double().cpu()[:, :, :nb], exp.detach()
        # nb = 1: softmax of one score, dq and dk are rounding errors of 0
        assert (got - exp).norm() <= 1e-2 * exp.norm() + (0.3 if nb == 1 else 0.0)
    for x in grads:
        assert (x[:, :, nb:] == 0).all()


@pytest.mark.parametrize("mode", ["token", "elem"])
def test_fusion_of_unaligned_gates(mode):
    """A gate that starts at 4 bytes of a 16-byte line takes the narrow loads: the same bits."""
    from self_trainable_or_free_attn_b200 import vsa as V
    g = torch.Generator().manual_seed(5)
    nb, D = 6, 128
    q, k, v, do = [torch.randn(1, 2, nb * 64, D, generator=g).to(torch.bfloat16).cuda() for _ in range(4)]
    cnt = torch.tensor([64, 1, 63, 17, 64, 40], dtype=torch.int32).cuda()
    sel = V.mask_to_selection(torch.rand(1, 2, nb, nb, generator=g).cuda() < 0.5)
    shape = q.shape[:3] if mode == "token" else q.shape
    flat = torch.randn(q.numel() + 2, generator=g).to(torch.bfloat16).cuda()
    outs = []
    for shift in (0, 2):
        n = q[..., 0].numel() if mode == "token" else q.numel()
        buf = torch.empty(n + 8, device="cuda", dtype=torch.bfloat16)
        gate = buf[shift: shift + n].copy_(flat[:n]).view(shape).requires_grad_(True)
        x = [t.clone().requires_grad_(True) for t in (q, k, v)]
        o = V.vsa2_attention(*x, gate, cnt, selection=sel)
        outs.append([o, *torch.autograd.grad(o, x + [gate], do)])
    for a, b in zip(*outs):
        assert torch.equal(a, b)
