"""The routing stages at the edges of their split over warps and clusters: block counts around multiples of 32 and 256, ties
across rows, budgets of 0, 1, everything. Lists and bitmaps are whole numbers: exact. Scores against the fp32 oracle: sums of up
to 64 probabilities from the same bf16-rounded means, 1e-3 of the largest (a mean that rounds the other way moves a logit by 2^-9 of its size)."""
import pytest
import torch

from oracle import vsa_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb", [1, 2, 31, 32, 33, 64, 255, 257, 300])
def test_global_topk_lists(nb):
    from self_trainable_or_free_attn_b200.vsa import ops
    g = torch.Generator().manual_seed(nb)
    scores = torch.rand(1, 3, nb, nb, generator=g)
    scores[:, 1] = (scores[:, 1] * 4).floor() / 4                 # many ties, zeros among them
    scores[:, 2] = 0.25
    for budget in sorted({0, 1, min(nb * nb, 3 * nb), nb * nb - 1, nb * nb}):
        sel = ops.global_topk(scores.cuda(), budget)
        mask = R.global_topk_mask(scores, budget)
        qp, qi, kp, ki = R.mask_to_csr(mask)
        assert torch.equal(sel.q2k_ptr.cpu(), qp) and torch.equal(sel.k2q_ptr.cpu(), kp)
        n = 3 * budget
        assert torch.equal(sel.q2k_idx.cpu()[:n], qi) and torch.equal(sel.k2q_idx.cpu()[:n], ki)


@pytest.mark.parametrize("pool", [1, 4, 8, 16, 32, 64])
@pytest.mark.parametrize("nb", [3, 17])
def test_router_scores(pool, nb):
    from self_trainable_or_free_attn_b200.vsa import ops
    g = torch.Generator().manual_seed(pool + nb)
    cnt = torch.randint(1, 65, (nb,), generator=g, dtype=torch.int32)
    valid = R.token_valid(cnt, nb * 64)[None, None, :, None]
    q, k = [(torch.randn(1, 2, nb * 64, 64, generator=g) * valid).to(torch.bfloat16) for _ in range(2)]
    for norm in ("paper", "valid_groups"):
        qr, kr = ops.pool_fwd(q.cuda(), k.cuda(), k.cuda(), cnt.cuda(), pool)[:2]
        got = ops.router_scores(qr, kr, cnt.cuda(), pool, ops.ROW_NORMS[norm]).cpu()
        want = R.psp_scores(q, k, cnt, pool, norm)
        assert (got - want).abs().max() <= 1e-3 * want.abs().max()


@pytest.mark.parametrize("pool", [1, 2, 4, 8, 16, 32, 64])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_router_scores_of_128_columns(pool, dtype):
    """At 128 columns the probabilities take the place of the Q tile. Both types, every group size; several key tiles."""
    from self_trainable_or_free_attn_b200.vsa import ops
    g = torch.Generator().manual_seed(pool)
    nb = 17 if pool < 4 else 33
    cnt = torch.randint(1, 65, (nb,), generator=g, dtype=torch.int32)
    valid = R.token_valid(cnt, nb * 64)[None, None, :, None]
    q, k = [(torch.randn(1, 2, nb * 64, 128, generator=g) * valid).to(dtype) for _ in range(2)]
    for norm in ("paper", "valid_groups"):
        qr, kr = ops.pool_fwd(q.cuda(), k.cuda(), k.cuda(), cnt.cuda(), pool)[:2]
        got = ops.router_scores(qr, kr, cnt.cuda(), pool, ops.ROW_NORMS[norm]).cpu()
        want = R.psp_scores(q, k, cnt, pool, norm, round_to=dtype)
        assert (got - want).abs().max() <= 1e-3 * want.abs().max()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("pool", [1, 8, 16, 32])
def test_router_scores_do_not_depend_on_the_number_of_heads(D, pool):
    """By the number of CTAs another kernel, or another number of them per SM, is launched: the same sums, so the same bits. On 148 SMs
    12 tiles x 52 heads = 624 CTAs are one round of five a SM (D = 64) and two of four; 12 x 40 = 480 one of four (D = 128), two of three."""
    from self_trainable_or_free_attn_b200.vsa import ops
    g = torch.Generator(device="cuda").manual_seed(pool)
    nb, H = 12 * pool, 52 if D == 64 else 40
    cnt = torch.randint(1, 65, (nb,), device="cuda", generator=g, dtype=torch.int32)
    q, k = (torch.randn(1, H, nb * 64, D, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    qr, kr = ops.pool_fwd(q, k, k, cnt, pool)[:2]
    assert qr.shape[2] == 12 * 64
    all_heads = ops.router_scores(qr, kr, cnt, pool)
    few = ops.router_scores(qr[:, -2:].contiguous(), kr[:, -2:].contiguous(), cnt, pool)
    assert torch.equal(all_heads[:, -2:], few) and bool(torch.isfinite(all_heads).all())
