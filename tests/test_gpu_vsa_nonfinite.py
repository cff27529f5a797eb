"""NaN and infinity among the inputs of the VSA2 attention come out as NaN in the rows that attend to them, in O, the LSE and the
gradients, and nowhere else: a diverged step must not look like a healthy one."""
import pytest
import torch

pytestmark = pytest.mark.gpu
NB, BLOCK, TOKEN = 9, 3, 5


def _inputs(D, which, value, seed=0):
    g = torch.Generator().manual_seed(seed)
    x = {n: torch.randn(1, 1, NB * 64, D, generator=g).to(torch.bfloat16).cuda() for n in ("q", "k", "v", "do")}
    # an infinite row gives logits of both signs and NaN, an infinite value infinite outputs
    x[which][0, 0, 64 * BLOCK + TOKEN] = value
    cnt = torch.full((NB,), 64, dtype=torch.int32)
    cnt[::4] = 37
    return x, cnt, g


def _rows(blocks, cnt):
    return (blocks[:, None] & (torch.arange(64)[None] < cnt[:, None])).reshape(-1)


def _one(row):
    m = torch.zeros(NB * 64, dtype=torch.bool)
    m[row] = True
    return m


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("which", ["q", "k", "v"])
@pytest.mark.parametrize("split", [None, 1, 2])
def test_fine_branch(D, value, which, split):
    from self_trainable_or_free_attn_b200 import vsa as V
    x, cnt, g = _inputs(D, which, value)
    mask = torch.rand(1, 1, NB, NB, generator=g) < 0.5
    mask[0, 0, 1] = False                                          # a query block without keys
    mask[0, 0, 2] = False
    mask[0, 0, 2, BLOCK] = True                                    # and one with only that block
    leaves = [x[n].clone().requires_grad_(True) for n in "qkv"]
    o, lse = V.fine_block_sparse_attention(*leaves, cnt.cuda(), V.mask_to_selection(mask.cuda()),
                                           split_kv=None if split is None else V.SplitKV(chunk=split))
    dq, dk, dv = torch.autograd.grad(o, leaves, x["do"])
    bad = _one(64 * BLOCK + TOKEN) if which == "q" else _rows(mask[0, 0, :, BLOCK], cnt)
    if which == "q" and not mask[0, 0, BLOCK].any():
        pytest.skip("nothing attends")
    off = lambda t: ~torch.isfinite(t[0, 0].float().cpu())
    assert torch.equal(off(o).any(1), bad)
    if which != "v":
        assert torch.equal(torch.isnan(lse[0, 0].cpu()), bad)
    # dS of the rows is NaN; P too, where the logits are not finite
    keys = mask[0, 0, BLOCK] if which == "q" else (mask[0, 0] & mask[0, 0, :, BLOCK, None]).any(0)
    assert torch.equal(off(dq).any(1), bad)
    assert torch.equal(off(dk).any(1), _rows(keys, cnt))
    assert torch.equal(off(dv).any(1), _rows(keys, cnt) if which != "v" else torch.zeros(NB * 64, dtype=torch.bool))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("which", ["q", "k", "v"])
def test_tiers_and_whole_operator(D, which):
    from self_trainable_or_free_attn_b200 import vsa as V
    from self_trainable_or_free_attn_b200.vsa import tiers as T
    x, cnt, g = _inputs(D, which, float("nan"))
    a = torch.rand(1, 1, NB, NB, generator=g) < 0.3
    ab = a | (torch.rand(1, 1, NB, NB, generator=g) < 0.4)
    valid = _rows(torch.ones(NB, dtype=torch.bool), cnt)
    bad = _one(64 * BLOCK + TOKEN) if which == "q" else valid      # every row attends to every block in some tier
    leaves = [x[n].clone().requires_grad_(True) for n in "qkv"]
    o, lse = T.rep_fine_attention(*leaves, cnt.cuda(), T.selection_from_masks(a.cuda(), ab.cuda()), mid_reps=4)
    assert torch.equal(torch.isnan(o[0, 0]).any(1).cpu(), bad)
    if which != "v":
        assert torch.equal(torch.isnan(lse[0, 0]).cpu(), bad)
    assert torch.isnan(torch.autograd.grad(o, leaves, x["do"])[0][0, 0]).any(1).cpu()[bad].all()
    # block means: the query block's (one row of the coarse branch), or every row
    o = V.vsa2_attention(x["q"], x["k"], x["v"], None, cnt.cuda(), selection=V.mask_to_selection(a.cuda()))
    rows = _rows(torch.arange(NB) == BLOCK, cnt) if which == "q" else valid
    assert torch.equal(torch.isnan(o[0, 0]).any(1).cpu(), rows)


@pytest.mark.parametrize("phases", [3, 4, 5, 6])
@pytest.mark.parametrize("which", ["k", "v"])
def test_blocks_of_a_tier_left_out(phases, which):
    """With a tier left out a block may not be attended to at all: what it holds does not reach the row, nor its dQ."""
    from self_trainable_or_free_attn_b200.vsa import tiers as T
    x, cnt, g = _inputs(128, which, float("nan"))
    a = torch.rand(1, 1, NB, NB, generator=g) < 0.3
    ab = a | (torch.rand(1, 1, NB, NB, generator=g) < 0.5)
    seen = ((a if phases & 1 else a & False) | (ab & ~a if phases & 2 else a & False) | (~ab if phases & 4 else a & False))[0, 0]
    leaves = [x[n].clone().requires_grad_(True) for n in "qkv"]
    o, _ = T.rep_fine_attention(*leaves, cnt.cuda(), T.selection_from_masks(a.cuda(), ab.cuda()), mid_reps=8, phases=phases)
    dq = torch.autograd.grad(o, leaves, x["do"])[0]
    bad = _rows(seen[:, BLOCK], cnt)
    assert torch.equal(torch.isnan(o[0, 0]).any(1).cpu(), bad)
    assert torch.equal(torch.isnan(dq[0, 0]).any(1).cpu(), bad)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("nb", [70, 1100])
def test_gathered_block_means(D, nb):
    """Tiers A and C alone: gathered rows (tier B left out) against masked tiles (tier B empty). 0, 1, 63 .. 65 and nearly all
    blocks in tier C, over the 1024-block window of the bitmaps. Same columns in another order: P and dS are rounded to bf16
    relative to another maximum, 4e-3 of the 2-norm."""
    from self_trainable_or_free_attn_b200.vsa import tiers as T
    g = torch.Generator(device="cuda").manual_seed(nb)
    q, k, v, do = [torch.randn(1, 1, nb * 64, D, device="cuda", generator=g).to(torch.bfloat16) for _ in range(4)]
    cnt = torch.randint(1, 65, (nb,), device="cuda", generator=g, dtype=torch.int32)
    n_c = torch.tensor([[0, 1, 63, 64, 65, nb - 2, nb - 1][i % 7] for i in range(nb)], device="cuda")
    a = (torch.rand(nb, nb, device="cuda", generator=g).argsort(1).argsort(1) >= n_c[:, None])[None, None]
    sel = T.selection_from_masks(a, a)
    outs = []
    for phases in (7, 5):
        x = [t.clone().requires_grad_(True) for t in (q, k, v)]
        o, lse = T.rep_fine_attention(*x, cnt, sel, mid_reps=4, phases=phases)
        outs.append([o, *torch.autograd.grad(o, x, do), lse])
    for name, full, gathered in zip(("o", "dq", "dk", "dv"), *outs):
        full, gathered = full.float(), gathered.float()
        assert (full - gathered).norm() <= 4e-3 * full.norm(), (name, float((full - gathered).norm() / full.norm()))
    fin = torch.isfinite(outs[0][4])
    assert torch.equal(fin, torch.isfinite(outs[1][4])) and (outs[0][4] - outs[1][4])[fin].abs().max() <= 1e-4
