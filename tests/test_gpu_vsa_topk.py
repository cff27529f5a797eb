"""The global top-k, as one cluster per head and as a launch per stage, against a stable sort."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one launch: one block; a word and one column; rows of 256 warps and one more; the largest. Seven: one block more, more rows than
# threads, more heads than clusters at once
@pytest.mark.parametrize("nb,H", [(1, 3), (33, 18), (257, 3), (384, 2), (385, 2), (1100, 3), (33, 19)])
@pytest.mark.parametrize("kind", ["random", "ties", "zeros"])
def test_lists_match_a_stable_sort(nb, H, kind):
    """Score descending, ties to the smaller flat index: the lists are whole numbers and have to be equal."""
    from self_trainable_or_free_attn_b200.vsa import ops
    g = torch.Generator(device=DEV).manual_seed(nb)
    B = 1
    s = torch.rand(B, H, nb, nb, device=DEV, generator=g)
    if kind == "ties":
        s = (s * 7).floor() / 7
    if kind == "zeros":
        s = torch.where(s < 0.9, torch.zeros_like(s), s)
    for budget in {0, 1, nb * nb // 3, nb * nb}:
        sel = ops.global_topk(s, budget)
        order = s.reshape(B * H, -1).sort(dim=1, descending=True, stable=True).indices[:, :budget]
        mask = torch.zeros(B * H, nb * nb, device=DEV, dtype=torch.bool).scatter_(1, order, True).reshape(B * H, nb, nb)
        for ptr, idx, m in ((sel.q2k_ptr, sel.q2k_idx, mask), (sel.k2q_ptr, sel.k2q_idx, mask.transpose(1, 2))):
            cnt = m.sum(2)
            want = torch.cat([cnt.cumsum(1) - cnt, cnt.sum(1, keepdim=True)], 1) + budget * torch.arange(B * H, device=DEV)[:, None]
            assert torch.equal(ptr.reshape(B * H, nb + 1).long(), want)
            assert torch.equal(idx[: B * H * budget].long(), m.nonzero()[:, 2])
