"""The split planner's two forms: rows in registers (up to 8,192) and rows through its workspace."""
import pytest
import torch

from oracle import vsa_ref as R

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one row; rows of a thread: 1, 7 of 8 (the last threads have none), 8, and more than its registers hold
@pytest.mark.parametrize("heads,nb", [(1, 1), (3, 341), (7, 1000), (16, 512), (24, 400)])
@pytest.mark.parametrize("policy", [{}, dict(min_len=9, rel_mean=1.5, tail_frac=0.001, resident=148, budget=3000)])
def test_plan_of_random_lists(heads, nb, policy):
    """Whole numbers: equal to the oracle's plan."""
    from self_trainable_or_free_attn_b200.vsa import ops
    g = torch.Generator().manual_seed(nb)
    n = torch.randint(0, 12, (1, heads, nb), generator=g) * (1 + 3 * (torch.rand(1, heads, nb, generator=g) < 0.1))
    incl = n.reshape(-1).cumsum(0).reshape(1, heads, nb)
    ptr = torch.cat([(incl - n)[..., :1], incl], 2).to(torch.int32)
    for cap in (40, 10 ** 5):
        tasks, merges, info = ops.split_plan(ptr.to(DEV), 4, cap, **policy)
        t_ref, m_ref, i_ref = R.split_plan(ptr, 4, cap, **policy)
        info = info.cpu().tolist()
        assert info == i_ref
        assert tasks[: info[0]].cpu().tolist() == t_ref and merges[: info[1]].cpu().tolist() == m_ref
