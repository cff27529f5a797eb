"""Flagged tiles shared out by the CTAs of the fallback kernels themselves, against one CTA per tile that tests its own flag."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# no flag, every flag, fewer tiles than SMs; 25,000 tiles: the flags in two ranges (24,576 tiles each), few and all of them
@pytest.mark.parametrize("L,H,share", [(200, 3, 0.0), (200, 3, 1.0), (4152, 5, 0.3), (64, 25000, 0.004), (64, 25000, 1.0)])
def test_walk_equals_one_cta_per_tile(L, H, share):
    """The same tiles are computed by the same code, so the bits are the same; tiles without a flag keep what they hold."""
    from self_trainable_or_free_attn_b200 import _native as N
    lib = N.load()
    g = torch.Generator(device=DEV).manual_seed(L + H)
    nq, nb = -(-L // 128), -(-L // 64)
    q, k, v = (torch.randn(L, H, 128, device=DEV, generator=g, dtype=torch.bfloat16) for _ in range(3))
    km, vm = (torch.randn(nb, H, 128, device=DEV, generator=g, dtype=torch.bfloat16) for _ in range(2))
    counts = torch.full((nq, H), nb, device=DEV, dtype=torch.int32)
    blocks = torch.arange(nb, device=DEV, dtype=torch.int32).expand(nq, H, nb).contiguous()
    keep = (torch.rand(H, nq, nb, device=DEV, generator=g) < 0.5).to(torch.uint8)
    flags = (torch.rand(nq, H, device=DEV, generator=g) < share).to(torch.int32) * 3
    res = []
    for scratch in (torch.empty(nq * H + 1, device=DEV, dtype=torch.int32), None):
        out, lse = torch.full_like(q, 7.0), torch.full((nq * 128, H), 5.0, device=DEV)
        N.check(lib.es_exact_fallback(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), counts.data_ptr(),
                                      blocks.data_ptr(), nb, lse.data_ptr(), flags.data_ptr(), L, H, N.ptr(scratch),
                                      N.stream_ptr()), "exact")
        N.check(lib.es_compensate_fallback(q.data_ptr(), km.data_ptr(), vm.data_ptr(), keep.data_ptr(), lse.data_ptr(),
                                           out.data_ptr(), flags.data_ptr(), L, H, N.ptr(scratch), N.stream_ptr()), "compensate")
        res.append((out, lse))
    assert N.device_status() == 0
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
    rows = (flags > 0).repeat_interleave(128, 0)
    assert (res[0][1][~rows] == 5.0).all() and (res[0][0][~rows[:L]] == 7.0).all()
    assert share == 0.0 or (res[0][0][rows[:L]] != 7.0).any(1).all()
