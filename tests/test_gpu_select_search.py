"""The K-th largest key of a (tile, head): the search that ends with the first threshold that exactly K keys reach against the
oracle's 31 halvings, bit for bit, over every lane count of the warp kernel (8, 16, 24, 32, 40, 48 and 64 keys a lane), the kernel
of one CTA per (tile, head) that takes over above 2,048 blocks, and rows where keys tie at the cut, are zero, NaN or infinite. The
plan packed from a selection gives its lists back."""
import pytest
import torch

from oracle import echosparse_ref as R

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nb,k,r,sink", [(65, 7, 19, 1 << 30), (256, 1, 0, 1 << 30), (301, 30, 90, 297), (513, 500, 13, 511),
                                         (1003, 100, 301, 1 << 30), (1024, 1, 1023, 1 << 30), (1182, 118, 355, 1 << 30),
                                         (1281, 128, 384, 1 << 30), (1536, 1535, 1, 1 << 30), (1861, 223, 545, 1856),
                                         (2048, 2048, 0, 1 << 30), (2049, 205, 615, 1 << 30), (2503, 0, 250, 2501),
                                         (4096, 4000, 96, 1 << 30)])
def test_selection_equals_the_oracle(nb, k, r, sink):
    from self_trainable_or_free_attn_b200.kernels import sm100 as K
    L, H = nb * 64 - 5, 2
    nq = R.cdiv(L, 128)
    g = torch.Generator(device=DEV).manual_seed(nb)
    mass = torch.rand(H, nq, nb, device=DEV, generator=g).pow(8)
    mass[:, 1::7] = (mass[:, 1::7] * 8).round() / 8                # ties at every cut
    mass[:, 2::7, ::3] = 0.0
    mass[:, 3::7] = 0.25
    mass[0, 4::7, 5] = float("nan")
    mass[1, 5::7, 6::11] = float("inf")
    keep_prev = (torch.rand(H, nq, nb, device=DEV, generator=g) < 0.2).to(torch.uint8)
    se, ss = (torch.rand(H, nq, device=DEV, generator=g) + 0.5 for _ in range(2))
    flags = (torch.rand(nq, H, device=DEV, generator=g) < 0.1).to(torch.int32)
    rw = R.cdiv(r, 32) * 32
    keep = torch.full((H, nq, nb), 9, device=DEV, dtype=torch.uint8)
    counts = torch.full((nq, H), -1, device=DEV, dtype=torch.int32)
    blocks = torch.zeros(nq, H, nb, device=DEV, dtype=torch.int32)
    bits = torch.full((H, nq, R.plan_words(nb)), -1, device=DEV, dtype=torch.int32)
    refine = torch.full((nq, H, rw), -5, device=DEV, dtype=torch.int32)
    K.select_blocks(mass, keep_prev, se, ss, keep, counts, blocks, flags, bits, refine, k, r, L, sink=sink)
    want = R.select_blocks(mass, keep_prev, se, ss, flags, k, r, L, rw, sink=sink)
    assert torch.equal(keep, want[0]) and torch.equal(counts, want[1])
    live = torch.arange(nb, device=DEV)[None, None] < counts[:, :, None]
    assert torch.equal(blocks[live], want[2][live])
    assert torch.equal(bits, want[3]) and torch.equal(refine, want[4])
    # the plan of the selection, expanded again
    exact = torch.zeros_like(bits)
    K.pack_plan(keep, exact)
    again = [torch.full_like(keep, 9), torch.zeros_like(counts), torch.zeros_like(blocks), torch.zeros_like(refine)]
    listed = torch.zeros_like(counts)
    K.rebuild_plan(exact, bits, *again, listed)
    assert torch.equal(again[0], keep) and torch.equal(again[1], counts) and torch.equal(again[2][live], blocks[live])
    assert torch.equal(again[3], refine) and torch.equal(listed, (refine < nb).sum(2).to(torch.int32))
