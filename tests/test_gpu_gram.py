"""Gram matrix and probes of es_reps_metric / es_reps_metric_static against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one row, a whole tile, one row more, the last tile of a split ragged; 20,000 rows: ten tiles a split, more than the ring holds;
# 130 heads of the scratch-free variant: one split each, 47 tiles
@pytest.mark.parametrize("L,H,static", [(1, 1, False), (64, 2, False), (65, 1, False), (4152, 3, False), (20000, 2, False), (3000, 130, True)])
def test_gram_and_probes(L, H, static):
    """bf16 products are exact in float32; a split of n rows is a float32 sum of n of them: at worst n 2^-24 of the sum of their
    magnitudes, here 2,944 rows at most, with the products of random rows far from adding up: 2e-5 of the largest entry. A probe is
    a mean of 64 bf16 rows rounded to bf16: 2^-8 of its largest value."""
    from self_trainable_or_free_attn_b200 import _native as N
    lib = N.load()
    g = torch.Generator(device=DEV).manual_seed(L)
    q = (torch.randn(L, H, 128, device=DEV, generator=g) + torch.randn(1, H, 128, device=DEV, generator=g)).to(torch.bfloat16)
    gram = torch.empty(H, 128, 128, device=DEV)
    metric = torch.empty(H, 128, 128, device=DEV, dtype=torch.bfloat16)
    probes = torch.full((H, 64, 128), 7.0, device=DEV, dtype=torch.bfloat16)
    if static:
        N.check(lib.es_reps_metric_static(q.data_ptr(), gram.data_ptr(), metric.data_ptr(), probes.data_ptr(), L, H, N.stream_ptr()), "s")
    else:
        parts = torch.empty(lib.es_reps_gram_splits(L), H, 128, 128, device=DEV)
        N.check(lib.es_reps_metric(q.data_ptr(), parts.data_ptr(), gram.data_ptr(), metric.data_ptr(), probes.data_ptr(), L, H,
                                   N.stream_ptr()), "m")
    assert N.device_status() == 0
    want = torch.einsum("lhi,lhj->hij", q.double(), q.double()) / (128 * L)
    want += 1e-3 * want.diagonal(dim1=1, dim2=2).mean(1)[:, None, None] * torch.eye(128, device=DEV, dtype=torch.float64)
    assert (gram - want).abs().max() <= 2e-5 * want.abs().max()
    nb = -(-L // 64)
    for i in range(64):
        b = int(i * (nb - 1) / 63 + 0.5)
        mean = q[64 * b: 64 * b + 64].double().mean(0) / 128 ** 0.5
        assert (probes[:, i].double() - mean).abs().max() <= 2 ** -8 * mean.abs().max()
