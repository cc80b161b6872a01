"""Decode attention with rings of two and of three tiles: which one runs follows from the number of CTAs, so both need
batches of their own."""
import pytest
import torch

from fastcache_b200 import ops
from helpers import launched

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _normal(*shape, seed):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(torch.bfloat16).to(DEV)


def _statement(q, kc, vc, table, lens, scale):
    B, Hq, D = q.shape
    out = torch.zeros(B, Hq, D, dtype=torch.float64, device=DEV)
    for i, n in enumerate(lens):
        k, v = (c[table[i].long()].transpose(1, 2).flatten(0, 1)[:n].double() for c in (kc, vc))       # [n, Hkv, D]
        k, v = (t.repeat_interleave(Hq // t.shape[1], dim=1) for t in (k, v))
        out[i] = torch.einsum("hn,nhd->hd", (torch.einsum("hd,nhd->hn", q[i].double(), k) * scale).softmax(-1), v)
    return out


@pytest.fixture(params=[False, True], ids=["merge kernel", "merge in the kernel"])
def merge(request):
    e = ops.ext()
    before = e.decode_merge_in_kernel()
    e.set_decode_merge_in_kernel(request.param)
    yield
    e.set_decode_merge_in_kernel(before)


# contexts: one tile, two, three (a ring that wraps), more; ends on and next to the edges of tiles
LENS = [1, 63, 64, 65, 127, 128, 129, 192, 193, 256, 257, 320, 385, 700]


@pytest.mark.parametrize("D,B,Hq,Hkv,bs,splits,stages", [
    (128, 40, 32, 8, 256, 1, 2), (128, 75, 32, 8, 16, 1, 2), (128, 14, 56, 8, 64, 3, 2), (128, 30, 32, 8, 64, 1, 3),
    (128, 60, 8, 8, 32, 1, 3), (64, 160, 4, 2, 16, 1, 2), (64, 56, 24, 2, 64, 3, 2), (64, 56, 24, 2, 64, 2, 3)])
def test_both_rings(merge, D, B, Hq, Hkv, bs, splits, stages):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the batches are made for 148 SMs")
    lens = (LENS * 12)[:B]
    pages = [-(-n // bs) for n in lens]
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(3)).int()
    table, at = torch.zeros(B, max(pages), dtype=torch.int32), 0
    for i, p in enumerate(pages):
        table[i, :p] = order[at:at + p]
        at += p
    kc, vc, q = _normal(at, Hkv, bs, D, seed=1), _normal(at, Hkv, bs, D, seed=2), _normal(B, Hq, D, seed=4)
    table, ctx = table.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV)

    def call():
        return ops.decode_attention(q, kc, vc, table, ctx, D ** -0.5, {"splits": splits})

    first, got = call(), call()
    assert torch.equal(got, first) and ops.ext().read_status(torch.cuda.current_device()) == 0
    want = _statement(q, kc, vc, table, lens, D ** -0.5)
    # weights and result are rounded to bf16 once each: 2^-9 of the largest value, and of the result
    assert ((got.double() - want).abs() <= 2.0 ** -9 * (vc.float().abs().max() + want.abs()) * 1.01 + 1e-5).all()
    name, = launched(call, "decode_attn_kernel")
    assert f"<{D},{stages}>" in name, name


@pytest.mark.parametrize("B,Hkv,bound,splits", [(32, 8, 2048, 1), (32, 8, 2304, 2), (28, 8, 4096, 2), (37, 8, 4096, 1), (27, 8, 1024, 2), (32, 8, 256, 1)])
def test_splits_of_batches_that_leave_sms_with_one_cta(B, Hkv, bound, splits):
    """The rule goes by the bound on the contexts: one long request among short ones is halved."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the batches are made for 148 SMs")
    bs = 64
    table = torch.arange(B * (bound // bs), dtype=torch.int32, device=DEV).view(B, -1) % 40
    kc, vc, q = _normal(40, Hkv, bs, 128, seed=1), _normal(40, Hkv, bs, 128, seed=2), _normal(B, 4 * Hkv, 128, seed=4)
    lens = [bound if i == 3 else 1 + 7 * i for i in range(B)]
    ctx = torch.tensor(lens, dtype=torch.int32, device=DEV)
    got = ops.decode_attention(q, kc, vc, table, ctx, 0.1)
    want = _statement(q, kc, vc, table, lens, 0.1)
    assert ((got.double() - want).abs() <= 2.0 ** -9 * (vc.float().abs().max() + want.abs()) * 1.01 + 1e-5).all()
    names = launched(lambda: ops.decode_attention(q, kc, vc, table, ctx, 0.1), "decode_attn_kernel", "decode_merge_kernel")
    assert any("attn" in n for n in names) and any("merge" in n for n in names) == (splits > 1), names
