"""Kernels that only stream rows (quantisers, eviction, norms, rotary store), at the sizes where their splits of the work
have edges."""
import pytest
import torch

from fastcache_b200 import ops
from fastcache_b200.compress import quant
from fastcache_b200.ops import reference as ref
from helpers import launched

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _normal(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(torch.bfloat16)


def _status():
    return ops.ext().status_tensor(torch.cuda.current_device())


@pytest.mark.parametrize("mode", ["int8", "int8_asym", "int4", "nf4", "fp8_e4m3", "fp8_e5m2"])
@pytest.mark.parametrize("g", [8, 24, 64, 128, 256, 264, 1024])
def test_codes_equal_the_division_where_the_quotient_is_near_a_border(mode, g):
    """Codes come from x * (1 / a) unless that is close to the border between two codes: they have to be those of the
    division, for values on and next to the borders, rows of one value, and scales at both ends of the range."""
    n = 601
    x = _normal(n, g, seed=g)
    steps = {"int8": 127, "int8_asym": 255, "int4": 7}.get(mode, 448)
    x[1::5] = ((torch.randint(-2 * steps, 2 * steps + 1, (n, g), generator=torch.Generator().manual_seed(1)) * 0.5) / steps).bfloat16()[1::5]
    x[2::5] = (x[2::5].float() * 2.0 ** torch.randint(-120, 120, (n, 1), generator=torch.Generator().manual_seed(2))[2::5]).bfloat16()
    x[3] = 0
    x[4] = 3.0
    x[8] = 1e-30
    x[9, 0] = torch.finfo(torch.bfloat16).max
    want, got = quant.quantize(x, mode, g), quant.quantize(x.to(DEV), mode, g)
    assert torch.equal(got["scale"].cpu(), want["scale"])
    assert torch.equal(got["q"].cpu().view(torch.uint8), want["q"].view(torch.uint8))
    assert torch.equal(quant.dequantize(got).cpu(), quant.dequantize(want))


# groups per block of the form for many (which takes more than four blocks an SM), and lanes and pieces per lane of both forms
@pytest.mark.parametrize("mode", ["int8", "int8_asym", "int4", "nf4", "fp8_e4m3", "fp8_e5m2"])
@pytest.mark.parametrize("g,per_block,many,few", [(8, 256, "4,1", "4,1"), (40, 256, "4,2", "8,1"), (64, 256, "4,2", "8,1"), (72, 128, "8,2", "16,1"),
                                                  (128, 128, "8,2", "16,1"), (136, 64, "16,2", "32,1"), (256, 64, "16,2", "32,1")])
def test_many_groups_and_few_give_the_same_codes(mode, g, per_block, many, few):
    n = 4 * torch.cuda.get_device_properties(0).multi_processor_count * per_block + 3
    x = _normal(n, g, seed=g).to(DEV)
    got = quant.quantize(x, mode, g)
    parts = [quant.quantize(x[a:a + n // 2], mode, g) for a in range(0, n, n // 2)]
    for k in ("q", "scale") + (("zero",) if mode == "int8_asym" else ()):
        assert torch.equal(got[k].view(torch.uint8), torch.cat([p[k] for p in parts]).view(torch.uint8))
    for rows, form in ((x, f",{many},false>"), (x[3:], f",{few},true>")):
        name, = launched(lambda: quant.quantize(rows, mode, g), "quantize_kernel")
        assert form in name, name


@pytest.mark.parametrize("D,Hkv,block", [(128, 8, 256), (128, 3, 16), (64, 2, 64)])
@pytest.mark.parametrize("ties", [False, True])
def test_select_compact_keeps_the_k_best_rows_in_order(D, Hkv, block, ties):
    lens = [1, 2, 255, 256, 257, 1023, 1300, 700, 512]
    kept = [1, 1, 254, 128, 1, 600, 1299, 700, 0]
    L, pages = 2, [-(-n // block) for n in lens]
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(3)).int()
    table, at = torch.zeros(len(lens), max(pages), dtype=torch.int32), 0
    for i, p in enumerate(pages):
        table[i, :p] = order[at:at + p]
        at += p
    pool = _normal(L, 2, sum(pages), Hkv, block, D, seed=4)
    stride = (max(lens) + 3) // 4 * 4
    scores = torch.randn(len(lens), L, Hkv, stride, generator=torch.Generator().manual_seed(5))
    if ties:
        scores = (scores * 2).round() + 0.0          # no -0.0, which the kernel ranks below 0.0
    want = pool.clone()
    for i, (n, k) in enumerate(zip(lens, kept)):
        if k >= n:
            continue
        at = [(int(table[i, r // block]), r % block) for r in range(n)]
        for layer in range(L):
            for h in range(Hkv):
                best = sorted(range(n), key=lambda r: (float(scores[i, layer, h, r]), r))[-max(1, k):]
                for j, r in enumerate(sorted(best)):
                    want[layer, :, at[j][0], h, at[j][1]] = pool[layer, :, at[r][0], h, at[r][1]]
    got = pool.to(DEV)
    ops.ext().select_compact(got, scores.to(DEV), table.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV),
                             torch.tensor(kept, dtype=torch.int32, device=DEV), _status())
    assert torch.equal(got.cpu(), want)


@pytest.mark.parametrize("D,Hkv", [(128, 8), (128, 16), (128, 6), (64, 8)])
@pytest.mark.parametrize("mode", [0, 1])
def test_key_norm_scores(D, Hkv, mode):
    lens, block = [1, 31, 33, 300], 16
    pages = [-(-n // block) for n in lens]
    table, at = torch.zeros(len(lens), max(pages), dtype=torch.int32), 0
    for i, p in enumerate(pages):
        table[i, :p] = torch.arange(at, at + p)
        at += p
    pool = _normal(2, 2, sum(pages), Hkv, block, D, seed=6)
    got = ops.ext().knorm_scores(pool.to(DEV), table.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), max(lens), mode, _status()).cpu()
    for i, n in enumerate(lens):
        rows = pool[:, 0, table[i, : pages[i]].long()].double().transpose(1, 2).flatten(2, 3)[:, :, :n]     # [L, Hkv, n, D]
        norm = rows.norm(dim=-1)
        want = -norm if mode == 0 else norm.mean(1, keepdim=True).expand_as(norm)
        # sums of D + Hkv terms in 32 bits: 2^-24 each
        torch.testing.assert_close(got[i, :, :, :n].double(), want, rtol=(D + Hkv) * 2.0 ** -24, atol=0)


@pytest.mark.parametrize("T", [1, 7, 8, 9, 300])
@pytest.mark.parametrize("H", [8, 256, 1024, 1032, 1152, 1280, 1288, 2048, 2056, 3584, 4096, 4104, 8192])
def test_layer_norm_row_lengths(T, H):
    x, w, b = (_normal(*s, seed=i) for i, s in enumerate([(T, H), (H,), (H,)]))
    x = x + 3
    got = ops.layer_norm(x.to(DEV), w.to(DEV), b.to(DEV), 1e-5).cpu().double()
    want = torch.nn.functional.layer_norm(x.double(), (H,), w.double(), b.double(), 1e-5)
    # one rounding to bf16, and 32-bit sums
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()


# a warp per row where there are more than five rows an SM, a block per row for fewer and for long rows
@pytest.mark.parametrize("rows,H,kernel", [(5, 512, "<4>"), (5, 520, "block"), (5, 1280, "block"), (6, 520, "<4>"), (6, 1032, "<5>"), (6, 1288, "<8>"),
                                           (6, 2048, "<8>"), (6, 2056, "block"), (6, 3584, "block")])
def test_layer_norm_by_rows_per_sm(rows, H, kernel):
    T = rows * torch.cuda.get_device_properties(0).multi_processor_count
    x, w, b = (_normal(*s, seed=i) for i, s in enumerate([(T, H), (H,), (H,)]))
    xd, wd, bd = (x + 3).to(DEV), w.to(DEV), b.to(DEV)
    want = torch.nn.functional.layer_norm(xd.double(), (H,), wd.double(), bd.double(), 1e-5)
    # one rounding to bf16, and 32-bit sums
    assert ((ops.layer_norm(xd, wd, bd, 1e-5).double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4).all()
    name, = launched(lambda: ops.layer_norm(xd, wd, bd, 1e-5), "layer_norm")
    assert kernel in name, name


@pytest.mark.parametrize("Hq,Hkv", [(32, 8), (32, 32), (5, 3), (12, 2)])
@pytest.mark.parametrize("norm", [False, True])
def test_rotary_store_of_many_rows_equals_that_of_few(Hq, Hkv, norm):
    """The prompt form (several heads per group of lanes) against the other one, which few rows take: bit for bit."""
    heads, block = Hq + 2 * Hkv, 16
    T = -(-16 * 148 * 48 // heads) + 3
    qkv = _normal(T, heads * 128, seed=7).to(DEV)
    pos = torch.randint(0, 500, (T,), generator=torch.Generator().manual_seed(8)).to(DEV)
    angle = torch.rand(500, 64, generator=torch.Generator().manual_seed(9)) * 6
    cs = torch.cat([angle.cos(), angle.sin()], 1).to(DEV)
    qw, kw = (_normal(128, seed=s).to(DEV) if norm else None for s in (10, 11))
    slots = torch.randperm(T + 5, generator=torch.Generator().manual_seed(12))[:T].int()
    slots[::17] = -1
    slots = slots.to(DEV)
    blocks = -(-(T + 5) // block)
    pools = [torch.zeros(2, blocks, Hkv, block, 128, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    q = ops.rope_qknorm_store(qkv, pos, cs, Hq, Hkv, 128, qw, kw, 1e-6, pools[0][0], pools[0][1], slots)
    few = [ops.rope_qknorm_store(qkv[a:a + 64], pos[a:a + 64], cs, Hq, Hkv, 128, qw, kw, 1e-6, pools[1][0], pools[1][1], slots[a:a + 64])
           for a in range(0, T, 64)]
    assert torch.equal(q, torch.cat(few)) and torch.equal(pools[0], pools[1])


# tokens x heads per SM; several heads per group of lanes for many rows of well filled warps without norms only, loads ahead of
# qkv for few rows only
@pytest.mark.parametrize("Hq,Hkv,per_sm,norm,kernel", [(32, 8, 95, False, "d128_kernel<true>"), (32, 8, 97, False, "d128_kernel<false>"),
                                                       (14, 2, 97, True, "d128_kernel<false>"), (32, 8, 770, False, "rows_kernel"),
                                                       (32, 8, 770, True, "d128_kernel<false>"), (14, 2, 770, False, "d128_kernel<false>"),
                                                       (16, 4, 770, False, "rows_kernel")])
def test_rotary_store_by_rows_per_sm(Hq, Hkv, per_sm, norm, kernel):
    heads, block = Hq + 2 * Hkv, 16
    T = per_sm * torch.cuda.get_device_properties(0).multi_processor_count // heads
    qkv, pos = _normal(T, heads * 128, seed=7).to(DEV), torch.randint(0, 500, (T,), generator=torch.Generator().manual_seed(8)).to(DEV)
    angle = torch.rand(500, 64, generator=torch.Generator().manual_seed(9)) * 6
    cs = torch.cat([angle.cos(), angle.sin()], 1).to(DEV)
    qw, kw = (_normal(128, seed=s).to(DEV) if norm else None for s in (10, 11))
    slots = torch.randperm(T + 5, generator=torch.Generator().manual_seed(12))[:T].int()
    slots[::17] = -1
    slots = slots.to(DEV)
    pools = [torch.zeros(2, -(-(T + 5) // block), Hkv, block, 128, dtype=torch.bfloat16, device=DEV) for _ in range(2)]
    args = (qkv, pos, cs, Hq, Hkv, 128, qw, kw, 1e-6)
    q = ops.rope_qknorm_store(*args, pools[0][0], pools[0][1], slots)
    few = [ops.rope_qknorm_store(qkv[a:a + 32], pos[a:a + 32], *args[2:], pools[1][0], pools[1][1], slots[a:a + 32]) for a in range(0, T, 32)]
    assert torch.equal(q, torch.cat(few)) and torch.equal(pools[0], pools[1])
    name, = launched(lambda: ops.rope_qknorm_store(*args, pools[0][0], pools[0][1], slots), "rope_")
    assert kernel in name, name
