"""Prompt-size GEMM epilogues and dense attention at the edges of their tiles."""
import pytest
import torch

from fastcache_b200 import ops
from fastcache_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _normal(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).to(torch.bfloat16).to(DEV)


def _clean():
    assert ops.ext().read_status(torch.cuda.current_device()) == 0


def _close(got, want, K):
    # one rounding to bf16, and a sum of K products in 32 bits of terms whose mean square is that of the result / K
    bound = 2.0 ** -8 * want.abs() + K * 2.0 ** -24 * want.pow(2).mean().sqrt() + 1e-6
    assert ((got.double() - want).abs() <= bound).all()


@pytest.fixture(params=[0, 1, 2], ids=["one CTA per tile", "CTA pairs", "by size"])
def pairs(request):
    e = ops.ext()
    before = e.gemm_pairs_mode()
    e.set_gemm_pairs(request.param)
    yield request.param
    e.set_gemm_pairs(before)


@pytest.mark.parametrize("M", [257, 384, 1000])
@pytest.mark.parametrize("N,K", [(256, 64), (264, 1024), (328, 2048), (1152, 4304), (3000, 136)])
def test_staged_epilogue_at_ragged_sizes(pairs, M, N, K):
    x, w, b, r = _normal(M, K, seed=1), _normal(N, K, seed=2, scale=K ** -0.5), _normal(N, seed=3), _normal(M, N, seed=4)
    sums = x.double() @ w.double().T + b.double()
    _close(ops.linear(x, w, b), sums, K)
    _close(ops.linear_add(x, w, b, r), sums + r.double(), K)
    wide = torch.full((M, N + 24), 7.0, dtype=torch.bfloat16, device=DEV)          # what lies beside the output stays
    ops.linear(x, w, b, out=wide[:, 8:N + 8])
    _close(wide[:, 8:N + 8], sums, K)
    assert (wide[:, :8] == 7).all() and (wide[:, N + 8:] == 7).all()
    odd = torch.full((M, N + 5), 7.0, dtype=torch.bfloat16, device=DEV)            # a pitch that only the plain epilogue takes
    ops.linear(x, w, b, out=odd[:, :N])
    _close(odd[:, :N], sums, K)
    assert (odd[:, N:] == 7).all()
    _clean()


# two tiles of a CTA and more, where a slab's last store may still be under way, and one tile of several groups of rows
@pytest.mark.parametrize("M,N,K", [(4616, 1024, 1024), (4616, 1024, 4096), (20001, 1032, 320)])
def test_staged_epilogue_of_many_tiles(pairs, M, N, K):
    x, w, b, r = _normal(M, K, seed=1), _normal(N, K, seed=2, scale=K ** -0.5), _normal(N, seed=3), _normal(M, N, seed=4)
    sums = x.double() @ w.double().T + b.double()
    _close(ops.linear(x, w, b), sums, K)
    _close(ops.linear_add(x, w, b, r), sums + r.double(), K)
    _clean()


@pytest.mark.parametrize("M,I,K", [(257, 128, 64), (1000, 384, 1024), (4616, 1024, 1024), (8655, 1024, 1024), (9001, 1152, 64), (300, 640, 2056)])
def test_gated_staged_epilogue(pairs, M, I, K):
    x, w = _normal(M, K, seed=1), _normal(2 * I, K, seed=2, scale=K ** -0.5)
    gate, up = (x.double() @ w.double().T).split(I, dim=1)
    got, want = ops.linear(x, w, None, act="swiglu"), gate * gate.sigmoid() * up
    # both sums carry K 2^-24 of their size; |silu'| <= 1.1; one rounding to bf16, and the fast exponential's 2^-21
    bound = (2.0 ** -8 + 2.0 ** -20) * want.abs() + 1.1 * K * 2.0 ** -24 * (1 + gate.abs()) * (1 + up.abs()) + 1e-6
    assert ((got.double() - want).abs() <= bound).all()
    _clean()


def test_added_residual_of_few_rows_and_other_pitches():
    x, w, b = _normal(300, 256, seed=1), _normal(512, 256, seed=2, scale=0.06), _normal(512, seed=3)
    sums = x.double() @ w.double().T + b.double()
    for rows, r in ((20, _normal(20, 512, seed=4)), (300, _normal(300, 520, seed=5)[:, :512]), (300, _normal(300, 515, seed=6)[:, :512])):
        got = ops.linear_add(x[:rows], w, b, r)
        want = sums[:rows] + r.double()
        assert ((got.double() - want).abs() <= 2.0 ** -7 * (sums[:rows].abs() + want.abs()) + 1e-5).all()      # two roundings at most


@pytest.mark.parametrize("rows", [20, 300])
@pytest.mark.parametrize("form", ["no bias", "batches", "one row for all", "columns", "fp32 residual", "fp32", "gradient"])
def test_added_residual_takes_what_linear_takes(rows, form):
    """Whatever `linear` and an addition behind it take, with their result."""
    x, w, b, r = _normal(rows, 256, seed=1), _normal(512, 256, seed=2, scale=0.06), _normal(512, seed=3), _normal(rows, 512, seed=4)
    if form == "no bias":
        b = None
    elif form == "batches":
        x, r = x.view(2, rows // 2, 256), r.view(2, rows // 2, 512)
    elif form == "one row for all":
        r = r[:1]
    elif form == "columns":                                # both with another unit stride than the kernel's
        x, r = x.t().contiguous().t(), r.t().contiguous().t()
    elif form == "fp32 residual":
        r = r.float()
    elif form == "fp32":
        x, w, b, r = x.float(), w.float(), b.float(), r.float()
    else:
        r.requires_grad_()
    got, want = ops.linear_add(x, w, b, r), r + ops.linear(x, w, b)
    assert got.dtype == want.dtype and got.shape == want.shape and got.requires_grad == want.requires_grad
    # the sum may be rounded once instead of twice
    assert ((got.float() - want.float()).abs() <= 2.0 ** -7 * (want.float().abs() + (want - r).float().abs()) + 1e-5).all()


@pytest.mark.parametrize("D", [8, 40, 64, 72, 80, 96, 128])
@pytest.mark.parametrize("Sq,Sk", [(1, 1), (127, 63), (128, 64), (129, 65), (256, 127), (257, 128), (130, 129), (64, 400)])
def test_dense_attention_at_tile_edges(D, Sq, Sk):
    B, H = 2, 3
    q, k, v = (_normal(B, n, H, D, seed=i) for i, n in enumerate((Sq, Sk, Sk)))
    hole = torch.rand(B, Sk, generator=torch.Generator().manual_seed(9)) < 0.7
    hole[:, Sk // 2] = True
    hole[1, :] = hole[1, :] & (torch.arange(Sk) >= Sk // 2)                         # a first tile without a key
    for mask in (None, hole.to(DEV)):
        got = ops.dense_attention(q, k, v, D ** -0.5, mask, impl=2)
        want = ref.dense_attention(q.float(), k.float(), v.float(), D ** -0.5, mask)
        # P and the result in bf16: 2^-8 of the largest value each
        assert (got.float() - want).abs().max() <= 2 * 2.0 ** -8 * v.float().abs().max()
    nothing = torch.zeros(B, Sk, dtype=torch.bool, device=DEV)
    assert torch.equal(ops.dense_attention(q, k, v, D ** -0.5, nothing, impl=2), torch.zeros_like(q))
    _clean()


@pytest.mark.parametrize("D", [64, 72])
@pytest.mark.parametrize("level", [-20.0, -200.0, 200.0])
def test_first_tiles_without_a_key_before_scores_far_from_zero(D, level):
    """The reference of a row's exponents is its first key's, not zero: no weight may vanish where all scores are low."""
    B, Sq, Sk, H = 2, 130, 400, 2
    q, k, v = (_normal(B, n, H, D, seed=i) for i, n in enumerate((Sq, Sk, Sk)))
    q[..., 0], k[..., 0] = 16.0, level                      # every score is near 16 * level / 8
    mask = torch.ones(B, Sk, dtype=torch.bool, device=DEV)
    mask[0, :128], mask[1, :256] = False, False
    for m in (mask, None):
        got = ops.dense_attention(q, k, v, 0.125, m, impl=2)
        want = ref.dense_attention(q.double(), k.double(), v.double(), 0.125, m)
        # P and the result in bf16 as above, and scores near 2 * level whose sums carry 2^-24 for each product
        assert (got.double() - want).abs().max() <= (2 * 2.0 ** -8 + D * 2.0 ** -24 * 2 * abs(level)) * v.float().abs().max()
    _clean()


@pytest.mark.parametrize("C", [64, 1152])
def test_grid_positions_equal_those_made_on_the_host(C):
    from fastcache_b200.models.vision import _SiglipEmbeddings
    emb = _SiglipEmbeddings(C, 14, 980).to(torch.bfloat16).to(DEV)
    emb.position_embedding.weight.data = _normal(70 * 70, C, seed=5)
    sizes = [[1, 1], [70, 3], [31, 30], [18, 32], [2, 70], [35, 29], [13, 1]]
    N = 1100
    x = _normal(len(sizes), N, C, seed=6)
    want = x + emb.position_embedding.weight[emb.position_ids(torch.tensor(sizes), N).to(DEV)]
    got, counts = emb.add_positions(x, sizes)
    assert torch.equal(got, want) and counts.tolist() == [h * w for h, w in sizes]


def test_one_grid_for_several_slices():
    """A tower takes one row of sizes for a batch of slices that all have them."""
    from types import SimpleNamespace
    from fastcache_b200.models.vision import SiglipVisionTower
    tower = SiglipVisionTower(SimpleNamespace(hidden_size=64, patch_size=14, image_size=140, num_hidden_layers=2, num_attention_heads=4,
                                              intermediate_size=128, layer_norm_eps=1e-6))
    for i, p in enumerate(tower.parameters()):
        p.data = _normal(*p.shape, seed=i, scale=0.1)
    pixels = _normal(3, 3, 56, 70, seed=40)
    one, mask = tower(pixels, torch.tensor([[4, 5]]))
    want, _ = tower(pixels, torch.tensor([[4, 5]] * 3))
    assert mask.shape == (1, 20) and torch.equal(one, want)
