"""Edges of the 256 x 256 tiles that two CTAs share, of their two ways to store rows, and of the widening copy."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tpw():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import torchpairwise_b200
    torchpairwise_b200.load_torch_ops()
    return torchpairwise_b200


SIZES = [(128, 256), (129, 257), (255, 300), (256, 259), (257, 511), (385, 130), (700, 1026)]


@pytest.mark.parametrize("n1,n2", SIZES)
@pytest.mark.parametrize("d", [64, 72, 65, 200])
def test_contractions_at_tile_edges(tpw, n1, n2, d):
    """The three-product split drops at most 2^-15 |x| |y| of a dot product (2^-17 of each factor, and the product of the low parts);
    float32 sums of d terms and the epilogue add (d + 8) 2^-24 of |x|^2 + |y|^2."""
    g = torch.Generator().manual_seed(n1 * n2 + d)
    x1, x2 = torch.randn(n1, d, generator=g).cuda(), torch.randn(n2, d, generator=g).cuda()
    a, b = x1.double(), x2.double()
    na, nb = a.norm(dim=1)[:, None], b.norm(dim=1)[None]
    bound = 2 ** -14 * na * nb + (d + 8) * 2 ** -24 * (na ** 2 + nb ** 2)
    sq = torch.cdist(a, b, compute_mode="donot_use_mm_for_euclid_dist") ** 2
    was = tpw.get_dot_engine()
    tpw.set_dot_engine("tcgen05")
    try:
        assert bool(((tpw.sqeuclidean_distances(x1, x2) - sq).abs() <= bound).all())
        out = tpw.euclidean_distances(x1, x2)
        assert bool(((out.double() ** 2 - sq).abs() <= 1.01 * bound + 2 ** -22 * sq).all())
        cos = 1 - (a @ b.T) / (na * nb)
        assert bool(((tpw.cosine_distances(x1, x2) - cos).abs() <= bound / (na * nb)).all())
        own = tpw.sqeuclidean_distances(x1, x1)
        assert bool((own.diagonal() == 0).all())
    finally:
        tpw.set_dot_engine(was)


def test_euclidean_root_of_infinite_zero_and_tiny_distances(tpw):
    """The root by Newton's step covers finite arguments, a warp with an infinite one takes sqrtf."""
    x1 = torch.randn(300, 64, generator=torch.Generator().manual_seed(1)).cuda()
    x2 = x1[:260].repeat(1, 1).clone()
    x1[3] = 1e25
    x2[7] = 3e19
    was = tpw.get_dot_engine()
    tpw.set_dot_engine("tcgen05")
    try:
        out = tpw.euclidean_distances(x1, x2)
        sq = tpw.sqeuclidean_distances(x1, x2)
        far = torch.zeros_like(out, dtype=torch.bool)
        far[3], far[:, 7], far[3, 7] = True, True, False      # inf - inf between the two: clamped to 0
        assert bool((out[far] == math.inf).all())
        fine = sq.isfinite()
        root = sq[fine].double().sqrt()
        assert bool(((out[fine].double() - root).abs() <= 2 ** -23 * root).all())
        assert bool((out[sq == 0] == 0).all()) and not bool(out.isnan().any())
        small = tpw.euclidean_distances(x1[10:200] * 1e-15, x2[10:] * 1e-15), tpw.sqeuclidean_distances(x1[10:200] * 1e-15, x2[10:] * 1e-15)
        assert bool(((small[0].double() - small[1].double().sqrt()).abs() <= 2 ** -23 * small[1].double().sqrt()).all())
    finally:
        tpw.set_dot_engine(was)


@pytest.mark.parametrize("n1,n2", SIZES)
@pytest.mark.parametrize("d", [167, 1024, 2050])
def test_boolean_counts_at_tile_edges(tpw, n1, n2, d):
    """Counts are exact integers, and every quotient is the correctly rounded one."""
    reps = max(1, math.ceil((1 << 28) / (n1 * n2 * d)))     # enough pairs for the tensor cores
    g = torch.Generator().manual_seed(d)
    x1, x2 = (torch.rand(reps, n1, d, generator=g) < 0.2).cuda(), (torch.rand(reps, n2, d, generator=g) < 0.2).cuda()
    x1[:, 5] = False
    x2[:, 9] = False
    both = x1.float() @ x2.float().transpose(1, 2)          # below 2^24: exact
    a, b = x1.float().sum(2)[..., None], x2.float().sum(2)[:, None]
    union, differ = a + b - both, a + b - 2 * both
    zero = torch.zeros((), device="cuda")
    assert torch.equal(tpw.jaccard_distances(x1, x2), torch.where(union == 0, zero, differ / union))
    assert torch.equal(tpw.hamming_distances(x1, x2), differ / torch.tensor(float(d), device="cuda"))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 2047, 2048 * 148 * 16 * 8 // 16 + 5])
def test_widen_is_exact(tpw, dtype, n):
    from torchpairwise_b200 import _abi
    x = torch.randn(n, generator=torch.Generator().manual_seed(n)).to(dtype).cuda()
    x[0] = math.inf
    out = torch.full((n + 4,), 7.0, device="cuda")
    _abi.check(_abi.lib.tpw_widen(int(dtype == torch.bfloat16), x.data_ptr(), out.data_ptr(), n, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(out[:n], x.float()) and bool((out[n:] == 7).all())
    assert _abi.lib.tpw_widen(1, x.data_ptr() + 2, out.data_ptr(), 1, None) == 1     # not 16-byte aligned: refused


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_narrow_views_equal_contiguous_inputs(tpw, dtype):
    """Views, rows off the 16-byte grid among them, go through the general converting copy: same results."""
    x = torch.randn(41, 70, generator=torch.Generator().manual_seed(2)).to(dtype).cuda()
    y = torch.randn(33 * 68 + 1, generator=torch.Generator().manual_seed(3)).to(dtype).cuda()
    off, view = y[1:].view(33, 68), x[:, 1:69]
    assert torch.equal(tpw.manhattan_distances(view, off), tpw.manhattan_distances(view.contiguous(), off.clone()))
