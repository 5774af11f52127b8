"""The pair-tile kernels where their rules change over: roots of very small distances, many tiles to a pair of CTAs, both ways to
store rows, and the kernels that problems with few gradient rows are handed to."""
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


@pytest.fixture
def tensor_cores(tpw):
    was = tpw.get_dot_engine()
    tpw.set_dot_engine("tcgen05")
    yield tpw
    tpw.set_dot_engine(was)


@pytest.mark.parametrize("n2", [260, 259])
@pytest.mark.parametrize("scale", [1e-14, 1e-16, 1e-17, 1e-18, 3e-19, 1e-19, 3e-20, 1e-20, 1e-21])
def test_euclidean_root_of_small_distances(tensor_cores, scale, n2):
    """The root of every squared distance, subnormal ones among them, is within one float32 of the exact one: 2^-23 of it."""
    g = torch.Generator().manual_seed(3)
    x1 = torch.randn(300, 64, generator=g) * scale
    x2 = torch.randn(n2, 64, generator=g) * scale
    x2[:200] = x1[:200] * (1 + 0.5 * torch.rand(200, 1, generator=g) ** 8)      # from next to nothing to ordinary distances
    x2[5] = x1[5]
    x1[9], x2[9] = 1.0, 2.0                                                     # ordinary ones in the same warps
    x1, x2 = x1.cuda(), x2.cuda()
    sq, out = tensor_cores.sqeuclidean_distances(x1, x2), tensor_cores.euclidean_distances(x1, x2)
    root = sq.double().sqrt()
    assert bool(((out.double() - root).abs() <= 2 ** -23 * root).all())
    x1[3] = 1e25                                                                # and an infinite one
    sq, out = tensor_cores.sqeuclidean_distances(x1, x2), tensor_cores.euclidean_distances(x1, x2)
    assert bool((out[3] == math.inf).all())
    root = sq.double().sqrt()
    root[3], out[3] = 0, 0
    assert bool(((out.double() - root).abs() <= 2 ** -23 * root).all())
