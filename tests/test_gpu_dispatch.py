"""The Python functions and the dispatcher's operators as torch programs call them: below autograd, under its checks, with its
tensor types and modes."""
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


def _inputs(lead=(), seed=1):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(*lead, 40, 12, generator=g).cuda(), torch.randn(*lead, 33, 12, generator=g).cuda()


BOTH = ["euclidean_distances", "manhattan_distances", "chebyshev_distances", "minkowski_distances", "sqeuclidean_distances", "cosine_distances",
        "cosine_similarity", "correlation_distances", "linear_kernel", "canberra_distances", "jaccard_distances"]


@pytest.mark.parametrize("layer", ["python", "dispatcher"])
@pytest.mark.parametrize("name", BOTH)
def test_calls_below_autograd(tpw, layer, name):
    """Inference mode and the body of a custom operator dispatch below autograd: the same values as under no_grad."""
    fn = getattr(tpw if layer == "python" else torch.ops.torchpairwise, name)
    f = (lambda a, b: fn(a > 0, b > 0)) if name == "jaccard_distances" else fn
    x1, x2 = _inputs()
    with torch.no_grad():
        want, narrow = f(x1, x2), f(x1.bfloat16(), x2.bfloat16())
    with torch.inference_mode():
        assert torch.equal(f(x1, x2), want)
        assert torch.equal(f(x1.clone(), x2.clone()), want)
        assert torch.equal(f(x1.bfloat16(), x2.bfloat16()), narrow)

    @torch.library.custom_op(f"tpwtest::{layer}_{name}", mutates_args=())
    def inside(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
        return f(a, b)
    assert torch.equal(inside(x1, x2), want)
    assert torch.equal(inside(x1.clone().requires_grad_(), x2).detach(), want)


def test_compositions_below_autograd(tpw):
    """What is built on those: cdist, pdist, the neighbour masks and the k nearest rows."""
    x1, x2 = _inputs()
    T = torch.ops.torchpairwise
    calls = [lambda: tpw.cdist(x1, x2, "minkowski", p=3.0), lambda: T.cdist(x1, x2, "cosine"), lambda: tpw.pdist(x1, "cosine"),
             lambda: T.pdist(x1, "correlation"), lambda: tpw.k_neighbors_mask(x1, x2, 3, "cosine"), lambda: T.k_neighbors_mask(x1, x2, 3, "cosine"),
             lambda: tpw.pairwise_argkmin(x1, x2, 3, "euclidean")[1], lambda: T.radius_neighbors_mask(x1, x2, 4.0, "euclidean")]
    for call in calls:
        with torch.no_grad():
            want = call()
        with torch.inference_mode():
            assert torch.equal(call(), want)
