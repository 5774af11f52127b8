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


SAVES_RESULT = ["euclidean_distances", "chebyshev_distances", "minkowski_distances", "cosine_distances", "cosine_similarity", "jensenshannon_distances"]


@pytest.mark.parametrize("layer", ["python", "dispatcher"])
@pytest.mark.parametrize("lead", [(), (2,)])
@pytest.mark.parametrize("name", SAVES_RESULT + ["manhattan_distances", "sqeuclidean_distances", "linear_kernel", "canberra_distances", "wminkowski_distances",
                                                 "haversine_distances", "directed_hausdorff_distances"])
def test_changes_in_place_before_backward_are_noticed(tpw, layer, lead, name):
    """A saved operand or result that the caller changes between forward and backward is an error, not a wrong gradient; changing
    something that was not saved stays allowed."""
    fn = getattr(tpw if layer == "python" else torch.ops.torchpairwise, name)

    def forward():
        x1, x2 = (t.abs().requires_grad_() for t in _inputs(lead))
        if name == "wminkowski_distances":
            w = torch.ones(*lead, 12, device="cuda", requires_grad=True)
            return (x1, x2, w), fn(x1, x2, 3.0, w)
        if name == "haversine_distances":
            x1, x2 = (t.detach()[..., :2].contiguous().requires_grad_() for t in (x1, x2))
        if name == "directed_hausdorff_distances":
            x1, x2 = (t.detach().unsqueeze(len(lead)).requires_grad_() for t in (x1, x2))
        return (x1, x2), fn(x1, x2, 3.0) if name == "minkowski_distances" else fn(x1, x2)

    def total(out):
        return (out[0] if isinstance(out, tuple) else out).sum()

    inputs, out = forward()
    total(out).backward()                                # unchanged: works
    for i in range(len(inputs)):
        inputs, out = forward()
        with torch.no_grad():
            inputs[i].mul_(1.5)
        with pytest.raises(RuntimeError, match="inplace"):
            total(out).backward()
    if name in SAVES_RESULT or name == "directed_hausdorff_distances":
        inputs, out = forward()
        with pytest.raises(RuntimeError, match="inplace"):
            out = out[0] if isinstance(out, tuple) else out
            loss = out.sum()
            with torch.no_grad():
                out.mul_(1.5)
            loss.backward()


@pytest.mark.parametrize("layer", ["python", "dispatcher"])
def test_converted_operands_may_change(tpw, layer):
    """Operands that were converted or made contiguous are saved as copies: changing the originals afterwards changes no gradient."""
    fn = getattr(tpw if layer == "python" else torch.ops.torchpairwise, "minkowski_distances")
    x1, x2 = _inputs()
    for make in (lambda t: t.bfloat16(), lambda t: t.t().contiguous().t()):
        grads = []
        for change in (False, True):
            a, b = make(x1).requires_grad_(), make(x2).requires_grad_()
            out = fn(a, b, 3.0)
            if change:
                with torch.no_grad():
                    a.mul_(2), b.mul_(2)
            out.sum().backward()
            grads.append((a.grad, b.grad))
        assert all(torch.equal(u, v) for u, v in zip(*grads))


@pytest.mark.parametrize("name", ["euclidean_distances", "minkowski_distances", "cosine_distances", "cosine_similarity"])
def test_refusals_and_result_types_do_not_depend_on_the_library_being_loaded(tpw, monkeypatch, name):
    """Transforms without a rule, subclasses and arguments out of range: with the dispatcher's library loaded, what happens without."""
    from torchpairwise_b200 import ops
    fn = getattr(tpw, name)
    x1, x2 = _inputs()

    class Sub(torch.Tensor):
        pass

    def dual():
        with torch.autograd.forward_ad.dual_level():
            return fn(torch.autograd.forward_ad.make_dual(x1, x1.clone()), x2)

    calls = [lambda: torch.func.vmap(fn)(torch.stack([x1, x1]), torch.stack([x2, x2])), lambda: torch.func.grad(lambda a: fn(a, x2).sum())(x1),
             lambda: torch.func.jvp(lambda a: fn(a, x2), (x1,), (x1,)), dual, lambda: fn(x1.as_subclass(Sub), x2), lambda: fn(x1, x2.as_subclass(Sub))]
    if name == "minkowski_distances":
        calls += [lambda p=p: fn(x1, x2, p) for p in (float("nan"), -1.0, float("-inf"))]
    seen = []
    for native in (True, False):
        if not native:
            monkeypatch.setattr(ops, "_native_ops", None)
        seen.append([])
        for call in calls:
            try:
                seen[-1].append(type(call()))
            except Exception as e:
                seen[-1].append(type(e))
    assert seen[0] == seen[1]
    assert all(issubclass(t, Exception) for t in seen[0][:4] + seen[0][6:]) and seen[0][4:6] == [torch.Tensor] * 2


@pytest.mark.parametrize("n", [96, 520])
def test_boolean_rows_of_a_matrix_against_its_columns(tpw, n):
    """x and x.t() share pointer and shape, and are not the same rows (96: packed words, 520: tensor-core counts)."""
    x = (torch.rand(n, n, generator=torch.Generator().manual_seed(n)) < 0.3).cuda()
    for fn in (tpw.jaccard_distances, tpw.hamming_distances, torch.ops.torchpairwise.jaccard_distances):
        assert torch.equal(fn(x, x.t()), fn(x, x.t().contiguous()))
        assert torch.equal(fn(x, x[:]), fn(x, x.clone()))
