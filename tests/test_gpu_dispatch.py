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


@pytest.mark.parametrize("name,kw", [("euclidean_distances", {}), ("manhattan_distances", {}), ("chebyshev_distances", {}), ("minkowski_distances", {"p": 3.0}),
                                     ("minkowski_distances", {"p": 2.5}), ("minkowski_distances", {"p": 0.0}), ("cosine_distances", {}), ("cosine_similarity", {})])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16])
@pytest.mark.parametrize("shape", [((40, 12), (33, 12)), ((2, 300, 70), (2, 257, 70)), ((2, 2048, 64), (2, 1100, 64))])
def test_python_functions_and_cpp_nodes_agree(tpw, monkeypatch, name, kw, dtype, shape):
    """The Python autograd functions, forced, against the C++ nodes that stand in for them: results and gradients, both or one of them,
    bit for bit (the launches are the same)."""
    from torchpairwise_b200 import ops
    g = torch.Generator().manual_seed(len(name))
    x1, x2 = (torch.randn(*s, generator=g).to(dtype).cuda() for s in shape)
    up = torch.randn(*shape[0][:-1], shape[1][-2], generator=g).to(dtype).cuda()
    seen = []
    for python in (True, False):
        monkeypatch.setattr(ops, "_native_ops", None if python else torch.ops.torchpairwise)
        a, b = x1.clone().requires_grad_(), x2.clone().requires_grad_()
        out = getattr(tpw, name)(a, b, **kw)
        if dtype != torch.bfloat16 and len(shape[0]) == 3:      # neither a view nor a conversion on top of the node
            assert (type(out.grad_fn).__name__ in ("_CdistFunctionBackward", "_CosineSimilarityFunctionBackward")) == python
        res = [out.detach(), *torch.autograd.grad(out, (a, b), up)]
        for need in ((True, False), (False, True)):
            a, b = x1.clone().requires_grad_(need[0]), x2.clone().requires_grad_(need[1])
            res += torch.autograd.grad(getattr(tpw, name)(a, b, **kw), (a,) if need[0] else (b,), up)
        with torch.no_grad():
            res.append(getattr(tpw, name)(x1, x2, **kw))
        seen.append(res)
    assert all(torch.equal(p, c) and p.dtype == c.dtype == dtype for p, c in zip(*seen))


@pytest.mark.parametrize("name", ["euclidean_distances", "manhattan_distances", "chebyshev_distances", "minkowski_distances", "cosine_distances",
                                  "seuclidean_distances"])
def test_one_requested_gradient(tpw, name):
    """One gradient out of two that could be asked for: that of the call for both, to rounding (it may be added in another order)."""
    for n1, n2, d in ((40, 33, 12), (700, 600, 192)):
        g = torch.Generator().manual_seed(n1)
        x1, x2 = torch.randn(n1, d, generator=g).cuda().requires_grad_(), torch.randn(n2, d, generator=g).cuda().requires_grad_()
        kw = {"seuclidean_distances": {"V": torch.rand(d, generator=g).cuda() + 0.5}, "minkowski_distances": {"p": 3.0}}.get(name, {})
        out = getattr(tpw, name)(x1, x2, **kw)
        up = torch.randn(n1, n2, generator=g).cuda()
        both = torch.autograd.grad(out, (x1, x2), up, retain_graph=True)
        for t, want in zip((x1, x2), both):
            got, = torch.autograd.grad(out, (t,), up, retain_graph=True)
            assert float((got - want).abs().max()) <= 2e-5 * float(want.abs().max())
