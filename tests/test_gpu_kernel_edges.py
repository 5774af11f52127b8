"""Edges of the kernels' tiles and of the rules that choose between them, each against the other route."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tpw():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    import torchpairwise_b200
    return torchpairwise_b200


@pytest.mark.parametrize("shape", [(1, 1030, 2051, 167), (1, 2048, 1025, 129), (2, 900, 1111, 255), (1, 1200, 1604, 1000), (1, 5000, 260, 257)])
def test_boolean_rows_of_any_length_equal_popcount(tpw, monkeypatch, shape):
    """Rows that fill no whole 16 bytes go to the tensor-core counts as padded copies, results of ragged rows leave word by
    word: every metric's float32 bits are those of the popcount kernels."""
    from torchpairwise_b200 import _abi
    b, n1, n2, d = shape
    g = torch.Generator().manual_seed(d)
    x1, x2 = (torch.rand(b, n1, d, generator=g) < 0.3).cuda(), (torch.rand(b, n2, d, generator=g) < 0.3).cuda()
    x1[0, 3], x2[0, 5] = False, False            # empty rows: 0 / 0 in the metrics that divide
    assert _abi.lib.tpw_bool_rows_pitch(b, n1, n2, d) == (d + 15) // 16 * 16
    for metric in ("hamming", "jaccard", "yule", "russellrao"):
        fn = getattr(tpw, metric + "_distances")
        got = fn(x1, x2)
        monkeypatch.setenv("TPW_DISABLE_BOOL_TC", "1")
        want = fn(x1, x2)
        monkeypatch.delenv("TPW_DISABLE_BOOL_TC")
        assert torch.equal(got.view(torch.int32), want.view(torch.int32)), (metric, shape)
    # any non-zero byte counts as true in a padded copy, as it does when the rows are packed to bits
    y = (torch.randint(0, 3, (n1, d), generator=g, dtype=torch.uint8)).cuda()
    torch.testing.assert_close(tpw.hamming_distances(y.view(torch.bool), x2[0]), tpw.hamming_distances(y != 0, x2[0]), rtol=0, atol=0)


@pytest.mark.parametrize("m1,m2,d", [(700, 1031, 3), (513, 2, 3), (1, 4097, 2), (1025, 1, 5), (600, 777, 8), (257, 1500, 16)])
def test_hausdorff_point_pairs_and_split_walks(tpw, monkeypatch, m1, m2, d):
    """Odd clouds (a lone last point), clouds shared by several CTAs, one to sixteen coordinates, NaN and infinite
    coordinates: values and indices of the exact loop."""
    g = torch.Generator().manual_seed(m1 + m2 + d)
    x1, x2 = torch.randn(2, 1, m1, d, generator=g), torch.randn(2, 1, m2, d, generator=g)
    x1[1, 0, m1 // 2, 0] = math.inf
    x2[1, 0, m2 // 2, d - 1] = math.nan
    got = tpw.directed_hausdorff_distances(x1.cuda(), x2.cuda())
    monkeypatch.setenv("TPW_HAUSDORFF_EXACT_LOOP", "1")
    want = tpw.directed_hausdorff_distances(x1.cuda(), x2.cuda())
    for a, w in zip(got, want):
        assert torch.equal(a, w)


@pytest.mark.parametrize("n2,d", [(1029, 320), (2047, 130), (258, 1030)])
@pytest.mark.parametrize("fn", ["sqeuclidean_distances", "cosine_distances"])
def test_tensor_core_matrix_with_ragged_rows(tpw, n2, d, fn):
    """Rows of the result that start on no 16-byte boundary leave the staged block word by word; an element does not depend on
    the other columns, so the bits are those of the same columns of a wider matrix."""
    g = torch.Generator().manual_seed(n2)
    x1, x2 = torch.randn(1100, d, generator=g).cuda(), torch.randn((n2 + 3) // 4 * 4, d, generator=g).cuda()
    wide = getattr(tpw, fn)(x1, x2)
    assert torch.equal(getattr(tpw, fn)(x1, x2[:n2]), wide[:, :n2])


@pytest.mark.parametrize("shape,p", [((8, 700, 301, 192), 3.0), ((3, 1000, 1035, 128), 1.0), ((20, 500, 45, 256), 2.5)])
def test_one_pass_backward_with_ragged_columns(tpw, shape, p):
    """x2 row counts that are no multiple of 4 take the one-pass backward as well; against the two-launch form, whose terms are
    the same in another order of addition (sums of up to 1035 float32 terms), and bit-reproducible."""
    from torchpairwise_b200 import _abi
    b, n1, n2, d = shape
    g = torch.Generator().manual_seed(n2)
    x1, x2 = torch.randn(b, n1, d, generator=g).cuda(), torch.randn(b, n2, d, generator=g).cuda()
    gr = torch.randn(b, n1, n2, generator=g).cuda()
    out = tpw.minkowski_distances(x1, x2, p)
    lib, stream = _abi.lib, torch.cuda.current_stream().cuda_stream
    want = lib.tpw_lp_backward_scratch_bytes(_abi.F32, _abi.LP_BWD_CDIST, b, n1, n2, d, p)
    assert want > 0
    res = []
    for scratch in (torch.empty(want, dtype=torch.uint8, device="cuda"), torch.empty(want, dtype=torch.uint8, device="cuda"), None):
        g1, g2 = torch.full_like(x1, math.nan), torch.full_like(x2, math.nan)
        _abi.check(lib.tpw_lp_backward_ws(_abi.F32, _abi.LP_BWD_CDIST, gr.data_ptr(), out.data_ptr(), x1.data_ptr(), x2.data_ptr(), None,
                                          g1.data_ptr(), g2.data_ptr(), b, n1, n2, d, p, None if scratch is None else scratch.data_ptr(),
                                          0 if scratch is None else want, stream))
        assert _abi.device_status(stream) == 0
        res.append((g1, g2))
    for one, again, two in zip(*res):
        assert torch.equal(one, again)
        assert float((one - two).abs().max()) <= 2e-5 * float(two.abs().max())   # sqrt(1035) * 2^-24 per sum, ten times over


@pytest.mark.parametrize("case", ["plain", "equal", "offset", "outlier", "infinite", "few coordinates"])
def test_hausdorff_expanded_form_and_hand_over(tpw, monkeypatch, case):
    """Large set pairs run the expanded form, and go over to the direct one where its error leaves too many rows undecided:
    values and indices of the exact loop either way, with and without a shuffled visiting order."""
    d = 2 if case == "few coordinates" else 3
    g = torch.Generator().manual_seed(len(case))
    x1 = torch.rand(2, 1, 8207, d, generator=g) * 2 - 1
    x2 = x1[:, :, torch.randperm(8207, generator=g)] + 0.05 * torch.randn(2, 1, 8207, d, generator=g)
    if case == "equal":
        x2 = x1.clone()
    elif case == "offset":
        x1, x2 = x1 + 3e3, x2 + 3e3
    elif case == "outlier":
        x2[1, 0, 17] = 1e19
    elif case == "infinite":
        x1[0, 0, 4000, 1], x2[1, 0, 0, 0] = math.inf, math.nan
    for shuffle in (False, True):
        res = []
        for exact in (False, True):
            if exact:
                monkeypatch.setenv("TPW_HAUSDORFF_EXACT_LOOP", "1")
            gen = torch.Generator(device="cuda").manual_seed(5) if shuffle else None
            res.append(tpw.directed_hausdorff_distances(x1.cuda(), x2.cuda(), shuffle=shuffle, generator=gen))
            monkeypatch.delenv("TPW_HAUSDORFF_EXACT_LOOP", raising=False)
        for a, w in zip(*res):
            assert torch.equal(a, w), (case, shuffle)


@pytest.mark.parametrize("d", [1023, 5003, 65535, 262139, 262143, 262145])
def test_quotients_of_large_counts_round_as_the_division(tpw, d):
    """The same up to and across 2^18, where the kernel goes over to the division: prefixes of lengths near d, near the powers of two
    below it and spread over the range, against each other."""
    from torchpairwise_b200 import _abi
    near = [d - t for t in range(60)] + [2 ** e + t for e in range(6, d.bit_length()) for t in (-1, 0, 1) if 2 ** e + t <= d]
    g = torch.Generator().manual_seed(d)
    i = torch.tensor(sorted(set(near)) + torch.randint(1, d + 1, (300,), generator=g).tolist())[:256]
    j = torch.cat([i, torch.randint(1, d + 1, (256,), generator=g)])[:300]
    k = torch.arange(d, device="cuda")
    x1, x2 = k[None] < i.cuda()[:, None], k[None] < j.cuda()[:, None]
    if d < 5000:                                  # enough pairs for the tensor-core counts
        x1, x2 = x1.repeat(9, 1), x2.repeat(9, 1)
    assert _abi.lib.tpw_bool_rows_pitch(1, x1.size(0), x2.size(0), d) > 0
    a, b = x1.sum(1).double(), x2.sum(1).double()
    diff, most = (a[:, None] - b[None]).abs(), torch.maximum(a[:, None], b[None])
    # a float64 quotient of integers this small, rounded once more to float32, is the correctly rounded quotient
    assert torch.equal(tpw.jaccard_distances(x1, x2), (diff / most).float())
    assert torch.equal(tpw.hamming_distances(x1, x2), (diff / d).float())


def test_quotients_of_counts_round_as_the_division(tpw):
    """Every quotient of counts with a denominator of up to 300 for four feature counts, through the metrics themselves: row i of
    x1 has its first i features set, row j of x2 its first j, so jaccard is |i - j| / max(i, j) and hamming |i - j| / D."""
    for d in (129, 160, 257, 300):
        n = d + 1
        x = (torch.arange(d)[None, :] < torch.arange(n)[:, None]).cuda()
        x2 = x.repeat(40, 1)                      # enough pairs for the tensor-core counts
        from torchpairwise_b200 import _abi
        if _abi.lib.tpw_bool_rows_pitch(1, n, 40 * n, d) == 0:
            x, x2 = x.repeat(2, 1), x.repeat(200, 1)
        assert _abi.lib.tpw_bool_rows_pitch(1, x.size(0), x2.size(0), d) > 0
        i, j = x.sum(1).float(), x2.sum(1).float()
        diff, most = (i[:, None] - j[None, :]).abs(), torch.maximum(i[:, None], j[None, :])
        # float64 division of integers this small, rounded once more to float32, is the correctly rounded quotient
        assert torch.equal(tpw.jaccard_distances(x, x2), torch.where(most > 0, diff.double() / most.double(), 0.0).float())
        assert torch.equal(tpw.hamming_distances(x, x2), (diff.double() / d).float())


@pytest.mark.parametrize("layer", ["python", "dispatcher"])
@pytest.mark.parametrize("p", [1.0, 3.0, math.inf])
def test_rows_padded_to_whole_vectors(tpw, monkeypatch, p, layer):
    """Large problems whose feature count is no multiple of 4 run on zero-padded copies; the same batches one at a time are too
    small for that.  The forward and the Chebyshev gradients add the same terms in the same order (bit-equal), the others in
    another order (sums of up to 600 float32 terms)."""
    from torchpairwise_b200 import ops
    tpw.load_torch_ops()
    monkeypatch.setattr(ops, "_native_ops", None if layer == "python" else torch.ops.torchpairwise)
    g = torch.Generator().manual_seed(7)
    n = 7   # 4e8 terms: forward, one-pass backward and Chebyshev backward are all padded
    x1, x2 = torch.randn(n, 600, 201, generator=g).cuda(), torch.randn(n, 500, 201, generator=g).cuda()
    gr = torch.randn(n, 600, 500, generator=g).cuda()

    def grads(a, c, up):
        a, c = a.clone().requires_grad_(), c.clone().requires_grad_()
        out = tpw.chebyshev_distances(a, c) if math.isinf(p) else tpw.minkowski_distances(a, c, p)
        return (out.detach(), *torch.autograd.grad(out, (a, c), up))

    whole = grads(x1, x2, gr)
    parts = [torch.stack(t) for t in zip(*(grads(x1[b], x2[b], gr[b]) for b in range(n)))]
    assert whole[1].shape == x1.shape and whole[2].shape == x2.shape and whole[1].is_contiguous()
    assert torch.equal(whole[0], parts[0])
    for w, q in zip(whole[1:], parts[1:]):
        if math.isinf(p):
            assert torch.equal(w, q)
        else:
            assert float((w - q).abs().max()) <= 2e-5 * float(q.abs().max())


@pytest.mark.parametrize("shape", [(1, 300, 1100, 192), (2, 1030, 1500, 256), (1, 20000, 1025, 72), (3, 1024, 2048, 260)])
def test_gradient_products_with_dealt_out_chunks(tpw, shape):
    """Products whose tiles do not fill the last wave share them chunk by chunk between CTAs: against float64, and bit-reproducible.
    The products keep 22 bits of each factor and add up to 20000 terms in float32: 1e-5 of the largest element, as for whole tiles."""
    b, n1, n2, d = shape
    g = torch.Generator().manual_seed(n1)
    x1, x2 = torch.randn(b, n1, d, generator=g).cuda().requires_grad_(), torch.randn(b, n2, d, generator=g).cuda().requires_grad_()
    up = torch.randn(b, n1, n2, generator=g).cuda()
    one = torch.autograd.grad(tpw.sqeuclidean_distances(x1, x2), (x1, x2), up)
    two = torch.autograd.grad(tpw.sqeuclidean_distances(x1, x2), (x1, x2), up)
    assert all(torch.equal(a, c) for a, c in zip(one, two))
    u, a, c = up.double(), x1.detach().double(), x2.detach().double()
    want = (2 * (u.sum(2, keepdim=True) * a - u @ c), 2 * (u.sum(1)[..., None] * c - u.transpose(1, 2) @ a))
    for got, ref in zip(one, want):
        assert float((got - ref).abs().max()) <= 1e-5 * float(ref.abs().max())


def test_chebyshev_backward_from_several_threads(tpw):
    """Threads that run the Chebyshev backward with different feature counts, each on its own stream: every launch is accepted and
    every gradient is that of a call alone.  (The kernels' shared-memory size depends on the feature count.)"""
    import threading
    from torchpairwise_b200 import _abi
    lib, n = _abi.lib, 64

    def problem(d):
        g = torch.Generator().manual_seed(d)
        x1, x2, up = torch.randn(1, n, d, generator=g).cuda(), torch.randn(1, n, d, generator=g).cuda(), torch.randn(1, n, n, generator=g).cuda()
        out = tpw.chebyshev_distances(x1, x2)
        scratch = torch.empty(lib.tpw_chebyshev_backward_scratch_bytes(_abi.F32, 1, n, n, d), dtype=torch.uint8, device="cuda")
        return x1, x2, up, out, scratch, torch.empty_like(x1), torch.empty_like(x2)

    def call(pr, d, stream):
        x1, x2, up, out, scratch, g1, g2 = pr
        return lib.tpw_chebyshev_backward_ws(up.data_ptr(), out.data_ptr(), x1.data_ptr(), x2.data_ptr(), g1.data_ptr(), g2.data_ptr(),
                                             scratch.data_ptr(), scratch.numel(), 1, n, n, d, stream)

    dims = [16, 256, 64, 252]
    problems = [problem(d) for d in dims]
    torch.cuda.synchronize()
    want = []
    for pr, d in zip(problems, dims):
        assert call(pr, d, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        want.append((pr[5].clone(), pr[6].clone()))
    status = [0] * len(dims)
    streams = [torch.cuda.Stream() for _ in dims]

    def work(t):
        torch.cuda.set_device(0)
        for _ in range(1000):
            status[t] |= call(problems[t], dims[t], streams[t].cuda_stream)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(len(dims))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert status == [0] * len(dims)
    for pr, (w1, w2) in zip(problems, want):
        assert torch.equal(pr[5], w1) and torch.equal(pr[6], w2)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", [(1, 15, 33, 9), (2, 17, 31, 33), (1, 300, 65, 32), (1, 64, 300, 40), (1, 1400, 40, 64), (1, 1420, 33, 64), (1, 45, 2100, 64),
                                   (3, 700, 31, 64)])
def test_small_backward_kernels_equal_the_tile_kernel(tpw, monkeypatch, dtype, shape):
    """Few gradient blocks run with one or two elements to a thread, by a rule on type, metric, side and number of elements; either
    way every metric's gradients are the tile kernel's bit for bit."""
    from torchpairwise_b200 import _abi
    lib, (b, n1, n2, d) = _abi.lib, shape
    g = torch.Generator().manual_seed(n1 + n2)
    x1, x2 = torch.randn(b, n1, d, generator=g).to(dtype).cuda(), torch.randn(b, n2, d, generator=g).to(dtype).cuda()
    up, aux, w = torch.randn(b, n1, n2, generator=g).to(dtype).cuda(), (torch.rand(b, n1, n2, generator=g) + 0.5).to(dtype).cuda(), torch.rand(b, d, generator=g).to(dtype).cuda()
    largest = (x1[:, :, None] - x2[:, None]).abs().amax(3)
    code = _abi.F32 if dtype == torch.float32 else _abi.F64
    modes = [(_abi.LP_BWD_CDIST, p) for p in (1.0, 2.0, 3.0, 2.5, math.inf)] + [(m, p) for m in (_abi.LP_BWD_PPMINKOWSKI, _abi.LP_BWD_WMINKOWSKI) for p in (1.0, 2.0, 3.0, 1.5)]
    for mode, p in modes + [(_abi.LP_BWD_MATMUL, 2.0)]:
        res = []
        for tile in (False, True):
            if tile:
                monkeypatch.setenv("TPW_DISABLE_SMALL_BWD", "1")
            g1, g2 = torch.full_like(x1, math.nan), torch.full_like(x2, math.nan)
            _abi.check(lib.tpw_lp_backward(code, mode, up.data_ptr(), (largest if math.isinf(p) else aux).data_ptr(), x1.data_ptr(), x2.data_ptr(),
                                           w.data_ptr() if mode == _abi.LP_BWD_WMINKOWSKI else None, g1.data_ptr(), g2.data_ptr(), b, n1, n2, d, p,
                                           torch.cuda.current_stream().cuda_stream))
            monkeypatch.delenv("TPW_DISABLE_SMALL_BWD", raising=False)
            res.append((g1, g2))
        assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1]), (mode, p)
        assert not torch.isnan(res[0][0]).any() and not torch.isnan(res[0][1]).any()


@pytest.mark.parametrize("n1,n2,d", [(1024, 2048, 128), (1280, 1408, 96), (1500, 1301, 64), (1500, 1301, 100)])
@pytest.mark.parametrize("p", [1.0, 3.0, math.inf])
def test_forward_tiles_of_either_size_agree(tpw, n1, n2, d, p):
    """The forward's tile size follows the number of tiles; an element does not depend on the other rows, so its bits are those of a
    call on fewer rows (smaller tiles) and of one on more (larger tiles)."""
    g = torch.Generator().manual_seed(d)
    x1, x2 = torch.randn(4 * n1, d, generator=g).cuda(), torch.randn(n2, d, generator=g).cuda()
    out = tpw.minkowski_distances(x1[:n1].clone(), x2, p)
    assert torch.equal(out, tpw.minkowski_distances(x1, x2, p)[:n1])
    assert torch.equal(out[:100, :70], tpw.minkowski_distances(x1[:100].clone(), x2[:70].clone(), p))


@pytest.mark.parametrize("n2", [129, 255, 257, 1000, 1025, 2049, 5000])
@pytest.mark.parametrize("order", ["random", "clusters", "falling", "equal rows", "not finite"])
def test_k_nearest_whatever_the_order_of_the_rows(tpw, n2, order):
    """The top-k bound comes from a sample of the x2 rows and from tiles that found k keys; whatever the order of x2, the values are those
    of a selection on the matrix the same engine writes, and the columns are distinct and hold them."""
    g = torch.Generator().manual_seed(n2)
    x1, x2 = torch.randn(700, 64, generator=g), torch.randn(n2, 64, generator=g)
    if order == "clusters":
        c = 5 * torch.randn(20, 64, generator=g)
        x1, x2 = 0.3 * x1 + c[torch.arange(700) % 20], 0.3 * x2 + c[torch.arange(n2) * 20 // n2]
    elif order == "falling":
        x2 = x2 * torch.linspace(3, 0.5, n2)[:, None]
    elif order == "equal rows":
        x2 = x2[:3].repeat(n2 // 3 + 1, 1)[:n2]
    elif order == "not finite":
        x1[5, 3], x1[6, 0], x2[n2 // 2, 1], x2[7, 2] = math.inf, math.nan, math.inf, math.nan
    x1, x2 = x1.cuda(), x2.cuda()
    was = tpw.get_dot_engine()
    tpw.set_dot_engine("tcgen05")
    try:
        for metric, fn in (("sqeuclidean", tpw.sqeuclidean_distances), ("cosine", tpw.cosine_distances)):
            full = fn(x1, x2)
            for k in (1, 2, 3, 8, 16):
                inds, vals = tpw.pairwise_argkmin(x1, x2, k, metric)
                # the kernels keep no NaN: a distance is clamped from below by 0, which a NaN becomes
                assert torch.equal(full.topk(k, dim=-1, largest=False, sorted=True).values, vals), (metric, k)
                assert torch.equal(full.gather(-1, inds), vals), (metric, k)
                assert all(len(set(r)) == k for r in inds.tolist())
                if order == "equal rows":                 # ties go to the smaller rows
                    assert bool((inds[:, 1:][vals[:, 1:] == vals[:, :-1]] > inds[:, :-1][vals[:, 1:] == vals[:, :-1]]).all())
    finally:
        tpw.set_dot_engine(was)


@pytest.mark.parametrize("d", [2, 3, 7, 12])
@pytest.mark.parametrize("case", ["sigma 0.01", "sigma 0.003", "sigma 0.001", "sigma 0.0003", "shells", "half equal", "one far point", "repeated points"])
def test_hausdorff_rows_handed_over(tpw, monkeypatch, case, d):
    """Set pairs whose largest row minima lie within the expanded form's error of one another hand those rows, from a few to all of them,
    over to the direct form; values and indices are the exact loop's, with and without a shuffled visiting order."""
    g, m = torch.Generator().manual_seed(d), 6701
    x1 = torch.rand(3, 1, m, d, generator=g) * 2 - 1
    noise = torch.randn(3, 1, m, d, generator=g)
    if case.startswith("sigma"):
        x2 = x1 + float(case.split()[1]) * noise
    elif case == "shells":                       # voxel shells of equal radius one voxel apart
        x1 = (40 * torch.nn.functional.normalize(x1, dim=-1)).round()
        x2 = (41 * torch.nn.functional.normalize(x1 + 0.02 * noise, dim=-1)).round()
    elif case == "half equal":
        x2 = torch.where(torch.arange(m)[None, None, :, None] % 2 == 0, x1, x1 + 1e-3 * noise)
    elif case == "one far point":
        x2 = x1 + 0.05 * noise
        x1[:, :, 4001] = 30.0
    else:
        x1 = x1[:, :, :50].repeat(1, 1, m // 50 + 1, 1)[:, :, :m].contiguous()
        x2 = x1.roll(7, 2) + 2e-3 * noise.roll(1, 2)
    for shuffle in (False, True):
        res = []
        for exact in (False, True):
            if exact:
                monkeypatch.setenv("TPW_HAUSDORFF_EXACT_LOOP", "1")
            gen = torch.Generator(device="cuda").manual_seed(5) if shuffle else None
            res.append(tpw.directed_hausdorff_distances(x1.cuda(), x2.cuda(), shuffle=shuffle, generator=gen))
            monkeypatch.delenv("TPW_HAUSDORFF_EXACT_LOOP", raising=False)
        for a, w in zip(*res):
            assert torch.equal(a, w), (case, shuffle)


@pytest.mark.parametrize("shape", [(1, 70, 50, 16), (2, 129, 67, 36), (1, 64, 64, 70), (1, 300, 130, 257)])
def test_chebyshev_backward_with_values_that_are_not_finite(tpw, shape):
    """Infinite and NaN coordinates in the group match: an infinite difference attains an infinite maximum, a NaN attains none and hides
    nothing; against the dense kernel, which tests every coordinate."""
    from torchpairwise_b200 import _abi
    b, n1, n2, d = shape
    g = torch.Generator().manual_seed(d)
    x1, x2 = torch.randn(b, n1, d, generator=g), torch.randn(b, n2, d, generator=g)
    x1[0, 3, 1], x1[0, 5, d - 1], x2[0, 7, 0], x2[0, 9, 2], x1[0, 11, 3], x2[0, 11, 3] = math.inf, math.nan, -math.inf, math.nan, math.inf, math.inf
    up = torch.randn(b, n1, n2, generator=g).cuda()
    a, c = x1.cuda().requires_grad_(), x2.cuda().requires_grad_()
    out = tpw.chebyshev_distances(a, c)
    g1, g2 = torch.autograd.grad(out, (a, c), up)
    d1, d2 = torch.empty_like(g1), torch.empty_like(g2)
    _abi.check(_abi.lib.tpw_lp_backward(_abi.F32, _abi.LP_BWD_CDIST, up.data_ptr(), out.data_ptr(), a.data_ptr(), c.data_ptr(), None, d1.data_ptr(),
                                        d2.data_ptr(), b, n1, n2, d, math.inf, torch.cuda.current_stream().cuda_stream))
    for got, want in ((g1, d1), (g2, d2)):
        torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-5 * float(want.nan_to_num().abs().max()), equal_nan=True)


@pytest.mark.parametrize("low", ["x1", "x2", "both", "neither"])
def test_low_parts_that_are_left_out_next_to_values_that_are_not_finite(tpw, low):
    """An operand that 16 bits hold exactly has no low part to multiply; an infinity or NaN in either operand still reaches every result it
    reaches in float64, and no other, forward and backward."""
    g = torch.Generator().manual_seed(3)
    x1, x2 = torch.randn(1100, 192, generator=g), torch.randn(1300, 192, generator=g)
    if low in ("x1", "both"):
        x1 = x1.bfloat16().float()
    if low in ("x2", "both"):
        x2 = x2.bfloat16().float()
    x1[17, 5], x2[33, 7], x2[40, 0] = math.inf, -math.inf, math.nan
    up = torch.randn(1100, 1300, generator=g).cuda()
    a, c = x1.cuda().requires_grad_(), x2.cuda().requires_grad_()
    out = tpw.linear_kernel(a, c)
    g1, g2 = torch.autograd.grad(out, (a, c), up)
    w, w1, w2 = x1.cuda().double() @ x2.cuda().double().T, up.double() @ x2.cuda().double(), up.double().T @ x1.cuda().double()
    for got, want in ((out.detach(), w), (g1, w1), (g2, w2)):
        # a split infinity has a NaN low part, so an infinite result may come out as NaN; finite ones are finite and right
        ok = torch.isfinite(want)
        assert torch.equal(torch.isfinite(got), ok)
        assert float((got[ok] - want[ok]).abs().max()) <= 1e-5 * float(want[ok].abs().max())
