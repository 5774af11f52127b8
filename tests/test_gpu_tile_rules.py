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


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("b,n1,n2", [(1, 1, 5), (2, 7, 300), (1, 8, 257), (2, 9, 31), (1, 17, 64), (1, 500, 3)])
def test_cosine_backward_column_sums(tpw, dtype, b, n1, n2):
    """colterm[j] = sum_i d(denominator) n1[i], n1 terms of up to five roundings added one after the other; pairs with a zero norm add nothing."""
    from torchpairwise_b200 import _abi
    g = torch.Generator().manual_seed(n1 + n2)
    up, out = torch.randn(b, n1, n2, generator=g).to(dtype).cuda(), (torch.rand(b, n1, n2, generator=g) * 2).to(dtype).cuda()
    a, c = (torch.rand(b, n, generator=g).to(dtype).cuda() + 0.5 for n in (n1, n2))
    a[:, n1 // 2] = 0
    dm, row, col = torch.empty_like(up), torch.empty_like(a), torch.empty_like(c)
    _abi.check(_abi.lib.tpw_cosine_backward_prepare(_abi.F32 if dtype == torch.float32 else _abi.F64, _abi.DOT_COSINE_DIST, up.data_ptr(), out.data_ptr(),
                                                    a.data_ptr(), c.data_ptr(), dm.data_ptr(), row.data_ptr(), col.data_ptr(), b, n1, n2,
                                                    torch.cuda.current_stream().cuda_stream))
    den = a.double()[:, :, None] * c.double()[:, None]
    term = torch.where(den == 0, 0.0, up.double() / den * (1 - out.double())) * a.double()[:, :, None]
    bound = (n1 + 8) * torch.finfo(dtype).eps * torch.where(den == 0, 0.0, (up.double() / den).abs() * (1 + out.double())).mul(a.double()[:, :, None]).sum(1)
    assert bool(((col.double() - term.sum(1)).abs() <= bound).all())


# Gradient products whose tiles are no multiple of the 74 pairs: 1, 28 and 73 left over, in parts of one chunk, of several, and nearly whole.
@pytest.mark.parametrize("b,n1,n2,d", [(15, 1131, 1393, 192), (1, 7000, 1030, 100), (1, 200, 9000, 130), (7, 900, 1200, 250), (1, 18600, 1100, 64)])
def test_gradients_of_tiles_that_several_pairs_share(tpw, b, n1, n2, d):
    """From the distances as they were returned: the coefficients' and the operands' splits and float32 sums of n2 (n1) terms in chunks are
    within 2^-18 of the terms' magnitudes."""
    g = torch.Generator().manual_seed(n1)
    x1, x2 = torch.randn(b, n1, d, generator=g).cuda().requires_grad_(), torch.randn(b, n2, d, generator=g).cuda().requires_grad_()
    up = torch.randn(b, n1, n2, generator=g).cuda()
    out = tpw.euclidean_distances(x1, x2)
    g1, g2 = torch.autograd.grad(out, (x1, x2), up)
    c = up.double() / out.detach().double()
    for got, x, y, m in ((g1, x1.detach().double(), x2.detach().double(), c), (g2, x2.detach().double(), x1.detach().double(), c.transpose(1, 2))):
        want = m.sum(2, keepdim=True) * x - m @ y
        size = m.abs().sum(2, keepdim=True) * x.abs() + m.abs() @ y.abs()
        assert bool(((got - want).abs() <= 2 ** -18 * size).all())


@pytest.mark.parametrize("lead,n1", [((), 128), ((), 129), ((), 256), ((), 257), ((), 300), ((), 385), ((3,), 300), ((2,), 640)])
@pytest.mark.parametrize("n2", [300, 2049, 30011])
def test_nearest_row_where_the_last_tile_is_half_empty(tensor_cores, lead, n1, n2):
    """The smallest of the row of distances that the same engine stores, and a column that holds it."""
    g = torch.Generator().manual_seed(n1 + n2)
    x1, x2 = torch.randn(*lead, n1, 72, generator=g).cuda(), torch.randn(*lead, n2, 72, generator=g).cuda()
    x1[..., -1, :] = x2[..., n2 - 1, :]
    at, nearest = tensor_cores.pairwise_argmin_min(x1, x2, "sqeuclidean")
    sq = tensor_cores.sqeuclidean_distances(x1, x2)
    assert torch.equal(nearest, sq.amin(-1)) and torch.equal(sq.gather(-1, at.unsqueeze(-1)).squeeze(-1), nearest)


@pytest.mark.parametrize("lead,n1,n2,d", [((), 5003, 4111, 167), ((), 6001, 6003, 167), ((3,), 6001, 2003, 1024), ((), 2300, 9999, 1024), ((5,), 2100, 1031, 1100), ((), 385, 259, 4096)])
def test_ragged_boolean_counts_in_steady_state(tpw, lead, n1, n2, d):
    from torchpairwise_b200 import _abi
    assert _abi.lib.tpw_bool_rows_pitch(lead[0] if lead else 1, n1, n2, d) > 0          # the tensor cores' problem
    g = torch.Generator().manual_seed(d)
    x1, x2 = (torch.rand(*lead, n1, d, generator=g) < 0.2).cuda(), (torch.rand(*lead, n2, d, generator=g) < 0.2).cuda()
    both = x1.float() @ x2.float().transpose(-1, -2)          # below 2^24: exact
    a, b = x1.float().sum(-1)[..., :, None], x2.float().sum(-1)[..., None, :]
    union, differ = a + b - both, a + b - 2 * both
    zero = torch.zeros((), device="cuda")
    assert torch.equal(tpw.jaccard_distances(x1, x2), torch.where(union == 0, zero, differ / union))
    assert torch.equal(tpw.hamming_distances(x1, x2), differ / torch.tensor(float(d), device="cuda"))


@pytest.mark.parametrize("b,n1,n2", [(1, 3000, 4112), (3, 700, 1024), (1, 4400, 2308), (2, 300, 260), (1, 6000, 6004)])
@pytest.mark.parametrize("d", [256, 720, 1040, 2064])
def test_boolean_results_on_and_off_the_16_byte_grid_agree(tpw, b, n1, n2, d):
    """Whichever form of the kernel runs -- it depends on the metric, on the features, on the result's size and on whether its rows start on
    16-byte boundaries -- writes the same bits, the popcount kernel's, and nothing beside them."""
    from torchpairwise_b200 import _abi
    g = torch.Generator().manual_seed(n1)
    x1, x2 = (torch.rand(b, n1, d, generator=g) < 0.3).cuda(), (torch.rand(b, n2, d, generator=g) < 0.3).cuda()
    pop1, pop2 = x1.sum(-1, dtype=torch.int32), x2.sum(-1, dtype=torch.int32)
    if b * n1 * n2 * d < 1 << 28:
        pytest.skip("too small for the tensor cores")
    words = (d + 127) // 128 * 4
    w1, w2 = (torch.empty(b, n, words, dtype=torch.int32, device="cuda") for n in (n1, n2))
    for x, w, pop, n in ((x1, w1, pop1, n1), (x2, w2, pop2, n2)):
        _abi.check(_abi.lib.tpw_bitpack(x.data_ptr(), w.data_ptr(), pop.data_ptr(), b * n, d, words, torch.cuda.current_stream().cuda_stream))
    for metric in (_abi.BOOL_METRICS[name] for name in ("jaccard", "eq_mean", "and_sum", "yule", "dice")):
        res = [torch.empty(b * n1 * n2, device="cuda")]
        _abi.check(_abi.lib.tpw_bool_metric_forward(metric, w1.data_ptr(), w2.data_ptr(), pop1.data_ptr(), pop2.data_ptr(), res[0].data_ptr(), b, n1, n2, d, words,
                                                    torch.cuda.current_stream().cuda_stream))
        for off in (0, 1):
            buf = torch.full((b * n1 * n2 + 8,), -7.0, device="cuda")
            _abi.check(_abi.lib.tpw_bool_metric_forward_tc(metric, x1.data_ptr(), x2.data_ptr(), pop1.data_ptr(), pop2.data_ptr(),
                                                           buf.data_ptr() + 4 * off, b, n1, n2, d, torch.cuda.current_stream().cuda_stream))
            assert bool((buf[:off] == -7).all()) and bool((buf[off + b * n1 * n2:] == -7).all())
            res.append(buf[off:off + b * n1 * n2].clone())
        assert torch.equal(res[0].view(torch.int32), res[1].view(torch.int32)) and torch.equal(res[0].view(torch.int32), res[2].view(torch.int32)), metric


# More tiles than two for each of the 74 pairs of SMs, or each of the 148 SMs, so that accumulators, slots and staging areas are used
# again, with last column tiles of one 64-column pass among them: rows of the result off the 16-byte grid and on it, few and many
# features, results within L2 and larger, which take a CTA by itself or a pair to a tile.
STEADY = [((), 5003, 4111, 72), ((), 2300, 9999, 65), ((5,), 2100, 1031, 64), ((), 6200, 6001, 64), ((), 5003, 4111, 264), ((), 5003, 4112, 72),
          ((3,), 2100, 2052, 100), ((), 5003, 4112, 200), ((3,), 2100, 2052, 200)]
EDGES = [((), n1, n2, d) for n1, n2 in [(128, 256), (129, 257), (256, 259), (257, 511), (385, 300), (700, 1026), (700, 1028)] for d in (64, 136, 320)]


@pytest.mark.parametrize("lead,n1,n2,d", STEADY + EDGES)
def test_contractions_of_one_cta_and_of_pairs(tensor_cores, lead, n1, n2, d):
    """The three-product split of the distances drops at most 2^-15 |x| |y| of a dot product, float32 sums of d terms and the epilogue add
    (d + 8) 2^-24 of |x|^2 + |y|^2; the plain product's split drops 2^-20 |x| |y|."""
    g = torch.Generator().manual_seed(n1 + d)
    x1, x2 = torch.randn(*lead, n1, d, generator=g).cuda(), torch.randn(*lead, n2, d, generator=g).cuda()
    a, b = x1.double(), x2.double()
    na, nb = a.norm(dim=-1)[..., :, None], b.norm(dim=-1)[..., None, :]
    bound = 2 ** -14 * na * nb + (d + 8) * 2 ** -24 * (na ** 2 + nb ** 2)
    dot = a @ b.transpose(-1, -2)
    sq = na ** 2 + nb ** 2 - 2 * dot
    assert bool(((tensor_cores.sqeuclidean_distances(x1, x2) - sq).abs() <= bound).all())
    assert bool(((tensor_cores.euclidean_distances(x1, x2).double() ** 2 - sq).abs() <= 1.01 * bound + 2 ** -22 * sq).all())
    assert bool(((tensor_cores.cosine_distances(x1, x2) - (1 - dot / (na * nb))).abs() <= bound / (na * nb)).all())
    assert bool(((tensor_cores.linear_kernel(x1, x2) - dot).abs() <= ((d + 8) * 2 ** -24 + 2 ** -20) * na * nb).all())
    if not lead:
        own = tensor_cores.sqeuclidean_distances(x1, x1)
        assert bool((own.diagonal() == 0).all()) and bool(((own - (na ** 2 + na.T ** 2 - 2 * a @ a.T)).abs() <= 2 ** -14 * na * na.T + (d + 8) * 2 ** -24 * (na ** 2 + na.T ** 2)).all())


# At least 148 blocks of 32 rows by 32 features, one to each SM, but fewer than 49 gradient blocks of 64 x 64 (float64) or 128 x 128.
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", [(1, 1500, 1480, 128), (3, 480, 500, 100), (1, 3000, 70, 60), (2, 33, 750, 128)])
def test_walk_of_four_rows_to_a_thread_equals_the_tile_kernel(tpw, monkeypatch, dtype, shape):
    """Both gradients of a call, and either alone, are the tile kernel's bit for bit."""
    from torchpairwise_b200 import _abi
    lib, (b, n1, n2, d) = _abi.lib, shape
    g = torch.Generator().manual_seed(n1 + n2)
    x1, x2 = torch.randn(b, n1, d, generator=g).to(dtype).cuda(), torch.randn(b, n2, d, generator=g).to(dtype).cuda()
    up, aux = torch.randn(b, n1, n2, generator=g).to(dtype).cuda(), (torch.rand(b, n1, n2, generator=g) + 0.5).to(dtype).cuda()
    w = torch.rand(b, d, generator=g).to(dtype).cuda()
    aux[:, 3, 5] = 0
    code = _abi.F32 if dtype == torch.float32 else _abi.F64
    modes = [(_abi.LP_BWD_CDIST, p) for p in (1.0, 2.0, 3.0, 2.5)] + [(m, p) for m in (_abi.LP_BWD_PPMINKOWSKI, _abi.LP_BWD_WMINKOWSKI) for p in (1.0, 2.0, 3.0, 1.5)]
    for mode, p in modes + [(_abi.LP_BWD_MATMUL, 2.0)]:
        def gradients(first, second):
            g1, g2 = torch.full_like(x1, math.nan), torch.full_like(x2, math.nan)
            _abi.check(lib.tpw_lp_backward(code, mode, up.data_ptr(), aux.data_ptr(), x1.data_ptr(), x2.data_ptr(),
                                           w.data_ptr() if mode == _abi.LP_BWD_WMINKOWSKI else None, g1.data_ptr() if first else None,
                                           g2.data_ptr() if second else None, b, n1, n2, d, p, torch.cuda.current_stream().cuda_stream))
            return g1, g2
        got, one, two = gradients(True, True), gradients(True, False)[0], gradients(False, True)[1]
        monkeypatch.setenv("TPW_DISABLE_SMALL_BWD", "1")
        want = gradients(True, True)
        monkeypatch.delenv("TPW_DISABLE_SMALL_BWD")
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), (mode, p)
        assert torch.equal(one, want[0]) and torch.equal(two, want[1]), (mode, p)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", [(1, 75, 5, 64), (2, 300, 200, 40), (1, 1500, 1480, 100), (1, 40, 70, 12)])
def test_jensenshannon_gradients_by_rows_equal_the_tile_kernel(tpw, monkeypatch, dtype, shape):
    from torchpairwise_b200 import _abi
    b, n1, n2, d = shape
    g = torch.Generator().manual_seed(n1)
    x1, x2 = (torch.rand(b, n, d, generator=g).to(dtype).cuda() for n in (n1, n2))
    x1[:, 2, 3:7], x2[:, 1, 5] = 0, 0
    up, out = torch.randn(b, n1, n2, generator=g).to(dtype).cuda(), (torch.rand(b, n1, n2, generator=g) + 0.5).to(dtype).cuda()
    code, res = _abi.F32 if dtype == torch.float32 else _abi.F64, []
    for tile in (False, True):
        if tile:
            monkeypatch.setenv("TPW_DISABLE_SMALL_BWD", "1")
        g1, g2 = torch.full_like(x1, math.nan), torch.full_like(x2, math.nan)
        _abi.check(_abi.lib.tpw_jensenshannon_backward(code, up.data_ptr(), out.data_ptr(), x1.data_ptr(), x2.data_ptr(), g1.data_ptr(), g2.data_ptr(),
                                                       b, n1, n2, d, 0.5, torch.cuda.current_stream().cuda_stream))
        res.append((g1, g2))
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_widen_takes_more_than_one_turn(tpw, dtype):
    """More elements than the largest grid has in one turn (16 blocks of 256 threads of 8 to an SM), no multiple of eight."""
    from torchpairwise_b200 import _abi
    n = torch.cuda.get_device_properties(0).multi_processor_count * 16 * 2048 + 3 * 2048 + 5
    x = torch.randn(n, generator=torch.Generator().manual_seed(n)).to(dtype).cuda()
    out = torch.full((n + 4,), 7.0, device="cuda")
    _abi.check(_abi.lib.tpw_widen(int(dtype == torch.bfloat16), x.data_ptr(), out.data_ptr(), n, torch.cuda.current_stream().cuda_stream))
    assert torch.equal(out[:n], x.float()) and bool((out[n:] == 7).all())
