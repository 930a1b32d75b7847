"""GPU parity: pairwise distance and k-means assignment against the oracle (the reference's torch
restatement, examples/my_kmeans.py:43-64,116-125, evaluated in double)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def labels_match(oracle, x, c, metric, got):
    """Identical assignments, ignoring ties: where the label differs from the oracle's, the chosen
    centre must be as close as the best one up to fp32 rounding of the distance."""
    want, best, second = oracle.kmeans_assign(x, c, metric, with_margin=True)
    diff = np.nonzero(got != want)[0]
    if diff.size == 0:
        return True
    d = oracle.pairwise_distance(x[diff], c, metric).astype(np.float64)
    chosen = d[np.arange(diff.size), got[diff]]
    scale = np.maximum(np.abs(best[diff]), 1e-30) if metric != "cosine" else 1.0
    ok = np.abs(chosen - best[diff]) <= 4e-6 * scale + 1e-7
    return bool(ok.all()) and diff.size <= max(3, x.shape[0] // 2000)


@pytest.mark.parametrize("metric", ["l2", "cosine"])
@pytest.mark.parametrize("n,k,d", [(1000, 256, 8), (777, 256, 32), (513, 256, 64), (300, 17, 5), (64, 300, 100), (50, 40, 200), (1, 1, 1)])
def test_pairwise_distance(capi, oracle, metric, n, k, d):
    rng = np.random.default_rng(n + k + d)
    x = rng.standard_normal((n, d)).astype(np.float32)
    c = rng.standard_normal((k, d)).astype(np.float32)
    got = capi.pairwise_distance(dev(x), dev(c), metric).cpu().numpy()
    want = oracle.pairwise_distance(x, c, metric)
    assert got.shape == (n, k)
    assert np.allclose(got, want, rtol=2e-5, atol=2e-6)


@pytest.mark.parametrize("metric", ["l2", "cosine"])
@pytest.mark.parametrize("n,k,d", [(20000, 256, 8), (9999, 256, 32), (5000, 256, 64), (3000, 17, 5), (700, 300, 100), (300, 40, 200)])
def test_kmeans_assign_identical_up_to_ties(capi, oracle, metric, n, k, d):
    rng = np.random.default_rng(n + k + d + 1)
    x = rng.standard_normal((n, d)).astype(np.float32)
    c = rng.standard_normal((k, d)).astype(np.float32)
    km = capi.KMeans(dev(c), metric)
    got = km.predict(dev(x)).cpu().numpy()
    assert got.dtype == np.int64 and got.shape == (n,)
    assert labels_match(oracle, x, c, metric, got)
    assert km.get_centers().data_ptr() == km.cluster_centers.data_ptr()


def test_kmeans_exact_ties_take_first_centre(capi):
    c = torch.randn(8, 16, device="cuda")
    c2 = torch.cat([c, c])  # every centre duplicated: the first copy must win
    x = torch.randn(500, 16, device="cuda")
    for metric in ("l2", "cosine"):
        lab = capi.KMeans(c2, metric).predict(x)
        assert int(lab.max()) < 8


def test_kmeans_zero_vectors_and_fit(capi):
    x = torch.randn(4000, 8, device="cuda")
    x[:5] = 0
    c = torch.randn(16, 8, device="cuda")
    d = capi.pairwise_distance(x, c, "cosine")
    assert torch.all(d[:5] == 1.0)  # NaN distances count as 1 (examples/my_kmeans.py:92-94)
    torch.manual_seed(0)
    for metric in ("l2", "cosine"):
        km = capi.KMeans(16, 8, metric, max_iter=30)
        km.fit(x)
        centers = km.get_centers()
        assert centers.shape == (16, 8) and bool(torch.isfinite(centers).all())
        lab = km.predict(x)
        # a fit must beat random centres on its own objective
        def inertia(cc, ll):
            if metric == "cosine":
                return float((1 - torch.nn.functional.cosine_similarity(x[5:], cc[ll[5:]], dim=1)).sum())
            return float(((x - cc[ll]) ** 2).sum())
        rnd = x[torch.randperm(4000, device="cuda")[:16]].contiguous()
        assert inertia(centers, lab) < inertia(rnd, capi.KMeans(rnd, metric).predict(x))


@pytest.mark.parametrize("metric", ["l2", "cosine"])
@pytest.mark.parametrize("n,k,d", [(100_000, 256, 8), (50_000, 256, 32), (30_000, 256, 64), (4097, 100, 5), (1000, 16, 24), (129, 256, 8),
                                   (20_000, 256, 40), (20_000, 200, 49), (10_000, 64, 33)])
def test_tensor_core_assignment_equals_exact_fp32_kernel(capi, oracle, metric, n, k, d):
    """The tcgen05 path must return the labels of the exact fp32 scorer, point for point: points it cannot
    decide within the error bound of the split product are re-scored by that scorer."""
    from f2cgt_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(n + k + d)
    x = torch.randn(n, d, device="cuda", generator=g)
    c = torch.randn(k, d, device="cuda", generator=g)
    x[:3] = 0                      # zero vectors: every distance ties
    c2 = c.clone()
    if k >= 8:
        c2[k // 2] = c2[1]         # an exact duplicate centre: the lower index must win
    for centers in (c, c2):
        tc = ops.kmeans_assign(x, centers, metric, scorer="tensor")  # the tensor-core path whatever the shape heuristic says
        undecided = ops.kmeans_assign.last_undecided
        exact = ops.kmeans_assign(x, centers, metric, scorer="exact")
        assert torch.equal(tc, exact), (metric, n, k, d, int((tc != exact).sum()))
        # the split product (three products of f16 pairs) decides almost everything itself
        # (a duplicated centre makes every point that prefers it an exact tie: about 1/k of the points)
        assert undecided <= (0.02 if d <= 32 else 0.05) * n + 8 + (3.0 * n / k if centers is c2 else 0)
        if centers is c:
            assert labels_match(oracle, x.cpu().numpy(), c.cpu().numpy(), metric, tc.cpu().numpy())


@pytest.mark.parametrize("d", [8, 32, 64])
def test_tensor_core_assignment_at_table_scale(capi, d):
    """The sizes the k-means profile times: 2,449,029 sub-vectors against 256 centres (one VQ subspace of the
    2.4 M-row table), tensor-core labels == exact-scorer labels point for point, both metrics."""
    from f2cgt_b200 import ops
    n, k = 2_449_029, 256
    g = torch.Generator(device="cuda").manual_seed(d)
    x = torch.randn(n, d, device="cuda", generator=g)
    c = torch.randn(k, d, device="cuda", generator=g)
    for metric in ("l2", "cosine"):
        tc = ops.kmeans_assign(x, c, metric, scorer="tensor")
        assert ops.kmeans_assign.last_undecided <= (0.02 if d <= 32 else 0.05) * n
        exact = ops.kmeans_assign(x, c, metric, scorer="exact")
        assert torch.equal(tc, exact), (metric, d, int((tc != exact).sum()))


@pytest.mark.parametrize("metric", ["l2", "cosine"])
@pytest.mark.parametrize("n,k,d", [(1, 1, 1), (257, 16, 5), (5000, 256, 8), (1023, 17, 600), (150_001, 256, 64), (200_000, 100, 24),
                                   (3000, 300, 100)])
def test_fit_iterations_equal_the_restated_loop(capi, metric, n, k, d):
    """The queued Lloyd iterations (fixed-point sums, convergence flag on the device) against the loop of
    examples/my_kmeans.py:73-113 written with the assignment operator and float64 sums."""
    g = torch.Generator(device="cuda").manual_seed(n + k + d)
    x = torch.randn(n, d, device="cuda", generator=g) * torch.logspace(-3, 2, d, device="cuda")
    start = x[torch.randint(0, n, (k,), device="cuda", generator=g)] + 1e-3
    for max_iter, tol in ((1, 0.0), (11, 0.0), (20, 1e30)):
        want = start.clone()
        for _ in range(max_iter):
            labels = capi.kmeans_assign(x, want, metric)
            sums = torch.zeros(k, d, dtype=torch.float64, device="cuda").index_add_(0, labels, x.double())
            cnt = torch.bincount(labels, minlength=k).unsqueeze(1)
            new = torch.where(cnt > 0, sums.float() / cnt.clamp_min(1), want)
            shift, want = float(((new - want) ** 2).sum()), new
            if shift <= tol:
                break
        km = capi.KMeans(start.clone(), metric, max_iter=max_iter, tol=tol)
        km.fit(x)
        got = km.get_centers()
        assert float((got - want).norm() / want.norm()) < 1e-5
        again = capi.KMeans(start.clone(), metric, max_iter=max_iter, tol=tol)
        again.fit(x)
        assert torch.equal(got, again.get_centers())


def _fit(x, centers, iterations, spoil=False, each=None, metric=0):
    """Lloyd iterations by the C entry points, queued at once or (each) one call after the other; centres and state words."""
    from f2cgt_b200 import ops
    from f2cgt_b200._lib import check, lib
    n, d = x.shape
    k = centers.shape[0]
    up = lambda v: (v + 255) // 256 * 256  # noqa: E731
    ws = torch.empty(lib.f2c_kmeans_fit_workspace(n, k, d), dtype=torch.uint8, device="cuda")
    head = ws[256 + up(k * d * 8) + up(k * 4) + up(n * 8):][:8].view(torch.int32)
    check(lib.f2c_kmeans_fit_begin(x.data_ptr(), n, k, d, ws.data_ptr(), ops._stream(x)))
    for take in each or [iterations]:
        if spoil:
            head[1] = 3
        check(lib.f2c_kmeans_fit_iterate(x.data_ptr(), centers.data_ptr(), n, k, d, metric, 0.0, take, ws.data_ptr(), ops._stream(x)))
        if each:
            torch.cuda.synchronize()
    return centers, ws[:16].view(torch.int32).tolist()


def test_fit_goes_on_after_an_assignment_whose_wait_ran_out(capi):
    """The tensor-core kernel's word for a bounded wait that ran out makes the exact scorer assign every point; the fit takes those
    labels and goes on.  The word is set by the host here."""
    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(5000, 16, generator=g, device="cuda")
    want, words = _fit(x, x[:64].clone(), 6)
    got, spoiled = _fit(x, x[:64].clone(), 6, spoil=True)
    assert spoiled[:3] == words[:3]
    assert spoiled[3] == 3 and torch.equal(want, got)


@pytest.mark.parametrize("n,k,d", [(1, 1, 4), (129, 100, 8), (40_000, 256, 13), (70_001, 200, 64)])
def test_a_lost_wait_leaves_the_exact_labels_and_sums(capi, n, k, d):
    """Every bounded wait of the tensor-core kernel runs out at once, with the first rows on their way into shared memory: the error word says
    so, all points have the exact scorer's labels, and a fit ends at the centres, bit for bit, of one without such waits."""
    from f2cgt_b200 import _lib, _native, ops
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, d, generator=g, device="cuda")
    c = torch.randn(k, d, generator=g, device="cuda")
    x[::5] = 0
    for metric in ("l2", "cosine"):
        flags = ops._metric(metric) | _lib.SCORER_TENSOR
        labels, head = _native.kmeans_assign(x, c, flags | _lib.NO_WAITS)
        assert torch.equal(labels, ops.kmeans_assign(x, c, metric, scorer="exact"))
        assert head[:2].tolist() == [n, 1]
        assert torch.equal(_native.kmeans_assign(x, c, flags)[0], labels)  # and the next call finds the device as it was
        want, words = _fit(x, c.clone(), 4, metric=ops._metric(metric))
        got, lost = _fit(x, c.clone(), 4, each=[1, 3], metric=ops._metric(metric) | _lib.NO_WAITS)
        assert torch.equal(want, got) and lost[:3] == words[:3] and words[3] == 0 and lost[3] == 1


def test_iterations_in_a_row_equal_iterations_one_by_one(capi):
    """Eight iterations queued at once, which one kernel makes, and eight with the device idle between."""
    g = torch.Generator(device="cuda").manual_seed(0)
    for n, d, k in ((5000, 16, 64), (30000, 8, 256), (20000, 64, 200)):
        x = torch.randn(n, d, generator=g, device="cuda")
        a, w1 = _fit(x, x[:k].clone(), 8)
        b, w2 = _fit(x, x[:k].clone(), 0, each=[1] * 8)
        assert torch.equal(a, b) and w1 == w2


def test_a_launch_of_a_large_fit_has_few_iterations(capi):
    """Other streams' kernels get in between: 3,000,000 points have five iterations per launch, so seven are two launches (or seven, one by one)."""
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(3_000_000, 8, generator=g, device="cuda")
    a, w1 = _fit(x, x[:100].clone(), 7)
    b, w2 = _fit(x, x[:100].clone(), 0, each=[1] * 7)
    assert torch.equal(a, b) and w1 == w2 and w1[:2] == [0, 7]
    import ctypes
    from f2cgt_b200._lib import check, lib
    rt = ctypes.CDLL("libcudart.so.12")  # torch's: the launches of a call are the nodes of its capture
    ws = torch.empty(lib.f2c_kmeans_fit_workspace(x.shape[0], 100, 8), dtype=torch.uint8, device="cuda")
    stream, graph, launches = torch.cuda.Stream(), ctypes.c_void_p(), ctypes.c_size_t()
    handle = ctypes.c_void_p(stream.cuda_stream)
    assert rt.cudaStreamBeginCapture(handle, 2) == 0
    rc = lib.f2c_kmeans_fit_iterate(x.data_ptr(), a.data_ptr(), x.shape[0], 100, 8, 0, 0.0, 7, ws.data_ptr(), stream.cuda_stream)
    assert rt.cudaStreamEndCapture(handle, ctypes.byref(graph)) == 0
    check(rc)
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(launches)) == 0 and rt.cudaGraphDestroy(graph) == 0
    assert launches.value == 2


@pytest.mark.parametrize("n,k,d", [(5000, 8, 5), (40_000, 16, 64), (3000, 4, 300), (700, 2, 5000)])
def test_fit_keeps_the_precision_of_small_columns(capi, n, k, d):
    """Columns of very different sizes: a centre's entries are as precise as fp32 in each of them (exact sums, one rounding to float32,
    one division), whatever the largest column holds."""
    g = torch.Generator(device="cuda").manual_seed(d)
    size = torch.logspace(9, -12, d, device="cuda")[torch.randperm(d, generator=g, device="cuda")]
    x = torch.rand(n, d, generator=g, device="cuda").add_(0.5) * size
    start = x[:k].clone()
    labels = capi.kmeans_assign(x, start, "l2")
    got, words = _fit(x, start.clone(), 1)
    want = torch.zeros(k, d, dtype=torch.float64, device="cuda").index_add_(0, labels, x.double())
    want /= torch.bincount(labels, minlength=k).double()[:, None]
    assert words[1] == 1 and float(((got.double() - want).abs() / want).max()) < 2.0**-22  # two roundings of 2^-24, doubled


@pytest.mark.parametrize("d", [1, 7, 8, 13, 16, 24, 31, 32, 40, 48, 52, 56, 64])
def test_tensor_core_assignment_at_the_edges_of_its_tiles(capi, d):
    """Chunk counts, both column counts, one to four tiles per CTA with ragged ends, rows that start off a 16-byte boundary, magnitudes far
    from one: labels of the exact fp32 scorer, call after call (a lost wait shows now and then only)."""
    from f2cgt_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(d)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n in (1, 127, 129, sms * 128 + 1, 3 * sms * 128 + 77):
        for k in (1, 128, 129, 256):
            offset = (n + k) % 3
            x = torch.randn(n * d + offset, device="cuda", generator=g)[offset:].view(n, d)
            c = torch.randn(k * d + offset, device="cuda", generator=g)[offset:].view(k, d)
            for metric, size in (("l2", 1.0), ("cosine", 1.0), ("cosine", 1e-15), ("cosine", 1e15)):
                y = x if size == 1.0 else (x * size).contiguous()
                exact = ops.kmeans_assign(y, c, metric, scorer="exact")
                for _ in range(3):
                    assert torch.equal(ops.kmeans_assign(y, c, metric, scorer="tensor"), exact), (n, k, metric, size)


@pytest.mark.parametrize("d", [5, 8, 32, 64])
def test_rows_and_centres_whose_squared_length_underflows(capi, d):
    """fp32 holds no square below 1.4e-45: the exact scorer gives short rows label 0 (all cosine distances are 1, all squared ones 0) and loses bits
    before that.  The tensor cores, which scale their operands, must not know better; nor where half the rows or one centre are that short."""
    from f2cgt_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(d)
    x = torch.randn(3001, d, device="cuda", generator=g)
    c = torch.randn(100, d, device="cuda", generator=g)
    x[7], c[7] = 0, 0
    for size in (1e-14, 1e-17, 1e-20, 1e-22, 1e-30, 1e-41):
        tiny, mixed, one = x * size, x.clone(), c.clone()
        mixed[::2] *= size
        one[11] *= size
        for metric in ("l2", "cosine"):
            for data, centres in ((tiny, c), (mixed, c), (x, one), (tiny, c * size), (tiny, one), (mixed, one)):
                exact = ops.kmeans_assign(data, centres, metric, scorer="exact")
                assert torch.equal(ops.kmeans_assign(data, centres, metric, scorer="tensor"), exact), (size, metric)


@pytest.mark.parametrize("d,k", [(8, 40), (40, 200)])
@pytest.mark.parametrize("twins", [1.0, 0.5])
def test_more_undecided_points_than_a_cta_lists(capi, d, k, twins):
    """A CTA lists 1024 undecided points and finds them by their labels when there are more, as many at a time as it has threads: all of its 1536
    points and more are undecided here (every centre has a twin: whole rounds), or about half of 5120 (the rest of a round moves on)."""
    from f2cgt_b200 import ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = sms * 128 * (12 if twins == 1.0 else 40) + 77
    g = torch.Generator(device="cuda").manual_seed(d)
    x = torch.randn(n, d, device="cuda", generator=g)
    c = torch.randn(k, d, device="cuda", generator=g)
    own = int(k / 2 if twins == 1.0 else k * twins / (1 + twins))
    c[k - own:] = c[:own]
    for metric in ("l2", "cosine"):
        labels = ops.kmeans_assign(x, c, metric, scorer="tensor")
        undecided = ops.kmeans_assign.last_undecided
        assert torch.equal(labels, ops.kmeans_assign(x, c, metric, scorer="exact"))
        assert undecided == n if twins == 1.0 else 1400 * sms < undecided < n - 704 * sms


@pytest.mark.parametrize("n,k,d", [(1, 1, 4), (127, 128, 8), (1025, 129, 24), (70_000, 256, 13), (200_003, 33, 64), (40_000, 200, 40)])
def test_fit_kernel_at_the_edges_of_its_tiles(capi, n, k, d):
    """Ragged tiles, one to many chunks of points per CTA, many points that the tensor cores leave open (every second centre is a copy,
    a third of the rows is zero), rows off a 16-byte boundary: the centres of a loop over the exact assignment with float64 sums."""
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n * d + 1, generator=g, device="cuda")[1:].view(n, d)
    x[::3] = 0
    start = torch.randn(k, d, generator=g, device="cuda")
    start[1::2] = start[:k - k % 2:2]
    from f2cgt_b200 import ops
    for metric in ("l2", "cosine"):
        want = start.clone()
        for _ in range(3):
            labels = ops.kmeans_assign(x.contiguous(), want, metric, scorer="exact")
            sums = torch.zeros(k, d, dtype=torch.float64, device="cuda").index_add_(0, labels, x.double())
            cnt = torch.bincount(labels, minlength=k).unsqueeze(1)
            want = torch.where(cnt > 0, sums.float() / cnt.clamp_min(1), want)
        km = capi.KMeans(start.clone(), metric, max_iter=3, tol=-1.0)
        km.fit(x)
        # fixed-point sums are exact, float64 ones to 2^-53 of the largest partial sum: both round to the same float32 but for its last bit
        assert float((km.get_centers() - want).abs().max()) <= 2.0**-22 * float(want.abs().max())
