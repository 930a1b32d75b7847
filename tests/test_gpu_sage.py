"""GPU: the DGL-free GraphSAGE stack (mirror of examples/conv.py, examples/models.py, examples/dataloader.py of the
reference) against a plain-torch restatement on decoded features."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def torch_mean_aggregate(h, indptr, indices):
    n_dst = indptr.numel() - 1
    indices = indices[:int(indptr[-1])]  # the loader's index tensors may carry an unused tail behind indptr[-1]
    deg = indptr[1:] - indptr[:-1]
    dst = torch.repeat_interleave(torch.arange(n_dst, device=h.device), deg)
    out = torch.zeros(n_dst, h.shape[1], device=h.device, dtype=h.dtype).index_add_(0, dst, h[indices])
    return out / deg.clamp_min(1).to(h.dtype)[:, None]


def test_mean_aggregate_forward_and_backward(capi):
    from f2cgt_b200 import sage
    g = torch.Generator(device="cuda").manual_seed(0)
    n_src, n_dst, H = 500, 200, 64
    deg = torch.randint(0, 9, (n_dst,), generator=g, device="cuda")
    indptr = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cumsum(deg, 0)])
    indices = torch.randint(0, n_src, (int(indptr[-1]),), generator=g, device="cuda")
    h = torch.randn(n_src, H, generator=g, device="cuda", requires_grad=True)
    w = torch.randn(n_dst, H, generator=g, device="cuda")
    out = sage._MeanAggregate.apply(h, indptr, indices, n_src)
    (out * w).sum().backward()
    got_grad = h.grad.clone()
    h.grad = None
    ref = torch_mean_aggregate(h, indptr, indices)
    (ref * w).sum().backward()
    assert torch.allclose(out, ref, rtol=1e-5, atol=1e-6)
    assert torch.allclose(got_grad, h.grad, rtol=1e-5, atol=1e-6)


def test_sage_forward_equals_torch_on_decoded_features(capi):
    """Two-level compressed input: the model's output equals the same network evaluated on features decoded row by row."""
    from f2cgt_b200 import ops, sage, synth
    dev = "cuda"
    n, D, hidden, classes = 30000, 128, 64, 10
    indptr, indices = synth.power_law_graph(n, 15, 2.1, seed=1, device=dev)
    g = torch.Generator(device=dev).manual_seed(2)
    vq_codes = torch.randint(0, 256, (n, 4), generator=g, dtype=torch.uint8, device=dev)
    vq_cbs = torch.randn(4, 256, 32, generator=g, device=dev)
    n_hot = 1500
    hot = torch.randperm(n, generator=g, device=dev)[:n_hot]
    slot = torch.full((n,), -1, dtype=torch.int32, device=dev)
    slot[hot] = torch.arange(n_hot, dtype=torch.int32, device=dev)
    sq_codes = torch.randint(-128, 128, (n_hot, D), generator=g, dtype=torch.int8, device=dev)
    sq_cb = synth.sq_codebook_from_sample(torch.randn(5000, D, generator=g, device=dev), D)
    cm = sage.CompressionManager(D, ["sq", "vq"], [(D, 8), (32, 8)], [sq_cb, vq_cbs], [sq_codes, vq_codes], slot)
    full = ops.vq_decompress(vq_codes, vq_cbs, D)
    full[hot] = ops.sq_decompress(sq_codes, sq_cb, 8, D, D)
    torch.manual_seed(0)
    model = sage.SAGE(D, hidden, classes, 3, 0.5, cm).to(dev).eval()
    seeds = torch.randperm(n, generator=g, device=dev)[:128]
    loader = sage.GPUSamplingDataloader(indptr, indices, seeds, 128, (5, 4, 3), shuffle=False)
    input_nodes, output_nodes, blocks = next(iter(loader))
    assert torch.equal(output_nodes, seeds) and torch.equal(blocks[0]["src_nodes"], input_nodes)
    assert torch.equal(cm.decode_rows(input_nodes), full[input_nodes])  # identity-CSC decode is the row decode, bit for bit
    got = model(blocks)
    h = full[input_nodes]
    for i, (layer, b) in enumerate(zip(model.layers, blocks)):
        n_dst = b["dst_nodes"].numel()
        h = layer.fc_self(h[:n_dst]) + layer.fc_neigh(torch_mean_aggregate(h, b["indptr"], b["indices_local"]))
        if i != 2:
            h = torch.relu(h)
    assert got.shape == (128, classes)
    assert torch.allclose(got, h, rtol=1e-4, atol=1e-4)


def test_training_learns_a_feature_rule(capi):
    """Labels that depend on the decoded features of the node itself are learnable through the compressed path."""
    from f2cgt_b200 import ops, sage, synth
    dev = "cuda"
    n, D = 20000, 128
    indptr, indices = synth.power_law_graph(n, 10, 2.1, seed=4, device=dev)
    codes, cb = synth.sq_table_from_normal(n, D, 8, D, seed=5, device=dev)
    cm = sage.CompressionManager(D, ["sq"], [(D, 8)], [cb], [codes])
    feats = ops.sq_decompress(codes, cb, 8, D, D)
    labels = (feats[:, 0] > 0).long() + 2 * (feats[:, 1] > 0).long()
    torch.manual_seed(0)
    model = sage.SAGE(D, 64, 4, 2, 0.0, cm).to(dev)
    opt = torch.optim.Adam(model.parameters(), lr=0.01)
    train_ids = torch.arange(8192, device=dev)
    loader = sage.GPUSamplingDataloader(indptr, indices, train_ids, 512, (5, 5), shuffle=True)
    first = last = None
    for epoch in range(6):
        for _, out_nodes, blocks in loader:
            loss = torch.nn.functional.cross_entropy(model(blocks), labels[out_nodes])
            opt.zero_grad()
            loss.backward()
            opt.step()
            first = float(loss.detach()) if first is None else first
            last = float(loss.detach())
    assert last < 0.5 * first, (first, last)


def _two_level_setup(dev="cuda"):
    from f2cgt_b200 import ops, sage, synth
    n, D = 30000, 128
    indptr, indices = synth.power_law_graph(n, 15, 2.1, seed=1, device=dev)
    g = torch.Generator(device=dev).manual_seed(2)
    vq_codes = torch.randint(0, 256, (n, 4), generator=g, dtype=torch.uint8, device=dev)
    vq_cbs = torch.randn(4, 256, 32, generator=g, device=dev)
    n_hot = 1500
    hot = torch.randperm(n, generator=g, device=dev)[:n_hot]
    slot = torch.full((n,), -1, dtype=torch.int32, device=dev)
    slot[hot] = torch.arange(n_hot, dtype=torch.int32, device=dev)
    sq_codes = torch.randint(-128, 128, (n_hot, D), generator=g, dtype=torch.int8, device=dev)
    sq_cb = synth.sq_codebook_from_sample(torch.randn(5000, D, generator=g, device=dev), D)
    cm = sage.CompressionManager(D, ["sq", "vq"], [(D, 8), (32, 8)], [sq_cb, vq_cbs], [sq_codes, vq_codes], slot)
    full = ops.vq_decompress(vq_codes, vq_cbs, D)
    full[hot] = ops.sq_decompress(sq_codes, sq_cb, 8, D, D)
    return n, D, indptr, indices, cm, full, g


def test_sage_gradients_equal_autograd_of_the_plain_network(capi):
    """The hand-written backward of the layers (rows padded to recurring counts and carried through the network) gives
    the gradients autograd computes for the same network written with Linear layers on decoded features."""
    from f2cgt_b200 import sage
    n, D, indptr, indices, cm, full, g = _two_level_setup()
    hidden, classes = 64, 10
    torch.manual_seed(0)
    model = sage.SAGE(D, hidden, classes, 3, 0.0, cm).cuda()
    seeds = torch.randperm(n, generator=g, device="cuda")[:300]  # 300: not a multiple of the row bucket
    loader = sage.GPUSamplingDataloader(indptr, indices, seeds, 300, (5, 4, 3), shuffle=False)
    input_nodes, _, blocks = next(iter(loader))
    y = torch.randint(0, classes, (300,), generator=g, device="cuda")
    got = model(blocks)
    assert got.shape == (300, classes)
    torch.nn.functional.cross_entropy(got, y).backward()
    mine = [p.grad.clone() for p in model.parameters()]
    model.zero_grad(set_to_none=True)
    h = full[input_nodes]
    for i, (layer, b) in enumerate(zip(model.layers, blocks)):
        n_dst = b["dst_nodes"].numel()
        h = layer.fc_self(h[:n_dst]) + layer.fc_neigh(torch_mean_aggregate(h, b["indptr"], b["indices_local"]))
        if i != 2:
            h = torch.relu(h)
    assert torch.allclose(got, h, rtol=1e-4, atol=1e-4)
    torch.nn.functional.cross_entropy(h, y).backward()
    for a, p in zip(mine, model.parameters()):
        assert torch.allclose(a, p.grad, rtol=1e-3, atol=1e-5), float((a - p.grad).abs().max())


def test_hidden_layer_on_unpadded_input(capi):
    """SAGEConv called by hand with exactly n_src rows (fewer than the row bucket of its n_dst): output and gradients."""
    from f2cgt_b200 import sage
    g = torch.Generator(device="cuda").manual_seed(3)
    n_src, n_dst, H = 150, 140, 32
    deg = torch.randint(0, 6, (n_dst,), generator=g, device="cuda")
    indptr = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), torch.cumsum(deg, 0)])
    indices = torch.randint(0, n_src, (int(indptr[-1]),), generator=g, device="cuda")
    block = dict(dst_nodes=torch.arange(n_dst, device="cuda"), indptr=indptr, indices_local=indices)
    torch.manual_seed(1)
    layer = sage.SAGEConv(H, 16).cuda()
    h = torch.randn(n_src, H, generator=g, device="cuda", requires_grad=True)
    w = torch.randn(n_dst, 16, generator=g, device="cuda")
    out = layer(block, h)
    assert out.shape == (n_dst, 16)
    (out * w).sum().backward()
    got = [h.grad.clone()] + [p.grad.clone() for p in layer.parameters()]
    h.grad = None
    layer.zero_grad(set_to_none=True)
    ref = layer.fc_self(h[:n_dst]) + layer.fc_neigh(torch_mean_aggregate(h, indptr, indices))
    (ref * w).sum().backward()
    assert torch.allclose(out, ref, rtol=1e-5, atol=1e-5)
    for a, b in zip(got, [h.grad] + [p.grad for p in layer.parameters()]):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-5)


def test_loader_builds_the_same_minibatches_ahead_or_in_step(capi):
    """Minibatches built one step early on the side stream (with and without poke() calls in between) are those of the
    in-step loader, tensor for tensor."""
    from f2cgt_b200 import sage, synth
    indptr, indices = synth.power_law_graph(20000, 12, 2.1, seed=7, device="cuda")
    seeds = torch.arange(0, 5000, device="cuda")

    def run(ahead, poke):
        loader = sage.GPUSamplingDataloader(indptr, indices, seeds, 512, (4, 3), shuffle=True, rng_seed=5, ahead=ahead)
        out = []
        for _epoch in range(2):
            for input_nodes, output_nodes, blocks in loader:
                for _ in range(poke):
                    torch.cuda.synchronize()
                    loader.poke()
                out.append([input_nodes.clone(), output_nodes.clone()] +
                           [b[k][:int(b["indptr"][-1])].clone() if k.startswith("indices") else b[k].clone()
                            for b in blocks for k in ("indptr", "indices_global", "indices_local", "src_nodes", "dst_nodes")])
        return out
    base = run(False, 0)
    assert len(base) == 2 * 10
    for ahead, poke in ((True, 0), (True, 1), (True, 3)):
        other = run(ahead, poke)
        assert len(other) == len(base)
        for a, b in zip(base, other):
            assert all(torch.equal(x, y) for x, y in zip(a, b))


def test_direct_fused_adam_equals_torch_adam(capi):
    """The trainer's optimizer calls the fused Adam kernel itself; three steps give torch.optim.Adam(fused=True)'s weights."""
    from f2cgt_b200 import train_graphsage as tg
    if not tg.DirectFusedAdam.available():
        pytest.skip("this torch does not expose the fused Adam kernel")
    torch.manual_seed(0)
    a = [torch.randn(64, 32, device="cuda", requires_grad=True), torch.randn(64, device="cuda", requires_grad=True)]
    b = [t.detach().clone().requires_grad_(True) for t in a]
    mine, ref = tg.DirectFusedAdam(a, lr=0.003), torch.optim.Adam(b, lr=0.003, fused=True)
    for step in range(3):
        g = [torch.randn_like(t) for t in a]
        for t, u, gg in zip(a, b, g):
            t.grad, u.grad = gg.clone(), gg.clone()
        mine.step()
        ref.step()
        mine.lr *= 0.978
        for grp in ref.param_groups:
            grp["lr"] *= 0.978
    for t, u in zip(a, b):
        assert torch.equal(t, u)


def test_bf16_product_operands_stay_close_to_fp32(capi):
    """``sage.products_in(torch.bfloat16)``: same network, product operands rounded to bf16, fp32 everywhere else - output
    and gradients within bf16 rounding of the fp32 run, all finite."""
    from f2cgt_b200 import sage
    n, D, indptr, indices, cm, full, g = _two_level_setup()
    torch.manual_seed(0)
    model = sage.SAGE(D, 64, 10, 3, 0.0, cm).cuda()
    seeds = torch.randperm(n, generator=g, device="cuda")[:256]
    loader = sage.GPUSamplingDataloader(indptr, indices, seeds, 256, (5, 4, 3), shuffle=False)
    _, _, blocks = next(iter(loader))
    y = torch.randint(0, 10, (256,), generator=g, device="cuda")
    want = model(blocks)
    torch.nn.functional.cross_entropy(want, y).backward()
    want_grads = [p.grad.clone() for p in model.parameters()]
    model.zero_grad(set_to_none=True)
    with sage.products_in(torch.bfloat16):
        got = model(blocks)
        torch.nn.functional.cross_entropy(got, y).backward()
    assert got.dtype == torch.float32 and torch.isfinite(got).all()
    # bf16 keeps 8 bits of mantissa: ~0.4 % per operand, through three layers of 64- to 128-term dot products
    scale = float(want.detach().abs().max())
    assert float((got.detach() - want.detach()).abs().max()) < 0.05 * scale
    for a, p in zip(want_grads, model.parameters()):
        assert p.grad.dtype == torch.float32 and torch.isfinite(p.grad).all()
        assert float((p.grad - a).abs().max()) < 0.15 * float(a.abs().max()) + 1e-6
    assert sage._PRODUCT_DTYPE is None  # the context manager restored the default


@pytest.mark.parametrize("m,n,k", [(1, 1, 4), (127, 16, 32), (128, 128, 128), (129, 172, 100), (1000, 171, 64), (4097, 128, 256), (300, 300, 260),
                                   (40_001, 64, 128), (600, 47, 12)])
def test_layer_product_on_tensor_cores(capi, m, n, k):
    """Forward product of a layer against float64 (operands carry 10 mantissa bits); rows behind m stay untouched."""
    from f2cgt_b200 import ops
    from f2cgt_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x1, x2, w1, w2, b = rnd(m, k), rnd(m, k), rnd(n, k), rnd(n, k), rnd(n)
    sums = x1.double() @ w1.double().t() + x2.double() @ w2.double().t()
    parts = x1.double().abs() @ w1.double().abs().t() + x2.double().abs() @ w2.double().abs().t()
    for relu in (0, 1):
        for bias in (b, None):
            y = torch.full((m + 1, n), float("nan"), device="cuda")
            check(lib.f2c_sage_forward(x1.data_ptr(), x2.data_ptr(), w1.data_ptr(), w2.data_ptr(), 0 if bias is None else bias.data_ptr(),
                                       y.data_ptr(), m, n, k, relu, ops._stream(x1)))
            want = sums if bias is None else sums + bias.double()
            want = want.clamp_min(0) if relu else want
            assert bool(((y[:m].double() - want).abs() <= 1.5e-3 * parts + 1e-6).all()) and bool(y[m].isnan().all())
    assert ops.device_status() == 0


@pytest.mark.parametrize("rows,n", [(1, 1), (1000, 128), (4097, 47), (333, 260), (5, 1500)])
def test_relu_dropout_mask_and_bias_gradient(capi, rows, n):
    from f2cgt_b200 import ops
    from f2cgt_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(rows + n)
    grad, h, db = torch.randn(rows, n, generator=g, device="cuda"), torch.randn(rows, n, generator=g, device="cuda"), torch.ones(n, device="cuda")
    dy = torch.empty_like(grad)
    check(lib.f2c_sage_mask(grad.data_ptr(), h.data_ptr(), 2.0, dy.data_ptr(), db.data_ptr(), rows, n, ops._stream(h)))
    want = torch.where(h > 0, grad * 2.0, 0.0)
    assert torch.equal(dy, want)
    assert torch.allclose(db.double(), 1 + want.double().sum(0), rtol=1e-5, atol=1e-5 * rows**0.5)


@pytest.mark.parametrize("tf32,product,D,hidden,classes,dropout", [(True, None, 128, 128, 172, 0.5), (True, None, 100, 64, 47, 0.0), (False, None, 64, 96, 10, 0.5),
                                                                   (True, torch.bfloat16, 128, 64, 20, 0.3), (True, None, 64, 30, 7, 0.5)])
def test_network_as_one_node_equals_the_layers(capi, tf32, product, D, hidden, classes, dropout):
    """One autograd node for the whole network == its layers called one by one (same dropout masks), forward and gradients;
    a batch that is no multiple of the padding, with and without gradients."""
    from f2cgt_b200 import sage, synth
    n = 20000
    indptr, indices = synth.power_law_graph(n, 12, 2.1, seed=1, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(5)
    codes = torch.randint(0, 256, (n, (D + 31) // 32), generator=g, dtype=torch.uint8, device="cuda")
    cm = sage.CompressionManager(D, ["vq"], [(32, -1)], [torch.randn((D + 31) // 32, 256, 32, generator=g, device="cuda")], [codes])
    seeds = torch.randperm(n, generator=g, device="cuda")[:233]
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = tf32
    try:
        torch.manual_seed(1)
        model = sage.SAGE(D, hidden, classes, 3, dropout, cm).to("cuda")
        _, _, blocks = next(iter(sage.GPUSamplingDataloader(indptr, indices, seeds, 233, (6, 5, 4), shuffle=False)))
        weight = torch.randn(233, classes, generator=g, device="cuda")
        got = []
        for one_node in (True, False):
            handle = None if one_node else model.layers[1].register_forward_pre_hook(lambda *_: None)  # a hook: layer by layer
            assert (model._plain_weights() is not None) == one_node
            torch.manual_seed(7)
            model.zero_grad(set_to_none=True)
            with sage.products_in(product):
                out = model(blocks)
                (out * weight).sum().backward()
            with torch.no_grad():
                quiet = model.eval()(blocks)
            model.train()
            got.append([out.detach(), quiet] + [p.grad for p in model.parameters()])
            if handle is not None:
                handle.remove()
        tol = 1e-5 if not tf32 else 5e-3 if product is None else 2e-2
        for a, b in zip(*got):
            assert a.shape == b.shape and float((a - b).norm() / b.norm()) < tol
    finally:
        torch.backends.cuda.matmul.allow_tf32 = before


@pytest.mark.parametrize("m,n,k", [(5, 7, 64), (300, 128, 128), (129, 172, 100)])
def test_layer_product_keeps_not_a_number(capi, m, n, k):
    """ReLU as torch.relu has it: a NaN sum stays NaN, infinities keep their sign's side."""
    from f2cgt_b200 import ops
    from f2cgt_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(m)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    x1, x2, w1, w2, b = rnd(m, k), rnd(m, k), rnd(n, k), rnd(n, k), rnd(n)
    x1[1, 3], x2[3, k - 1], b[2], b[3], b[4] = float("nan"), float("inf"), float("nan"), float("inf"), float("-inf")
    y = torch.empty((m, n), device="cuda")
    check(lib.f2c_sage_forward(x1.data_ptr(), x2.data_ptr(), w1.data_ptr(), w2.data_ptr(), b.data_ptr(), y.data_ptr(), m, n, k, 1, ops._stream(x1)))
    want = torch.relu(x1.double() @ w1.double().t() + b.double() + x2.double() @ w2.double().t())
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf())


def _with_specials(shape, g, values):
    t = torch.randn(*shape, generator=g, device="cuda")
    pick = torch.randint(0, 3 * len(values), shape, generator=g, device="cuda")
    for i, v in enumerate(values):
        t[pick == i] = v
    return t


@pytest.mark.parametrize("rows,n", [(1, 3), (700, 96), (333, 47), (6, 1500)])
@pytest.mark.parametrize("dropout", [False, True])
def test_relu_dropout_gradient_equals_torch_for_every_value(capi, rows, n, dropout):
    """Zeros, infinities and NaN in the activations and in the gradient: element by element what torch's own backward gives."""
    from f2cgt_b200 import ops
    from f2cgt_b200._lib import check, lib
    inf, nan = float("inf"), float("nan")
    g = torch.Generator(device="cuda").manual_seed(rows + n)
    grad, x = _with_specials((rows, n), g, [0.0, inf, -inf, nan]), _with_specials((rows, n), g, [0.0, -0.0, inf, -inf, nan])
    x.requires_grad_()
    active = torch.relu(x)
    keep = torch.rand(rows, n, generator=g, device="cuda") < 0.6
    active.backward(torch.ops.aten.native_dropout_backward(grad, keep, 2.5) if dropout else grad)
    active = active.detach()
    dy, db = torch.empty_like(grad), torch.zeros(n, device="cuda")
    if dropout:
        h = active * keep * 2.5
        check(lib.f2c_sage_mask_dropout(grad.data_ptr(), h.data_ptr(), active.data_ptr(), keep.data_ptr(), 2.5, dy.data_ptr(), db.data_ptr(), rows, n,
                                        ops._stream(dy)))
    else:
        check(lib.f2c_sage_mask(grad.data_ptr(), active.data_ptr(), 1.0, dy.data_ptr(), db.data_ptr(), rows, n, ops._stream(dy)))
    assert torch.equal(dy.nan_to_num(7.0, 8.0, 9.0), x.grad.nan_to_num(7.0, 8.0, 9.0))
    assert torch.equal(db.isnan(), x.grad.sum(0).isnan())


def _small_network(dropout, classes=10, hidden=64, layers=3, codebook=None, n=20000, D=128):
    from f2cgt_b200 import sage, synth
    indptr, indices = synth.power_law_graph(n, 12, 2.1, seed=1, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(5)
    codes = torch.randint(0, 256, (n, D // 32), generator=g, dtype=torch.uint8, device="cuda")
    books = torch.randn(D // 32, 256, 32, generator=g, device="cuda")
    if codebook is not None:
        codebook(books)
    cm = sage.CompressionManager(D, ["vq"], [(32, -1)], [books], [codes])
    torch.manual_seed(1)
    model = sage.SAGE(D, hidden, classes, layers, dropout, cm).to("cuda")
    seeds = torch.randperm(n, generator=g, device="cuda")[:233]
    _, _, blocks = next(iter(sage.GPUSamplingDataloader(indptr, indices, seeds, 233, (6, 5, 4)[:layers], shuffle=False)))
    return model, blocks, g


@pytest.mark.parametrize("tf32", [True, False])
@pytest.mark.parametrize("dropout", [0.0, 0.5, 1.0])
@pytest.mark.parametrize("where", ["features", "gradient", "weight"])
def test_network_as_one_node_keeps_not_a_number_where_the_layers_do(capi, tf32, dropout, where):
    """NaN and infinities in the features, in a weight or in the gradient of the output show up in the same outputs and gradients
    as when the layers are called one by one."""
    inf, nan = float("inf"), float("nan")

    def spoil(books):
        books[0, 3, 5], books[1, 7, 2] = nan, inf
    model, blocks, g = _small_network(dropout, codebook=spoil if where == "features" else None)
    if where == "weight":
        with torch.no_grad():
            model.layers[0].fc_self.weight[3, 4] = nan
            model.layers[1].fc_neigh.weight[5, 6] = inf
    weight = torch.randn(233, 10, generator=g, device="cuda")
    if where == "gradient":
        weight[5, 3], weight[100, 4], weight[7] = nan, inf, 0.0
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = tf32
    try:
        got = []
        for one_node in (True, False):
            handle = None if one_node else model.layers[1].register_forward_pre_hook(lambda *_: None)  # a hook: layer by layer
            torch.manual_seed(7)
            model.zero_grad(set_to_none=True)
            out = model(blocks)
            out.backward(weight)
            got.append([out.detach()] + [p.grad for p in model.parameters()])
            if handle is not None:
                handle.remove()
    finally:
        torch.backends.cuda.matmul.allow_tf32 = before
    assert any(bool(t.isnan().any()) for t in got[1])
    for i, (a, b) in enumerate(zip(*got)):
        assert torch.equal(a.isnan(), b.isnan()), (i, int(a.isnan().sum()), int(b.isnan().sum()))
        assert torch.equal(a.isinf(), b.isinf()), i


def _report(code):
    from f2cgt_b200._lib import check, lib
    check(lib.f2c_device_status_report(code, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()


def test_network_raises_when_a_wait_ran_out_in_an_earlier_kernel(capi):
    """A bounded wait that ran out leaves a report; the passes that follow raise until it has been read."""
    from f2cgt_b200 import ops
    model, blocks, _ = _small_network(0.5)
    out = model(blocks)
    assert ops.device_status() == 0
    _report(3)
    with pytest.raises(RuntimeError, match="bounded wait"):
        model(blocks)
    with pytest.raises(RuntimeError, match="bounded wait"):
        out.sum().backward()
    assert ops.device_status() == 3 and ops.device_status() == 0
    model(blocks).sum().backward()
    assert ops.device_status() == 0


def test_training_does_not_return_when_a_wait_ran_out(capi, monkeypatch):
    from f2cgt_b200 import ops, sage, train_graphsage as tg
    monkeypatch.setitem(tg.PRESETS, "small", dict(tg.PRESETS["small"], nodes=5000, degree=10, train=512, fan_out=(3, 3)))
    assert tg.train(epochs=1, batch_size=256)["epochs_run"] == 1
    pokes = []
    monkeypatch.setattr(sage.GPUSamplingDataloader, "poke", lambda self: pokes.append(0) or len(pokes) == 3 and _report(1))  # behind the last step
    with pytest.raises(RuntimeError, match="bounded wait"):
        tg.train(epochs=1, batch_size=256, max_steps=1)
    assert ops.device_status() == 0 and not torch.backends.cuda.matmul.allow_tf32  # the switch is back where it was


@pytest.mark.parametrize("layers", [1, 2, 3])
def test_gradients_with_a_graph(capi, layers):
    """create_graph=True: one layer is differentiable twice, as its products are; more layers give the same first gradients and
    refuse the second derivative instead of leaving it out."""
    model, blocks, _ = _small_network(0.0, layers=layers)
    params = list(model.parameters())
    plain = torch.autograd.grad(model(blocks).square().mean(), params)
    grads = torch.autograd.grad(model(blocks).square().mean(), params, create_graph=True)
    assert all(x.requires_grad for x in grads)
    assert all(torch.allclose(a, b, rtol=1e-4, atol=1e-6) for a, b in zip(plain, grads))
    if layers > 1:
        with pytest.raises(RuntimeError, match="differentiated twice"):
            sum(x.square().sum() for x in grads).backward()
        with pytest.raises(RuntimeError, match="differentiated twice"):
            torch.autograd.grad(grads[0].sum(), params)
        return
    sum(x.square().sum() for x in grads).backward()
    got = [p.grad.clone() for p in params]
    model.zero_grad(set_to_none=True)
    model.layers[0].register_forward_pre_hook(lambda *_: None)  # a hook: the layer on its own
    grads = torch.autograd.grad(model(blocks).square().mean(), params, create_graph=True)
    sum(x.square().sum() for x in grads).backward()
    assert all(torch.allclose(a, p.grad, rtol=1e-4, atol=1e-6) for a, p in zip(got, params))


def test_saved_tensor_hooks_see_the_activations(capi):
    """What the backward pass needs goes through saved-tensor hooks (here: kept on the host) and checkpoint(): same gradients, and
    the activations are among it.  A hook that gives back something else is refused."""
    from torch.autograd.graph import saved_tensors_hooks
    from torch.utils.checkpoint import checkpoint
    model, blocks, g = _small_network(0.5)
    weight = torch.randn(233, 10, generator=g, device="cuda")
    seen = []

    def pack(t):
        seen.append(t.numel())
        return t.cpu()

    def run(forward):
        torch.manual_seed(3)
        model.zero_grad(set_to_none=True)
        out = forward()
        out.backward(weight)
        return [out.detach()] + [p.grad.clone() for p in model.parameters()]

    def hooked(unpack):
        with saved_tensors_hooks(pack, unpack):
            return model(blocks)
    want = run(lambda: model(blocks))
    rows = blocks[0]["dst_nodes"].numel()
    for got in (run(lambda: hooked(lambda t: t.cuda())), run(lambda: checkpoint(model, blocks, use_reentrant=False))):
        for a, b in zip(want, got):
            assert torch.allclose(a, b, rtol=1e-4, atol=1e-5)
    assert sum(n >= rows * 64 for n in seen) >= 5  # both inputs of the first two layers, what the first ReLU gave
    for bad in (lambda t: t, lambda t: t.cuda()[:1], lambda t: t.cuda().double()):
        with pytest.raises(RuntimeError):
            run(lambda: hooked(bad))


@pytest.mark.parametrize("forward,backward", [(torch.bfloat16, None), (None, torch.bfloat16)])
def test_products_have_the_type_in_force_when_they_run(capi, forward, backward):
    """Operand type of the forward products and of the backward products: each that of its own time, as with the layers on their
    own.  Bound: values that differ by some 1e-6 (sums in another order) round to different bf16 numbers, 2^-8 apart, once in
    1e-6 / 2^-8 times, so operands and results are off by 2^-8 sqrt(2.6e-4) = 6e-5 each, about 1e-4 together; 5e-4 is asked, and
    products of the other type would be off by 4.6e-3."""
    from f2cgt_b200 import sage
    model, blocks, g = _small_network(0.0)
    weight = torch.randn(233, 10, generator=g, device="cuda")
    got = []
    for one_node in (True, False):
        if not one_node:
            model.layers[1].register_forward_pre_hook(lambda *_: None)
        model.zero_grad(set_to_none=True)
        with sage.products_in(forward):
            out = model(blocks)
        with sage.products_in(backward):
            out.backward(weight)
        got.append([p.grad for p in model.parameters()])
    for a, b in zip(*got):
        assert float((a - b).norm() / b.norm()) < 5e-4


@pytest.mark.parametrize("rows,n", [(40, 8191), (40, 8192), (37, 8193), (9, 16_388), (3, 30_000)])
def test_relu_dropout_gradient_of_wide_rows(capi, rows, n):
    from f2cgt_b200 import ops
    from f2cgt_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(n)
    grad, h = torch.randn(rows, n, generator=g, device="cuda"), torch.randn(rows, n, generator=g, device="cuda")
    keep = torch.rand(rows, n, generator=g, device="cuda") < 0.5
    dy, db = torch.empty_like(grad), torch.zeros(n, device="cuda")
    active, h = h, h * keep * 2.0
    check(lib.f2c_sage_mask_dropout(grad.data_ptr(), h.data_ptr(), active.data_ptr(), keep.data_ptr(), 2.0, dy.data_ptr(), db.data_ptr(), rows, n,
                                    ops._stream(h)))
    want = torch.where(active > 0, grad * keep * 2.0, 0.0)
    assert torch.equal(dy, want) and torch.allclose(db.double(), want.double().sum(0), rtol=1e-5, atol=1e-5 * rows**0.5)


def _one_node_and_layers(model, blocks, weight):
    got = []
    for one_node in (True, False):
        if not one_node:
            model.layers[1].register_forward_pre_hook(lambda *_: None)  # a hook: layer by layer
        assert (model._plain_weights() is not None) == one_node
        model.zero_grad(set_to_none=True)
        out = model(blocks)
        out.backward(weight)
        got.append([out.detach()] + [p.grad for p in model.parameters()])
    return got


@pytest.mark.parametrize("classes,hidden", [(10_000, 64), (10, 9001)])
def test_network_of_many_columns(capi, classes, hidden):
    model, blocks, g = _small_network(0.0, classes=classes, hidden=hidden, layers=2)
    for a, b in zip(*_one_node_and_layers(model, blocks, torch.randn(233, classes, generator=g, device="cuda"))):
        assert float((a - b).norm()) <= 1e-4 * float(b.norm())


def test_network_of_many_layers(capi):
    from f2cgt_b200 import sage
    first, blocks, g = _small_network(0.0, layers=1)
    rows = blocks[0]["dst_nodes"].numel()
    around = torch.arange(rows, device="cuda")
    ring = dict(indptr=torch.arange(rows + 1, device="cuda"), indices_local=around.roll(1), dst_nodes=blocks[0]["dst_nodes"], n_edges=rows)
    torch.manual_seed(2)
    model = sage.SAGE(128, 16, 5, 20, 0.0, first.layers[0].sm).cuda()
    got = _one_node_and_layers(model, list(blocks) + [ring] * 19, torch.randn(rows, 5, generator=g, device="cuda"))
    for a, b in zip(*got):
        assert float((a - b).norm()) <= 1e-4 * float(b.norm())


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_weights_that_are_views_of_a_flat_buffer(capi, shift):
    """Parameters that start anywhere in one buffer: same outputs (to tf32's 10 bits, sums in another order) and gradients."""
    model, blocks, g = _small_network(0.0)
    weight = torch.randn(233, 10, generator=g, device="cuda")
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = True
    try:
        got = []
        for flat in (False, True):
            if flat:
                buffer, at = torch.empty(sum(p.numel() + 3 for p in model.parameters()) + 4, device="cuda"), shift
                for p in model.parameters():
                    part = buffer[at:at + p.numel()].view_as(p)
                    part.copy_(p.data)
                    p.data = part
                    at += p.numel() + 3
            model.zero_grad(set_to_none=True)
            out = model(blocks)
            out.backward(weight)
            got.append([out.detach()] + [p.grad for p in model.parameters()])
        for a, b in zip(*got):
            assert float((a - b).norm() / b.norm()) < 5e-3
    finally:
        torch.backends.cuda.matmul.allow_tf32 = before


@pytest.mark.parametrize("k,ms,ns", [(32, (2, 3, 128, 1024, 61_440), (4, 47, 256)), (64, (2, 128, 3072, 16_384), (10, 64, 172)), (128, (2, 640, 8192, 61_440), (4, 47, 128, 172)),
                                     (256, (17, 2048, 40_960), (10, 128, 256, 300)), (104, (16_384, 28_672), (5, 64, 128)), (200, (16_384, 53_248), (47, 128, 256)),
                                     (36, (32_768, 65_536), (64, 68, 128)), (100, (32_768, 40_960, 102_400), (64, 100, 128, 256)), (300, (32_768, 49_152), (64, 172))])
def test_layer_product_equals_the_library_products_bit_for_bit(capi, k, ms, ns):
    """Where a training network takes the library's own product it must not change a bit of what torch's two products give
    (use_own() in native/sage.cpp)."""
    from f2cgt_b200 import ops
    from f2cgt_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(k)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = True
    try:
        for m in ms:
            for n in ns:
                x1, x2, w1, w2, b = rnd(m, k), rnd(m, k), rnd(n, k), rnd(n, k), rnd(n)
                y = torch.empty((m, n), device="cuda")
                check(lib.f2c_sage_forward(x1.data_ptr(), x2.data_ptr(), w1.data_ptr(), w2.data_ptr(), b.data_ptr(), y.data_ptr(), m, n, k, 0, ops._stream(x1)))
                assert torch.equal(y, torch.addmm(b, x1, w1.t()).addmm_(x2, w2.t())), (m, n, k)
    finally:
        torch.backends.cuda.matmul.allow_tf32 = before


@pytest.mark.parametrize("classes", [1, 2, 47])
def test_outputs_of_the_network_equal_the_layers_bit_for_bit(capi, classes):
    """tf32 products allowed, with gradients: the one-node network gives the layers' outputs.  One output column: fp32 in both."""
    before = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = True
    try:
        model, blocks, g = _small_network(0.0, classes=classes, hidden=128)
        got = _one_node_and_layers(model, blocks, torch.randn(233, classes, generator=g, device="cuda"))
        assert torch.equal(got[0][0], got[1][0])
        with torch.no_grad():
            for layer in model.layers:
                layer._forward_pre_hooks.clear()
            assert model._plain_weights() is not None and torch.equal(model(blocks), got[0][0])
    finally:
        torch.backends.cuda.matmul.allow_tf32 = before


def test_hooks_of_all_modules_see_the_dropout_layers(capi):
    model, blocks, _ = _small_network(0.5)
    torch.manual_seed(3)
    want, seen = model(blocks), []
    handle = torch.nn.modules.module.register_module_forward_hook(lambda module, *_: seen.append(type(module).__name__))
    try:
        torch.manual_seed(3)
        got = model(blocks)
    finally:
        handle.remove()
    assert seen.count("Dropout") == 2 and torch.allclose(got, want, rtol=1e-4, atol=1e-4)


def test_forward_mode_derivatives_are_refused_not_left_out(capi):
    import torch.autograd.forward_ad as fwd
    model, blocks, _ = _small_network(0.0)
    with fwd.dual_level():
        weights = {name: fwd.make_dual(p.detach(), torch.ones_like(p)) for name, p in model.named_parameters()}
        with pytest.raises((RuntimeError, NotImplementedError)):
            torch.func.functional_call(model, weights, (blocks,))


def test_dropout_in_place_draws_its_own_masks(capi):
    """nn.Dropout(inplace=True) draws from the generator as torch's in-place dropout does, with or without hooks on a layer."""
    model, blocks, _ = _small_network(0.5)
    model.dropout.inplace = True
    got = []
    for _ in range(2):
        torch.manual_seed(3)
        with torch.no_grad():
            got.append(model(blocks))
        model.layers[1].register_forward_pre_hook(lambda *_: None)
    assert torch.allclose(got[0], got[1], rtol=1e-4, atol=1e-4)


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_network_on_another_device_than_its_blocks_is_refused(capi):
    model, blocks, _ = _small_network(0.0)
    model.layers[1].to("cuda:1")
    with pytest.raises(RuntimeError, match="same device"):
        model(blocks)
