"""GPU: kernels are launched so that they may start while the previous kernel of the stream still runs; none may read its inputs
before that one is through.  Each call follows a kernel that clears half a gigabyte and, last of all, one of the call's inputs."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def calls(capi):
    from f2cgt_b200 import compress, ops
    from f2cgt_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(0)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    ints = lambda hi, dt, *s: torch.randint(0, hi, s, generator=g, device="cuda", dtype=dt)  # noqa: E731
    n_src, n_dst = 3000, 2000
    ip = torch.arange(0, 12 * n_dst + 1, 12, device="cuda")
    ix = ints(n_src, torch.int64, 12 * n_dst)
    cb = lambda n: torch.tensor([[1e-3, 4.0, -9.97, 2.0, 0.8]], device="cuda").repeat(n, 1).contiguous()  # noqa: E731
    out = []
    for D, bits, kinds in ((128, 1, ("stream", "prefetch", "prefetch_arith", "auto")), (128, 2, ("stream", "prefetch", "auto")), (128, 4, ("stream", "prefetch")),
                           (128, 8, ("prefetch", "prefetch_arith", "general", "auto")), (128, 16, ("auto",)), (101, 8, ("auto",)), (77, 2, ("auto",))):
        width = (D * bits + 7) // 8
        codes = ints(255, torch.uint8, n_src, width).view(torch.int8) if bits < 16 else ints(30000, torch.int16, n_src, D)
        for k in kinds:
            out.append((f"sq{bits} {D} {k}", [codes, cb(1), ip, ix],
                        lambda a, b, c, d, bits=bits, D=D, k=k: capi.sq_decompress_spmm_csr(a, b, c, d, bits, (D + 7) // 8 * 8, D, kernel=k)))
        for rows in (3000, 300):
            if rows == 300:
                codes = codes[:300].contiguous()
                big = codes.repeat(20, 1)
                out.append((f"decode sq{bits} {D} long", [big, cb(1)], lambda a, b, bits=bits, D=D: capi.sq_decompress(a, b, bits, (D + 7) // 8 * 8, D)))
            out.append((f"decode sq{bits} {D} {rows}", [codes, cb(1)], lambda a, b, bits=bits, D=D: capi.sq_decompress(a, b, bits, (D + 7) // 8 * 8, D)))
    hot, slot = ints(255, torch.uint8, 200, 128).view(torch.int8), (torch.arange(n_src, device="cuda", dtype=torch.int32) % 15 - 1).clamp_max(13)
    for n_cb, cs, K, D, kinds in ((4, 32, 256, 128, ("stream", "prefetch", "general")), (16, 8, 256, 128, ("prefetch",)), (7, 16, 256, 110, ("auto",)), (8, 16, 1024, 128, ("auto",))):
        codes = ints(K, torch.uint8 if K <= 256 else torch.int16, n_src, n_cb)
        books = rnd(n_cb, K, cs)
        for k in kinds:
            out.append((f"vq {n_cb} {cs} {k}", [codes, books, ip, ix], lambda a, b, c, d, D=D, k=k: capi.vq_decompress_spmm_csr(a, b, c, d, D, kernel=k)))
            if K == 256 and D == 128:
                out.append((f"two {n_cb} {cs} {k}", [hot, cb(1), codes, books, slot, ip, ix],
                            lambda a, b, c, d, e, f, h, k=k: capi.two_level_decompress_spmm_csr(a, b, 8, 128, c, d, e, f, h, 128, kernel=k)))
        out.append((f"decode vq {n_cb} {cs}", [codes, books], lambda a, b, D=D: capi.vq_decompress(a, b, D)))
        if K == 256:
            out.append((f"fusion {n_cb} {cs}", [hot[:, :D].contiguous(), cb(1), codes, books],
                        lambda a, b, c, d, D=D: capi.fusion_decompress(a, b, 8, 128, c, d, D)))
    for dt in (torch.float32, torch.float16):
        out.append((f"spmm {dt}", [rnd(n_src, 100).to(dt), ip, ix], lambda a, b, c: capi.spmm_csr(a, b, c)))
    out.append(("spmm backward", [rnd(n_dst, 64).round(), ip, ix], lambda a, b, c: ops.spmm_csr_backward(a, b, c, n_src, reduce="sum")))
    for d in (4, 8, 64, 200):
        out.append((f"kmeans {d}", [rnd(5000, d), rnd(256, d)], lambda a, b: capi.kmeans_assign(a, b, "l2")))
    out.append(("distance", [rnd(500, 16), rnd(40, 16)], lambda a, b: capi.pairwise_distance(a, b, "cosine")))
    out.append(("compress", [rnd(2000, 64), cb(1)], lambda a, b: capi.sq_compress(a, b, 4, 64)))
    for D in (64, 63):
        out.append((f"sq features {D}", [rnd(30000, D)], lambda a: list(compress.sq_compress_features(a, 4, 64, sample_size=1 << 30))))
    out.append(("pack", [ints(4, torch.uint8, 500, 64)], lambda a: capi.packbits(a, 2)))
    out.append(("unpack", [ints(255, torch.uint8, 500, 64)], lambda a: capi.unpackbits(a, 2, 256)))
    out.append(("dropout", [rnd(5000, 64)], lambda a: ops.dropout_inplace(a.view(-1)[:], 0.5, True, seed=1).clone()))

    def layer(x1, x2, w1, w2, b):
        y = torch.empty(700, 96, device="cuda")
        check(lib.f2c_sage_forward(x1.data_ptr(), x2.data_ptr(), w1.data_ptr(), w2.data_ptr(), b.data_ptr(), y.data_ptr(), 700, 96, 64, 0, ops._stream(y)))
        return y

    def mask(grad, h):
        dy = torch.empty_like(grad)
        check(lib.f2c_sage_mask(grad.data_ptr(), h.data_ptr(), 2.0, dy.data_ptr(), 0, 700, 96, ops._stream(dy)))
        return dy
    out.append(("layer", [rnd(700, 64), rnd(700, 64), rnd(96, 64), rnd(96, 64), rnd(96)], layer))
    out.append(("mask", [rnd(700, 96), rnd(700, 96)], mask))
    return out


def test_no_kernel_reads_before_the_previous_one_is_through(capi):
    from f2cgt_b200 import ops
    from f2cgt_b200._lib import check, lib
    dummy = torch.ones(1 << 27, device="cuda")

    def clear(t):
        at = (ctypes.c_void_p * 2)(dummy.data_ptr(), t.data_ptr())
        size = (ctypes.c_int64 * 2)(dummy.numel() * 4, t.numel() * t.element_size() // 4 * 4)
        check(lib.f2c_zero_ranges(at, size, 2, ops._stream(t)))

    def values(out):
        return [t.clone() for t in (out if isinstance(out, list) else [out])]

    for name, inputs, call in calls(capi):
        inputs = [t.clone() for t in inputs]
        for i in range(len(inputs)):
            kept = inputs[i].clone()
            for _ in range(2):  # the first call loads the kernel
                inputs[i].copy_(kept)
                torch.cuda.synchronize()
                clear(inputs[i])
                got = values(call(*inputs))
                torch.cuda.synchronize()
            inputs[i].copy_(kept)
            torch.cuda.synchronize()
            clear(inputs[i])
            torch.cuda.synchronize()
            want = values(call(*inputs))
            for a, b in zip(got, want):
                assert np.array_equal(a.cpu().numpy(), b.cpu().numpy(), equal_nan=a.is_floating_point()), (name, i)
            inputs[i].copy_(kept)


def clear_late(dummy, t):
    """Queue one kernel that clears dummy and, last of all, t."""
    from f2cgt_b200 import ops
    from f2cgt_b200._lib import check, lib
    at = (ctypes.c_void_p * 2)(dummy.data_ptr(), t.data_ptr())
    size = (ctypes.c_int64 * 2)(dummy.numel() * 4, t.numel() * t.element_size() // 4 * 4)
    check(lib.f2c_zero_ranges(at, size, 2, ops._stream(t)))


@pytest.mark.parametrize("n,d,k", [(5000, 8, 256), (3000, 64, 100), (2000, 32, 17)])
def test_an_iteration_of_a_fit_reads_nothing_early(capi, n, d, k):
    """Assignment, exact re-score (which stages the centres before the assignment is through) and sums, right behind the kernel that
    writes the centres or the points: no copy or memset stands in between, as between the iterations of a fit."""
    from f2cgt_b200 import ops
    from f2cgt_b200._lib import check, lib
    g = torch.Generator(device="cuda").manual_seed(n)
    x0, c0 = torch.randn(n, d, generator=g, device="cuda"), torch.randn(k, d, generator=g, device="cuda")
    x, c = x0.clone(), c0.clone()
    ws = torch.empty(lib.f2c_kmeans_fit_workspace(n, k, d), dtype=torch.uint8, device="cuda")
    dummy = torch.ones(1 << 27, device="cuda")
    for cleared in (c, x):
        got = []
        for apart in (False, False, True):  # the first call loads the kernels
            x.copy_(x0)
            c.copy_(c0)
            check(lib.f2c_kmeans_fit_begin(x.data_ptr(), n, k, d, ws.data_ptr(), ops._stream(x)))
            torch.cuda.synchronize()
            clear_late(dummy, cleared[:len(cleared) // 2])
            if apart:
                torch.cuda.synchronize()
            check(lib.f2c_kmeans_fit_iterate(x.data_ptr(), c.data_ptr(), n, k, d, 0, 0.0, 2, ws.data_ptr(), ops._stream(x)))
            got.append(c.clone())
            torch.cuda.synchronize()
        assert torch.equal(got[1], got[2])
