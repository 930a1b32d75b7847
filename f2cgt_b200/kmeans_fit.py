"""Lloyd iterations for ``KMeans.fit`` (reference: RAFT ``kmeans::fit`` behind src/kmeans.cu:61-75, and
the torch loop around ``capi.pairwise_distance`` in examples/my_kmeans.py:73-113).

The iterations - assignment, the n*k*d contraction, and centre update - are the library's kernels; torch only does the
k-means++ / random initialisation.  Initial centres are random, so a fit
is comparable with the reference's by inertia only, never label by label.
"""
import torch

from . import ops
from ._lib import check, lib


def _init_random(x, k, gen):
    # examples/my_kmeans.py:27-31: k distinct non-zero rows
    nz = (x != 0).any(dim=1).nonzero().squeeze(1)
    if nz.numel() < k:
        raise RuntimeError(f"KMeans.fit: need at least {k} non-zero rows, have {nz.numel()}")
    pick = nz[torch.randperm(nz.numel(), generator=gen, device=x.device)[:k]]
    return x[pick].clone()


def _init_kmeanspp(x, k, gen):
    n = x.shape[0]
    centers = torch.empty((k, x.shape[1]), dtype=torch.float32, device=x.device)
    first = int(torch.randint(0, n, (1,), generator=gen, device=x.device).item())
    centers[0] = x[first]
    d2 = ops.pairwise_distance(x, centers[:1].contiguous(), "l2").squeeze(1)
    for c in range(1, k):
        probs = d2.clamp_min(0)
        if float(probs.sum()) <= 0:
            probs = torch.ones_like(probs)
        nxt = int(torch.multinomial(probs, 1, generator=gen).item())
        centers[c] = x[nxt]
        d2 = torch.minimum(d2, ops.pairwise_distance(x, centers[c:c + 1].contiguous(), "l2").squeeze(1))
    return centers


_AHEAD = 16  # iterations queued between two looks at the convergence flag (those behind the converged one do nothing)


def _iterate(x, centers, metric, max_iter, tol):
    """Lloyd iterations from ``centers`` (float32, replaced in place) until the summed squared shift is at most ``tol``.  The
    whole loop runs on the device (``f2c_kmeans_fit_iterate``); the host queues a few iterations ahead and reads one flag."""
    if x.dim() != 2 or centers.dim() != 2 or x.shape[1] != centers.shape[1]:
        raise RuntimeError("data must be [n, d] and centers [k, d]")
    n, d = x.shape
    k = centers.shape[0]
    seen = [(torch.empty(4, dtype=torch.int32, pin_memory=True), torch.cuda.Event()) for _ in range(2)]
    stream = torch.cuda.current_stream(x.device)
    queued = rounds = 0
    with ops._on(x):
        ws = torch.empty((lib.f2c_kmeans_fit_workspace(n, k, d),), dtype=torch.uint8, device=x.device)
        words = ws[:16].view(torch.int32)
        check(lib.f2c_kmeans_fit_begin(x.data_ptr(), n, k, d, ws.data_ptr(), stream.cuda_stream))
        while True:
            take = min(_AHEAD, max_iter - queued)
            if take > 0:
                check(lib.f2c_kmeans_fit_iterate(x.data_ptr(), centers.data_ptr(), n, k, d, ops._metric(metric), float(tol), take,
                                                 ws.data_ptr(), stream.cuda_stream))
                queued += take
            host, event = seen[rounds % 2]
            host.copy_(words, non_blocking=True)
            event.record(stream)
            rounds += 1
            if take > 0 and rounds == 1:
                continue  # look at a round's flag only when the next round is queued: the GPU never waits for the host
            host, event = seen[rounds % 2] if take > 0 else (host, event)
            event.synchronize()
            done, _, not_finite, _ = host.tolist()
            if done or take <= 0:
                return bool(not_finite)


def _inertia(x, labels, centers, metric):
    c = centers[labels]
    if metric == "cosine":
        return float((1 - torch.nn.functional.cosine_similarity(x, c, dim=1)).sum())
    return float(((x - c) ** 2).sum())


def lloyd_fit(x, k, metric, init, init_centers, max_iter, tol, n_init, seed=None):
    gen = torch.Generator(device=x.device)
    gen.manual_seed(torch.initial_seed() if seed is None else seed)
    best, best_inertia = None, float("inf")
    for _ in range(max(1, n_init if init != "array" else 1)):
        if init == "array":
            centers = init_centers.float().clone()
        elif init == "random":
            centers = _init_random(x, k, gen)
        else:
            centers = _init_kmeanspp(x, k, gen)
        centers = centers.contiguous()
        not_finite = x.shape[0] > 0 and max_iter > 0 and _iterate(x, centers, metric, max_iter, tol)
        if max(1, n_init) == 1 or init == "array":
            if not_finite or not bool(torch.isfinite(centers).all()):
                raise RuntimeError("KMeans.fit: the data or the centres are not finite")
            return centers
        inertia = float("nan") if not_finite else _inertia(x, ops.kmeans_assign(x, centers, metric), centers, metric)
        if inertia < best_inertia:
            best, best_inertia = centers, inertia
    return best
