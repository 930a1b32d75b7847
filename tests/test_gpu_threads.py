"""GPU: calls that wait for a place in the launch queue leave the interpreter to the other Python threads; first calls of a process
under capture."""
import os
import subprocess
import sys
import threading
import time

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _network():
    from f2cgt_b200 import sage, synth
    n = 5000
    indptr, indices = synth.power_law_graph(n, 12, 2.1, seed=1, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(5)
    codes = torch.randint(0, 256, (n, 4), generator=g, dtype=torch.uint8, device="cuda")
    cm = sage.CompressionManager(128, ["vq"], [(32, -1)], [torch.randn(4, 256, 32, generator=g, device="cuda")], [codes])
    model = sage.SAGE(128, 64, 10, 3, 0.0, cm).to("cuda").eval()
    _, _, blocks = next(iter(sage.GPUSamplingDataloader(indptr, indices, torch.arange(100, device="cuda"), 100, (4, 3, 2), shuffle=False)))
    return model, blocks


def _longest_pause_beside(call):
    """Longest time for which another Python thread stood still while call() ran, and the longest single call()."""
    stop, pauses = threading.Event(), [0.0]

    def watch():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            pauses[0] = max(pauses[0], now - last)
            last = now
    call()
    torch.cuda.synchronize()
    thread = threading.Thread(target=watch)
    thread.start()
    torch.cuda._sleep(800_000_000)  # about 0.4 s; the launches behind it fill the queue
    longest = 0.0
    for _ in range(1500):
        t0 = time.perf_counter()
        call()
        longest = max(longest, time.perf_counter() - t0)
    stop.set()
    thread.join()
    torch.cuda.synchronize()
    return pauses[0], longest


@pytest.mark.parametrize("which", ["decode", "sq", "vq", "two", "spmm", "kmeans", "network"])
def test_other_threads_run_while_the_launch_queue_is_full(capi, which):
    g = torch.Generator(device="cuda").manual_seed(0)
    codes = torch.randint(0, 255, (64, 4), generator=g, dtype=torch.uint8, device="cuda")
    books = torch.randn(4, 256, 32, generator=g, device="cuda")
    hot = torch.randint(0, 100, (64, 128), generator=g, dtype=torch.int8, device="cuda")
    cb = torch.tensor([[1e-3, 4.0, -9.97, 2.0, 0.8]], device="cuda")
    slot = torch.arange(64, device="cuda", dtype=torch.int32)
    ip = torch.arange(0, 65, device="cuda")
    ix = torch.arange(0, 64, device="cuda")
    h = torch.randn(64, 32, device="cuda")
    if which == "network":
        model, blocks = _network()

        def call():
            with torch.no_grad():
                model(blocks)
    else:
        call = dict(decode=lambda: capi.vq_decompress(codes, books, 128),
                    sq=lambda: capi.sq_decompress_spmm_csr(hot, cb, ip, ix, 8, 128, 128),
                    vq=lambda: capi.vq_decompress_spmm_csr(codes, books, ip, ix, 128),
                    two=lambda: capi.two_level_decompress_spmm_csr(hot, cb, 8, 128, codes, books, slot, ip, ix, 128),
                    spmm=lambda: capi.spmm_csr(h, ip, ix), kmeans=lambda: capi.kmeans_assign(h, h[:8].contiguous(), "l2"))[which]
    pause, longest = _longest_pause_beside(call)
    assert longest > 0.05, "the queue did not fill"
    assert pause < 0.5 * longest


CAPTURED = """
import torch
import F2CGTLib as capi
g = torch.Generator(device="cuda").manual_seed(0)
codes = torch.randint(-128, 128, (20000, 32), generator=g, device="cuda", dtype=torch.int8)
cb = torch.tensor([[1e-3, 4.0, -9.97, 2.0, 0.8]], device="cuda")
ip = torch.arange(0, 12 * 40000 + 1, 12, device="cuda")
ix = torch.randint(0, 20000, (12 * 40000,), generator=g, device="cuda")
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    out = capi.sq_decompress_spmm_csr(codes, cb, ip, ix, 2, 128, 128)
graph.replay()
assert torch.equal(out, capi.sq_decompress_spmm_csr(codes, cb, ip, ix, 2, 128, 128, kernel="general"))
from f2cgt_b200 import ops
assert ops.device_status() == 0
"""


def test_first_use_of_the_status_word_under_capture(capi):
    """The streamed kernel's status word and its host copy are set up by the first call, which here is part of a graph."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", CAPTURED], cwd=root, check=True, timeout=120)
