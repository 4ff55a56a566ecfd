"""The register-tiled forward pass at the edges of its tiles (64 and 128 samples), of the
choice between them and on rows that are not 16-byte aligned, against fp64 numpy."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo
from warpvbd_b200 import warmstart as ws

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 130, 148 * 256 - 1, 148 * 256, 148 * 256 + 129])
@pytest.mark.parametrize("offset", [0, 1])
def test_forward_tiles(n, offset):
    import torch
    p = ws.init_params(1)
    tr = ws.MLPTrainer(p, max_batch=64)
    g = torch.Generator(device="cuda").manual_seed(n)
    flat = torch.randn(n * ws.FEAT_WIDTH + offset, device="cuda", generator=g)
    X = flat[offset:].view(n, ws.FEAT_WIDTH)
    out = tr.forward(X).cpu().numpy()
    ref = mo.forward(p.astype(np.float64), X[:, :ws.N_IN].cpu().numpy().astype(np.float64))
    ref = ref[0] if isinstance(ref, tuple) else ref
    # three layers of at most 64 fp32 roundings (2^-24 each) of values of the result's size
    assert np.abs(out - ref).max() < 3 * 64 * 2.0 ** -24 * max(1.0, np.abs(ref).max())


def test_forward_from_several_threads():
    """First calls of both tile sizes at once, a thread and a stream each."""
    import threading
    import torch
    p = ws.init_params(2)
    g = torch.Generator(device="cuda").manual_seed(3)
    X = [torch.randn(148 * 256 + 64 if k % 2 else 1000, ws.FEAT_WIDTH, device="cuda", generator=g)
         for k in range(8)]
    torch.cuda.synchronize()
    out = [None] * 8

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            out[k] = ws.MLPTrainer(p, max_batch=64).forward(X[k])  # its stream: this one
            torch.cuda.current_stream().synchronize()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(8):
        assert torch.equal(out[k], ws.MLPTrainer(p, max_batch=64).forward(X[k]))


def test_training_step_under_capture():
    """Gradient and Adam update captured in a graph and replayed: the bits of the eager calls
    (the reduction and the update are launched before the kernel ahead of them has ended)."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(5)
    X = torch.randn(1000, ws.FEAT_WIDTH, device="cuda", generator=g)
    Y = torch.randn(1000, ws.N_OUT, device="cuda", generator=g)
    idx = torch.randperm(1000, device="cuda", generator=g).to(torch.int32)
    p = ws.init_params(4)
    ref = ws.MLPTrainer(p, max_batch=1024)
    grad, loss = ref.gradient(X, Y, idx)
    grad, loss = grad.clone(), loss.clone()
    ref.step(2e-3)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        tr = ws.MLPTrainer(p, max_batch=1024)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = tr.gradient(X, Y, idx)
        tr.step(2e-3)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out[0], grad) and torch.equal(out[1], loss)
    assert torch.equal(tr.P, ref.P)
