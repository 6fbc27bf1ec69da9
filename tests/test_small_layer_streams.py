"""The one-launch backward of small layers clears dx itself, by counters that belong to the stream: several streams, captured graphs, and a
wait that runs out."""
import numpy as np
import pytest

import test_gpu_parity as parity
from oracle import port

pytestmark = pytest.mark.gpu

I, O, F = 300, 40, 600                               # dx is 22 slices to clear


class Layer:
    """A layer, its gradients by the oracle, and calls that start from a dx that holds something."""

    def __init__(self, seed, binary):
        import torch
        from binarybrain_b200 import ops
        from gpu_util import dev, dev_fp32, wiring
        rng = np.random.default_rng(seed)
        idx, W = wiring(rng, I, O), np.clip(rng.normal(0.5, 0.25, (O, 64)), 0, 1).astype(np.float32)
        x, dy = rng.random((I, F), dtype=np.float32), rng.standard_normal((O, F), dtype=np.float32)
        self.want = port.sl6_backward(x, dy, idx, W, I, binary=int(binary))
        self.ops, self.binary = ops, binary
        self.x, self.dy, self.idx, self.W = dev_fp32(x), dev_fp32(dy), dev(idx), dev(W)
        self.dx, self.dW = torch.empty_like(self.x), torch.empty_like(self.W)
        torch.cuda.synchronize()

    def poison(self):
        self.dx.fill_(1000.0)
        self.dW.zero_()

    def backward(self):
        self.ops.stochastic_lut6_backward(self.x, self.dy, self.idx, self.W, self.dW, I, F, dx=self.dx, binary=self.binary)

    def correct(self):
        from gpu_util import err, host_fp32
        return err(host_fp32(self.dx, F), self.want[0]) <= parity.TOL and err(self.dW.cpu().numpy(), self.want[1]) <= parity.TOL


def heap_block_of(word):
    """The one block that the device heap now has to give, filled with `word`; the next request of up to 512 bytes gets it."""
    import torch
    from binarybrain_b200 import abi
    L = abi.lib()
    torch.cuda.synchronize()
    L.bbcu_LocalHeap_GarbageCollect()
    p = L.bbcu_LocalHeap_Malloc(512)
    abi.call("bbcu_fp32_Vector_set", p, word, 128, None)
    torch.cuda.synchronize()
    L.bbcu_LocalHeap_Free(p)
    return p


@pytest.mark.parametrize("binary", [False, True])
def test_two_streams_at_once(binary):
    import torch
    layers, streams = [Layer(k, binary) for k in range(2)], [torch.cuda.Stream() for _ in range(2)]
    for _ in range(20):
        for l, s in zip(layers, streams):
            with torch.cuda.stream(s):
                l.poison()
                l.backward()
    torch.cuda.synchronize()
    assert all(l.correct() for l in layers)


@pytest.mark.parametrize("binary", [False, True])
def test_first_call_of_a_stream_is_captured(binary):
    import torch
    eager, captured = Layer(3, binary), Layer(4, binary)
    eager.backward()                                                      # (loads the kernel)
    stream, other, graph = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    heap_block_of(1.0)                                                    # counters made of this would say: everything is cleared already
    with torch.cuda.graph(graph, stream=stream):
        captured.backward()
    with torch.cuda.stream(stream):                                       # the stream's own calls, before any replay
        eager.poison()
        eager.backward()
    torch.cuda.synchronize()
    assert eager.correct()
    for _ in range(20):                                                   # replays on another stream, beside calls on the captured one
        with torch.cuda.stream(other):
            captured.poison()
            graph.replay()
        with torch.cuda.stream(stream):
            eager.poison()
            eager.backward()
    torch.cuda.synchronize()
    assert eager.correct() and captured.correct()


@pytest.mark.parametrize("binary", [False, True])
def test_a_wait_that_runs_out_shows_in_the_gradients(binary):
    """The stream's counters say that every slice has been taken by somebody, and none is ever reported cleared: each block gives up after its
    bounded wait, and the fault word and all that it adds to say so.  The next call is as if nothing had been."""
    import torch
    from binarybrain_b200 import abi
    layer, stream = Layer(5, binary), torch.cuda.Stream()
    assert abi.lib().bbcu_b200_device_fault() == 0
    counters = heap_block_of(0.0)
    with torch.cuda.stream(stream):
        layer.poison()
        layer.backward()                                                  # makes the stream's counters, of that block
    torch.cuda.synchronize()
    assert layer.correct()
    with torch.cuda.stream(stream):
        layer.poison()
        abi.call("bbcu_fp32_Vector_set", counters, 1.0, 1, stream.cuda_stream)      # (slices claimed: the bits of 1.0f)
        layer.backward()
    torch.cuda.synchronize()
    assert abi.lib().bbcu_b200_device_fault() == 1
    assert torch.isnan(layer.dW).all() and torch.isnan(layer.dx[layer.idx.unique().long(), :F]).all()
    with torch.cuda.stream(stream):
        layer.poison()
        layer.backward()
    torch.cuda.synchronize()
    assert layer.correct() and abi.lib().bbcu_b200_device_fault() == 0
