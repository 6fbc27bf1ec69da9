"""GPU kernels at the sizes where their tiling can go wrong (edges of tiles, remainders, smallest and largest of a range), against
the CPU oracle."""
import numpy as np
import pytest

from oracle import port

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from binarybrain_b200 import ops as o
    return o


# blocks of 2048 output frames (real -> binary), of 32 output frames and 8 x 32 input frames (binary -> real)
@pytest.mark.parametrize("nodes,frames,mod,depth,points", [(3, 1, 1, 1, 3), (4, 33, 7, 3, 2), (5, 293, 7, 1, 1), (2, 100, 41, 2, 2), (1, 2049, 1, 1, 1),
                                                           (2, 7, 300, 1, 2)])
def test_modulation_edges(ops, nodes, frames, mod, depth, points):
    from gpu_util import dev_fp32, dev_bits, host_bits, host_fp32
    rng = np.random.default_rng(nodes * 1000 + frames)
    x = rng.random((nodes, frames), dtype=np.float32)
    th = rng.random((nodes, frames * mod), dtype=np.float32)
    for t in (None, th):
        y = ops.real_to_binary(dev_fp32(x), frames, frame_mod=mod, depth_mod=depth, thresholds=None if t is None else dev_fp32(t), point_size=points)
        want = port.real_to_binary(x, mod, depth, thresholds=t, point_size=points)
        assert (host_bits(y, frames * mod) == want).all()
    rows = want.shape[0]
    got = ops.binary_to_real(dev_bits(want, frames * mod), rows, nodes, frames, frame_mux=mod)
    assert np.array_equal(host_fp32(got, frames), port.binary_to_real(want, nodes, frames, mod))
    dy = rng.random((nodes, frames), dtype=np.float32)
    dx = ops.binary_to_real_backward(dev_fp32(dy), rows, frames, frame_mux=mod)
    assert np.abs(host_fp32(dx, frames * mod) - port.binary_to_real_backward(dy, rows, mod)).max() <= 1e-7


# one chunk, a first and a last chunk only, full-width chunks with a one-word remainder
@pytest.mark.parametrize("n_in,n_out,words,spare", [(9, 7, 1, 0), (700, 400, 130, 30), (4096, 64, 257, 31), (1024, 1100, 1793, 5)])
def test_binary_lut6_host_chunks(ops, n_in, n_out, words, spare):
    import torch
    from gpu_util import wiring
    rng = np.random.default_rng(words)
    F = words * 32 - spare
    idx, table = wiring(rng, n_in, n_out), rng.integers(-2**31, 2**31, (n_out, 2)).astype(np.int32)
    x = rng.integers(0, 2**32, (n_in, ops.bit_stride(F)), dtype=np.uint64).astype(np.uint32)
    y = torch.zeros((n_out, x.shape[1]), dtype=torch.int32)
    ops.binary_lut6_forward_host(torch.from_numpy(x.view(np.int32)), torch.from_numpy(idx), torch.from_numpy(table), F, y=y)
    want = port.binary_lut6_forward(x, idx, table, F)
    live = np.full(words, 0xffffffff, np.uint32)
    live[-1] >>= spare
    assert ((y.numpy().view(np.uint32)[:, :words] ^ want[:, :words]) & live == 0).all()
