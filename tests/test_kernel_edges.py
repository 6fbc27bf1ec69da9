"""GPU kernels at the sizes where their tiling can go wrong (edges of tiles, remainders, smallest and largest of a range), against
the CPU oracle."""
import numpy as np
import pytest

import test_gpu_parity as parity
from oracle import port, pack_bits, unpack_bits

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


# a word per thread and, above 1024 x 148 words a round of 256-word tiles, the pipeline: one word, no whole quad of words, unaligned rows, nodes that fill no CTA
@pytest.mark.parametrize("n_in,n_out,frames,stride", [(6, 1, 1, 1), (9, 7, 129, 5), (300, 420, 200, 8), (64, 4736, 1024, 32), (64, 4737, 1024, 32), (64, 600, 8100, 256), (50, 37, 131073, 4100),
                                                      (50, 37, 131073, 4099)])
def test_binary_lut6_words_and_pipeline(ops, n_in, n_out, frames, stride):
    import torch
    from gpu_util import dev, wiring
    rng = np.random.default_rng(n_out)
    words = (frames + 31) // 32
    x = rng.integers(-2**31, 2**31, (n_in, stride), dtype=np.int64).astype(np.int32)
    idx, table = wiring(rng, n_in, n_out), rng.integers(-2**31, 2**31, (n_out, 2), dtype=np.int64).astype(np.int32)
    y = ops.binary_lut6_forward(dev(x), dev(idx), dev(table), frames, y=torch.zeros((n_out, stride), dtype=torch.int32, device="cuda"))
    want = port.binary_lut6_forward(x.view(np.uint32), idx, table, frames)
    live = np.full(words, 0xffffffff, np.uint32)
    live[-1] >>= words * 32 - frames
    assert ((y.cpu().numpy().view(np.uint32)[:, :words] ^ want[:, :words]) & live == 0).all()


# table bytes as immediates: one quad of words, a segment and a quad, whole tiles and a part of one; two tiles a node, the last run of one tile (2000 nodes)
@pytest.mark.parametrize("n_in,n_out,words,spare", [(6, 1, 1, 5), (9, 13, 260, 0), (64, 777, 1024, 3), (50, 37, 2051, 31), (300, 1501, 1300, 1), (300, 2000, 3 * 1024 - 2, 9)])
def test_binary_lut6_by_immediates(ops, n_in, n_out, words, spare):
    import torch
    from gpu_util import dev, wiring
    rng = np.random.default_rng(words)
    F, stride = words * 32 - spare, (words + 3) // 4 * 4 + 4
    x = rng.integers(-2**31, 2**31, (n_in, stride), dtype=np.int64).astype(np.int32)
    idx, table = wiring(rng, n_in, n_out), rng.integers(-2**31, 2**31, (n_out, 2), dtype=np.int64).astype(np.int32)
    table[0] = [0x03020100, 0x7f80feff]
    want = port.binary_lut6_forward(x.view(np.uint32), idx, table, F)
    live = np.full(words, 0xffffffff, np.uint32)
    live[-1] >>= spare
    for forced in (True, False):
        y = torch.full((n_out, stride), 0x5a5a5a5a, dtype=torch.int32, device="cuda")
        y = ops.binary_lut6_forward(dev(x), dev(idx), dev(table), F, y=y, lop3_immediate=forced).cpu().numpy().view(np.uint32)
        assert ((y[:, :words] ^ want[:, :words]) & live == 0).all()
        assert (y[:, (words + 3) // 4 * 4:] == 0x5a5a5a5a).all()


# more input rows than two tiles of a node at a time are for, and the most for which they are
@pytest.mark.parametrize("n_in,n_out,words,spare", [(7000, 2000, 3 * 1024 - 2, 9), (6001, 2000, 3 * 1024 - 2, 9)])
def test_binary_lut6_by_immediates_of_many_rows(ops, n_in, n_out, words, spare):
    test_binary_lut6_by_immediates(ops, n_in, n_out, words, spare)


# rows 2^30 words apart, beyond the 32-bit arithmetic of that kernel
def test_binary_lut6_by_immediates_of_far_rows(ops):
    import torch
    from gpu_util import dev
    rng = np.random.default_rng(5)
    F, stride, words = 250, 1 << 30, 8
    x, table = rng.integers(-2**31, 2**31, (2, words)).astype(np.int32), rng.integers(-2**31, 2**31, (2, 2)).astype(np.int32)
    idx = np.array([[0, 1, 0, 0, 1, 1], [1, 1, 0, 1, 0, 0]], np.int32)
    xd, yd = torch.empty(stride + words, dtype=torch.int32, device="cuda"), torch.empty(stride + words, dtype=torch.int32, device="cuda")
    for k in range(2):
        xd[k * stride: k * stride + words] = dev(x[k])
    from binarybrain_b200 import abi
    idx_d, table_d = dev(idx), dev(table)
    abi.call("bbcu_bit_BinaryLut6_Forward_Lop3Immediate", xd.data_ptr(), yd.data_ptr(), idx_d.data_ptr(), table_d.data_ptr(), 2, F, stride, None)
    torch.cuda.synchronize()
    y = np.stack([yd[k * stride: k * stride + words].cpu().numpy() for k in range(2)]).view(np.uint32)
    want = port.binary_lut6_forward(x.view(np.uint32), idx, table, F)
    live = np.full(words, 0xffffffff, np.uint32)
    live[-1] >>= words * 32 - F
    assert ((y ^ want[:, :words]) & live == 0).all()


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


# two-valued inputs.  One launch per direction (up to 2^21 node-frames and 4096 frames): one warp, whole warps, a ragged last one, eight
# warps and several rounds of them.  General kernels: many consumers per input row (shared between warps) and rows without any, rows
# that are not 16-byte aligned, tiles of 512 frames with every kind of remainder, several tiles per node.
@pytest.mark.parametrize("I,O,F,stride", [(6, 1, 1, None), (9, 5, 3, 4), (40, 64, 127, None), (33, 70, 128, None), (50, 31, 129, 131), (30, 40, 1153, None),
                                          (48, 33, 4096, None),
                                          (40, 64, 4100, None), (7, 48, 5000, None), (3000, 400, 5377, 5380), (20, 30, 4609, 4611), (500, 1100, 2113, None)])
def test_two_valued_layers_edges(ops, I, O, F, stride):
    import torch
    from gpu_util import dev, dev_bits, dev_fp32, err, host_bits, host_fp32, wiring
    rng = np.random.default_rng(I + O + F)
    idx = wiring(rng, I, O)
    W = np.clip(rng.normal(0.5, 0.25, (O, 64)), 0, 1).astype(np.float32)
    x, dy = rng.random((I, F), dtype=np.float32), rng.standard_normal((O, F), dtype=np.float32)
    rm, rv = rng.random(O, dtype=np.float32), rng.random(O, dtype=np.float32) + 0.5
    parity._dl6_fp32_check(ops, x, idx, W, dy, rm, rv, dict(binary=1, lut_binarize=0), stride)
    xb = pack_bits(x > 0.5)
    for src, bits in ((dev_fp32(x, stride), False), (dev_bits(xb, F), True)):
        dW = torch.zeros((O, 64), device="cuda")
        dx = ops.stochastic_lut6_backward(src, dev_fp32(dy, stride), dev(idx), dev(W), dW, I, F, binary=True)
        dx_w, dW_w = port.sl6_backward(x, dy, idx, W, I, binary=1)
        assert err(host_fp32(dx, F), dx_w) <= parity.TOL and err(dW.cpu().numpy(), dW_w) <= parity.TOL
        assert not dx[:, F:].any()                                                    # the padding of dx stays clear
    p = port.dl6_forward_train(xb, idx, W, rm, rv, frames=F)
    amp = max(1.0, 0.3 * float(p["rstd"].max()))
    y, mean, rstd = ops.differentiable_lut6_forward_training(dev_bits(xb, F), dev(idx), dev(W), dev(rm.copy()), dev(rv.copy()), F)
    bad = unpack_bits(host_bits(y, F), F) != unpack_bits(p["y_bits"], F)
    assert (np.abs(p["y_pre"][bad] - 0.5) < 1e-4 * amp).all() and err(mean.cpu().numpy(), p["mean"]) <= parity.TOL
    dy = np.where(parity._edges(p["y_pre"], amp), np.float32(0), dy).astype(np.float32)
    dx_w, dW_w = port.dl6_backward(xb, dy, idx, W, p["mean"], p["rstd"], I)
    dW = torch.zeros((O, 64), device="cuda")
    dx = ops.differentiable_lut6_backward(dev_bits(xb, F), dev_fp32(dy, stride), dev(idx), dev(W), dW, dev(p["mean"]), dev(p["rstd"]), I, F)
    assert err(host_fp32(dx, F), dx_w) <= parity.BN_GRAD_FACTOR * parity.TOL * amp and err(dW.cpu().numpy(), dW_w) <= parity.BN_GRAD_FACTOR * parity.TOL * amp


# above the one-launch range; the forward by node, and (rows that are not aligned) by way of packed rows
@pytest.mark.parametrize("I,O,F,stride", [(700, 1025, 2049, None), (70, 40, 4129, 4131), (60, 33, 70001, None), (1300, 513, 4200, None)])
def test_large_two_valued_layers_edges(ops, I, O, F, stride):
    test_two_valued_layers_edges(ops, I, O, F, stride)


# the gather's last tile of 512 and of 256 frames: half of its chunks have frames, one frame more, and all but one frame
@pytest.mark.parametrize("I,O,F,stride", [(300, 60, 4352, None), (300, 60, 4353, None), (300, 60, 4607, None), (200, 60, 4224, None), (200, 60, 4225, None)])
def test_last_tile_of_the_gather(ops, I, O, F, stride):
    test_two_valued_layers_edges(ops, I, O, F, stride)


# bit rows that start anywhere beside gradients on 16-byte boundaries, above the one-launch range: whole steps of 512 frames, a remainder and one frame more
@pytest.mark.parametrize("I,O,F", [(30, 600, 4608), (50, 700, 5121), (9, 40, 60001)])
def test_bit_rows_that_start_anywhere(ops, I, O, F):
    import torch
    from gpu_util import dev, dev_bits, dev_fp32, err, host_fp32, wiring
    rng = np.random.default_rng(F)
    idx = wiring(rng, I, O)
    W = np.clip(rng.normal(0.5, 0.25, (O, 64)), 0, 1).astype(np.float32)
    x, dy = (rng.random((I, F)) > 0.5).astype(np.float32), rng.standard_normal((O, F), dtype=np.float32)
    dx_w, dW_w = port.sl6_backward(x, dy, idx, W, I, binary=1)
    xb, words = pack_bits(x > 0.5), (F + 31) // 32
    for stride in (words // 4 * 4 + 5, words // 4 * 4 + 6):
        dW = torch.zeros((O, 64), device="cuda")
        dx = ops.stochastic_lut6_backward(dev_bits(xb, F, stride), dev_fp32(dy), dev(idx), dev(W), dW, I, F)
        assert err(host_fp32(dx, F), dx_w) <= parity.TOL and err(dW.cpu().numpy(), dW_w) <= parity.TOL


# They take the loop of the others with narrower loads, 1.03 times as long; without it they took 1.42 times as long.
def test_bit_rows_that_start_anywhere_keep_the_pipelined_loop(ops):
    import torch
    I, O, F = 316, 617, 49185
    g = torch.Generator(device="cuda").manual_seed(1)
    words = (F + 31) // 32
    rows = [torch.randint(-2**31, 2**31 - 1, (I, s), dtype=torch.int32, device="cuda", generator=g) for s in ((words + 7) // 8 * 8, words | 1)]
    dy, idx = torch.rand((O, ops.fp32_stride(F)), device="cuda", generator=g), torch.randint(0, I, (O, 6), dtype=torch.int32, device="cuda", generator=g)
    W, dW, dx = torch.rand((O, 64), device="cuda", generator=g), torch.zeros((O, 64), device="cuda"), torch.empty((I, dy.shape[1]), device="cuda")
    start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))

    def time(x):
        start.record()
        for _ in range(10):
            ops.stochastic_lut6_backward(x, dy, idx, W, dW, I, F, dx=dx)
        end.record()
        end.synchronize()
        return start.elapsed_time(end)

    times = [[time(x) for x in rows] for _ in range(10)][2:]
    aligned, anywhere = (min(t) for t in zip(*times))
    assert anywhere <= 1.2 * aligned


# probability mode, one launch per direction: one warp, ragged and whole warps, eight warps and several rounds, unaligned rows, the largest
@pytest.mark.parametrize("I,O,F,stride", [(6, 1, 1, None), (9, 5, 3, 4), (33, 70, 128, None), (50, 31, 129, 131), (30, 40, 1025, None), (12, 8, 4096, 4099),
                                          (700, 512, 4096, None)])
def test_small_probability_layers_edges(ops, I, O, F, stride):
    from gpu_util import wiring
    rng = np.random.default_rng(I + O + F)
    idx = wiring(rng, I, O)
    W = np.clip(rng.normal(0.5, 0.25, (O, 64)), 0, 1).astype(np.float32)
    x = (rng.random((I, F), dtype=np.float32) * 1.2 - 0.1).astype(np.float32)
    dy, dW0 = rng.standard_normal((O, F), dtype=np.float32), rng.random((O, 64), dtype=np.float32)
    y = port.sl6_forward(x, idx, W)
    dx, dW = port.sl6_backward(x, dy, idx, W, I, dW=dW0)
    parity._sl6_check(ops, x, idx, W, dy, dW0, {}, dict(y=y, dx=dx, dW=dW), stride)
    parity._dl6_fp32_check(ops, x, idx, W, dy, rng.random(O, dtype=np.float32), rng.random(O, dtype=np.float32) + 0.5, dict(binary=0, lut_binarize=0), stride)


# many nodes: CTAs of fewer warps than rounds of 128 frames, of whole and of ragged rounds, aligned rows and others
@pytest.mark.parametrize("I,O,F,stride", [(60, 1300, 701, None), (33, 3100, 259, 263)])
def test_small_layers_of_several_rounds(ops, I, O, F, stride):
    test_small_probability_layers_edges(ops, I, O, F, stride)
    test_two_valued_layers_edges(ops, I, O, F, stride)


# above the one-launch range: persistent kernels (tile remainders, a short last group of nodes, one and several chunks of the statistics), rows that are not aligned
@pytest.mark.parametrize("I,O,F,stride", [(6, 1, 4097, None), (33, 17, 4225, 4228), (33, 17, 4225, 4227), (700, 1025, 2049, None), (9, 5, 20011, None)])
def test_large_probability_layers_edges(ops, I, O, F, stride):
    test_small_probability_layers_edges(ops, I, O, F, stride)


# The reverse pass stands in one piece and in two, the forward pass that keeps its operands for one frame and for two: the same operations, whose results
# agree in every bit.  Two at once and one piece in the plain backward, one and two pieces behind batch norm (here the identity, which has no part in the
# gradients), one and one piece in the one-launch layers.  Every input feeds one node, so that a gradient is no sum.
@pytest.mark.parametrize("O,F", [(3, 4097), (40, 5000)])
def test_forms_of_the_forward_and_reverse_pass_agree(ops, O, F):
    import torch
    g = torch.Generator(device="cuda").manual_seed(O)
    I, stride, small = 6 * O, ops.fp32_stride(F), 4096
    x, dy = torch.rand((I, stride), device="cuda", generator=g) * 1.2 - 0.1, torch.randn((O, stride), device="cuda", generator=g)
    idx = torch.randperm(I, device="cuda", generator=g).to(torch.int32).reshape(O, 6)
    W = torch.rand((O, 64), device="cuda", generator=g) * 0.8 + 0.1                      # inside the band that the batch norm's clipping passes
    dW = [torch.zeros((O, 64), device="cuda") for _ in range(3)]
    plain = ops.stochastic_lut6_backward(x, dy, idx, W, dW[0], I, F)
    bn = ops.dl6_backward_apply(x, dy, torch.empty_like(x), idx, W, dW[1], torch.zeros(O, device="cuda"), torch.ones(O, device="cuda"),
                                torch.zeros((O, 2), dtype=torch.float64, device="cuda"), I, F, F, gamma=1.0, beta=0.0, binary=False)
    one = ops.stochastic_lut6_backward(x[:, :small].contiguous(), dy[:, :small].contiguous(), idx, W, dW[2], I, small)
    assert plain[:, :F].any() and torch.equal(plain[:, :F], bn[:, :F]) and torch.equal(plain[:, :small], one)
    # sums of the same products in another order: F roundings of the sum of their magnitudes, which is no more than that of |dy|, each to 2^-24
    bound = F * 2.0**-24 * dy[:, :F].abs().sum(1, keepdim=True)
    assert ((dW[0] - dW[1]).abs() <= bound).all()


# one CTA (up to 2^14 target values) and the general form; Adam with the gradients cleared on the way, whole quads and a remainder
@pytest.mark.parametrize("classes,frames", [(1, 1), (10, 129), (10, 3276), (10, 3277), (3, 20000)])
def test_mean_loss_and_adam_update(ops, classes, frames):
    import torch
    from gpu_util import dev, dev_fp32, host_fp32
    rng = np.random.default_rng(frames)
    y = rng.random((classes, frames), dtype=np.float32)
    t = np.zeros_like(y)
    t[rng.integers(0, classes, frames), np.arange(frames)] = 1.0
    dy, loss = ops.softmax_cross_entropy(dev_fp32(y), dev_fp32(t), frames)
    dy_w, loss_w = port.softmax_cross_entropy(y, t)
    assert np.abs(host_fp32(dy, frames) - dy_w).max() <= 1e-6 and abs(float(loss.item()) - loss_w) <= 1e-5
    for n in (frames, frames + 1):
        W, dW = rng.random(n, dtype=np.float32), rng.standard_normal(n).astype(np.float32)
        Wd, dWd = dev(W.copy()), dev(dW.copy())
        ops.Adam([Wd], [dWd]).update()
        port.adam_update(W, dW, np.zeros_like(W), np.zeros_like(W), np.ones(2, np.float32))
        assert np.abs(Wd.cpu().numpy() - W).max() <= 1e-6 and not dWd.any()


# a frame per thread (up to 16 classes and 1024 frames): one class, all sixteen and one more, whole and ragged warps, one block's frames and one more;
# frames with one target above 0, several and none
@pytest.mark.parametrize("classes,frames", [(1, 33), (2, 1), (16, 1024), (16, 1025), (17, 64), (10, 100)])
def test_mean_loss_of_weighted_targets(ops, classes, frames):
    from gpu_util import dev_fp32, host_fp32
    rng = np.random.default_rng(classes * frames)
    y = (rng.standard_normal((classes, frames)) * 4).astype(np.float32)
    t = (rng.random((classes, frames)) * (rng.random((classes, frames)) < 1.5 / classes)).astype(np.float32)
    t[0, 0] = 0.75
    dy, loss = ops.softmax_cross_entropy(dev_fp32(y), dev_fp32(t), frames)
    dy_w, loss_w = port.softmax_cross_entropy(y, t)
    # both sides form a frame's loss in fp32, each to 8 ulp of it (exponentials, their sum, the quotient, its logarithm, the weight): 16 * 2^-24 of the sum
    assert np.abs(host_fp32(dy, frames) - dy_w).max() <= 1e-6 and abs(float(loss.item()) - loss_w) <= 16 * 2**-24 * max(1.0, abs(loss_w))


# the kernels for up to 4, 8 and 16 classes: the most and the fewest of each
@pytest.mark.parametrize("classes,frames", [(4, 1024), (5, 1000), (8, 65), (9, 1024)])
def test_mean_loss_of_few_classes(ops, classes, frames):
    test_mean_loss_of_weighted_targets(ops, classes, frames)


# Im2Col by quads of pixels (filters 3 and 5 wide, one band and several, a short last band, every border) and bit Im2Col with several word columns
# a block, several periods a warp, split blocks, windows beyond four and words without any
@pytest.mark.parametrize("c,h,w,fh,fw,ys,xs,pad,F", [
    (2, 5, 8, 3, 3, 1, 1, "same", 33), (3, 19, 12, 5, 5, 1, 1, "same", 70), (2, 9, 36, 3, 3, 1, 1, "valid", 31), (1, 20, 64, 3, 5, 1, 1, "same", 100),
    (64, 8, 8, 3, 3, 1, 1, "same", 600), (40, 6, 8, 3, 3, 1, 1, "same", 300), (1, 4, 4, 1, 1, 1, 1, "same", 65), (5, 3, 7, 5, 4, 2, 1, "same", 290)])
def test_im2col_quads_and_bit_columns(ops, c, h, w, fh, fw, ys, xs, pad, F):
    import test_conv_lowering as lowering
    lowering.test_im2col_bands_and_bit_words_against_oracle(c, h, w, fh, fw, ys, xs, pad, F)


# a layer of one launch and one of several (in probability mode: of the split operators); the second step's frames are other ones
@pytest.mark.parametrize("binary", [False, True])
@pytest.mark.parametrize("O,F", [(20, 300), (20, 4200)])
def test_layer_keeps_its_statistics_tensors(ops, O, F, binary):
    from binarybrain_b200.dist import ShardedDifferentiableLut6
    from gpu_util import dev, dev_fp32, wiring
    rng = np.random.default_rng(F)
    idx, W = wiring(rng, 30, O), np.clip(rng.normal(0.5, 0.25, (O, 64)), 0, 1).astype(np.float32)
    layer = ShardedDifferentiableLut6(dev(idx), dev(W), 30, sharded=False, binary=binary)
    mean, rstd = layer.mean, layer.rstd
    for _ in range(2):
        x = rng.random((30, F), dtype=np.float32)
        layer.forward(dev_fp32(x), F, F)
        want = port.dl6_forward_train(x, idx, W, np.zeros(O), np.ones(O), binary=int(binary))
        assert layer.mean is mean and layer.rstd is rstd
        assert np.abs(mean.cpu().numpy() - want["mean"]).max() <= 1e-6 and np.abs(rstd.cpu().numpy() / want["rstd"] - 1).max() <= 1e-4


# Training forward of a binary-mode layer on fp32 frames: the rows go through bits, or the frames through per-node passes, by a rule on the
# sizes.  Both sides of each of its lines; which way a call went shows in the scratch it asked the heap for.  The entry point that is not
# told the number of rows always takes the per-node passes, and the two ways agree in every bit.
@pytest.mark.parametrize("I,O,F,stride,packed", [
    (1, 2731, 3072, None, True), (1, 2730, 3072, None, False), (1, 2732, 3071, None, False), (4096, 2731, 3072, None, True), (4097, 2731, 3072, None, False),
    (12288, 12288, 4096, None, True), (24576, 12288, 4096, None, True), (24577, 12288, 4096, None, False), (12287, 12287, 4096, None, True),
    (24574, 12287, 4096, None, False), (49152, 49152, 1024, None, True), (49201, 49201, 1023, None, False), (140, 70, 30001, 30003, True)])
def test_binary_training_forward_by_bits_or_by_node(ops, I, O, F, stride, packed):
    import torch
    from binarybrain_b200 import abi
    L = abi.lib()
    g = torch.Generator(device="cuda").manual_seed(I + O)
    stride = ops.fp32_stride(F) if stride is None else stride
    x = torch.rand((I, stride), device="cuda", generator=g)
    idx = torch.randint(0, I, (O, 6), device="cuda", generator=g, dtype=torch.int32)
    W = torch.rand((O, 64), device="cuda", generator=g)

    def run(rows):
        y, s = torch.full((O, stride), -1.0, device="cuda"), [torch.ones(O, device="cuda") for _ in range(4)]
        torch.cuda.synchronize()
        L.bbcu_LocalHeap_GarbageCollect()
        before = L.bbcu_LocalHeap_GetAllocatedSize()
        args = [y.data_ptr(), idx.data_ptr(), W.data_ptr(), *[t.data_ptr() for t in s], 0.3, 0.5, 0.9, 0.25] + ([I] if rows else []) + [O, F, stride, 0, 1, None]
        abi.call("bbcu_fp32_DifferentiableLut6_ForwardTraining" + ("Rows" if rows else ""), x.data_ptr(), *args)
        torch.cuda.synchronize()
        return y[:, :F], s, L.bbcu_LocalHeap_GetAllocatedSize() - before

    def block(n):
        return (n + 511) // 512 * 512

    words, tables = (F + 127) // 128 * 4, 776 * O
    y, s, scratch = run(True)
    want = block((I + O) * words * 4) + block((tables + 255) // 256 * 256) if packed else block((tables + 255) // 256 * 256 + O * stride)
    assert scratch == want
    y2, s2, _ = run(False)
    if stride % 4 == 0:
        assert torch.equal(y, y2) and all(torch.equal(a, b) for a, b in zip(s, s2))
    else:                                                # per-frame kernel: sums of the values instead of counts of the patterns
        assert float((y != y2).float().mean()) < 1e-3 and all(torch.allclose(a, b, rtol=1e-4) for a, b in zip(s, s2))


# Two-valued inputs, uneven wiring: row 0 feeds every node and row 1 every other one, far more than the average (rows of several chunks of
# consumers, shared by blocks that add to dx), beside rows without any consumer.  One warp and several a block, tiles of 128 frames and more,
# rows that are not aligned.
@pytest.mark.parametrize("I,O,F,stride", [(2400, 150, 4200, None), (2400, 80, 4097, 4099), (60, 330, 4099, 4099), (60, 330, 4100, None), (9, 8, 4100, None)])
def test_two_valued_backward_uneven_wiring(ops, I, O, F, stride):
    import torch
    from gpu_util import dev, dev_bits, dev_fp32, err, host_fp32
    rng = np.random.default_rng(I + O + F)
    idx = np.stack([rng.permutation(np.arange(2, I))[:6] for _ in range(O)]).astype(np.int32)
    idx[:, 3] = 0
    idx[::2, 5] = 1
    W = np.clip(rng.normal(0.5, 0.25, (O, 64)), 0, 1).astype(np.float32)
    x, dy = rng.random((I, F), dtype=np.float32), rng.standard_normal((O, F), dtype=np.float32)
    xb = pack_bits(x > 0.5)
    dx_w, dW_w = port.sl6_backward(x, dy, idx, W, I, binary=1)
    p = port.dl6_forward_train(xb, idx, W, np.zeros(O), np.ones(O), frames=F)
    amp = max(1.0, 0.3 * float(p["rstd"].max()))
    dy_n = np.where(parity._edges(p["y_pre"], amp), np.float32(0), dy).astype(np.float32)
    dxn_w, dWn_w = port.dl6_backward(xb, dy_n, idx, W, p["mean"], p["rstd"], I)
    for src in (dev_fp32(x, stride), dev_bits(xb, F)):
        dW = torch.zeros((O, 64), device="cuda")
        dx = torch.full((I, ops.fp32_stride(F) if stride is None else stride), 7.0, device="cuda")
        ops.stochastic_lut6_backward(src, dev_fp32(dy, stride), dev(idx), dev(W), dW, I, F, dx=dx, binary=True)
        assert err(host_fp32(dx, F), dx_w) <= parity.TOL and err(dW.cpu().numpy(), dW_w) <= parity.TOL and not dx[:, F:].any()
        dW.zero_()
        dx.fill_(7.0)
        ops.differentiable_lut6_backward(src, dev_fp32(dy_n, stride), dev(idx), dev(W), dW, dev(p["mean"]), dev(p["rstd"]), I, F, dx=dx, binary=True)
        tol = parity.BN_GRAD_FACTOR * parity.TOL * amp
        assert err(host_fp32(dx, F), dxn_w) <= tol and err(dW.cpu().numpy(), dWn_w) <= tol and not dx[:, F:].any()


# the largest call of one CTA and the smallest of the general form
@pytest.mark.parametrize("classes,frames", [(4, 4096), (10, 1638), (10, 1639)])
def test_mean_loss_at_the_line(ops, classes, frames):
    test_mean_loss_and_adam_update(ops, classes, frames)


def test_mean_loss_without_scratch(ops):
    """A heap that has nothing left to give: the one block takes calls of the general form too."""
    import torch
    from binarybrain_b200 import abi
    torch.cuda.synchronize()
    abi.lib().bbcu_LocalHeap_GarbageCollect()
    others = abi.lib().bbcu_LocalHeap_GetAllocatedSize()                   # (what earlier tests in this process still hold)
    abi.lib().bbcu_LocalHeap_SetByteLimit(1)
    try:
        test_mean_loss_and_adam_update(ops, 10, 3277)
        assert abi.lib().bbcu_LocalHeap_GetAllocatedSize() == others
    finally:
        abi.lib().bbcu_LocalHeap_SetByteLimit(0)


# The apply half of a frame-sharded binary-mode backward uses what the statistics half left in the stream's scratch, unless something else has
# used or released that scratch in between, or the call is another one.
@pytest.mark.parametrize("between", ["nothing", "another layer", "garbage collection", "another gamma", "captured"])
def test_apply_half_after_the_scratch_was_used(ops, between):
    import torch
    from binarybrain_b200 import abi
    from gpu_util import dev, dev_fp32, wiring
    rng = np.random.default_rng(17)
    I, O, F = 40, 30, 700
    x, dy, idx = dev_fp32(rng.random((I, F))), dev_fp32(rng.standard_normal((O, F))), dev(wiring(rng, I, O))
    W = dev(np.clip(rng.normal(0.5, 0.25, (O, 64)), 0, 1).astype(np.float32))
    mean, rstd = torch.full((O,), 0.5, device="cuda"), torch.full((O,), 4.0, device="cuda")
    sums, dx, dW = torch.zeros((O, 2), dtype=torch.float64, device="cuda"), torch.empty_like(x), torch.zeros_like(W)
    gamma = 0.1 if between == "another gamma" else 0.3

    def apply(dx, dW):
        return ops.dl6_backward_apply(x, dy, dx, idx, W, dW, mean, rstd, sums, I, F, F, gamma=gamma)

    ops.dl6_backward_stats(x, dy, idx, W, mean, rstd, F, sums)
    abi.lib().bbcu_LocalHeap_GarbageCollect()                              # nothing of the statistics half is left
    want_dW = W.new_zeros(O, 64)
    want_dx = apply(torch.empty_like(x), want_dW)
    if between == "captured":
        side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            ops.dl6_backward_stats(x, dy, idx, W, mean, rstd, F, sums)
            apply(dx, dW)
            ops.dl6_backward_stats(x, dy, idx, W, mean, rstd, F, sums)     # outside of the graph: nothing that a replay could count on
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=side):
            apply(dx, dW)
        with torch.cuda.stream(side):
            ops.dl6_backward_stats(x, torch.zeros_like(dy), idx, W, mean, rstd, F, torch.zeros_like(sums))
            dx.fill_(7.0)
            dW.zero_()
            graph.replay()
        torch.cuda.synchronize()
    else:
        ops.dl6_backward_stats(x, dy, idx, W, mean, rstd, F, sums)
        if between == "another layer":
            ops.stochastic_lut6_forward(dev_fp32(rng.random((I, 40000))), dev(wiring(rng, I, 60)), torch.rand((60, 64), device="cuda"), 40000)
        if between == "garbage collection":
            abi.lib().bbcu_LocalHeap_GarbageCollect()
        apply(dx, dW)
    assert torch.allclose(dx, want_dx, rtol=1e-5, atol=1e-5) and torch.allclose(dW, want_dW, rtol=1e-5, atol=1e-4)
