"""The bbcu_* operators on torch CUDA tensors.

torch only provides device memory and the current stream here; every operator is one call through
the C ABI (binarybrain_b200._native, which parses the tensors straight into the C signature and adds the current stream).
Frame buffers are 2-D tensors ``[nodes, frame_stride]``: fp32 buffers hold one float per frame, bit buffers (dtype int32) 32 frames
per element, LSB first -- the FrameBuffer layout of the reference (include/bb/FrameBuffer.h:28-46).  ``frames`` is the number
of valid frames; the stride is taken from the tensor.
"""
import torch

from . import abi

BIAS = 0.25   # unbinarize_bias of the reference's layers (include/bb/DifferentiableLutN.h:63)


def __getattr__(name):
    """SMALL_NODE_FRAMES, SMALL_FRAMES: a layer of at most this many node-frames and frames runs in one launch per direction when its
    operators are called unsplit.  The numbers are the library's (include/bbcu_b200.h), looked up once."""
    if name in ("SMALL_NODE_FRAMES", "SMALL_FRAMES"):
        from . import _native
        return globals().setdefault(name, getattr(_native, name))
    raise AttributeError(f"module {__name__!r} has no attribute {name!r}")


class _Native:
    """Stands for binarybrain_b200._native until the first operator is called: importing this module needs no built extension."""

    def __getattr__(self, name):
        global _n
        from . import _native
        _n = _native
        return getattr(_native, name)


_n = _Native()


def _chk(t, dtype, name):
    if not t.is_cuda:
        raise ValueError(f"{name}: expected a CUDA tensor (the bbcu_* operators have no CPU path)")
    if t.dtype != dtype:
        raise ValueError(f"{name}: expected dtype {dtype}, got {t.dtype}")
    if not t.is_contiguous():
        raise ValueError(f"{name}: expected a contiguous tensor")
    return t


def fp32_stride(frames):
    """Row stride in floats: rows padded to 32 bytes (include/bb/FrameBuffer.h:414-417)."""
    return (frames + 7) // 8 * 8


def bit_stride(frames):
    """Row stride in 32-bit words: rows padded to 256 bits."""
    return (frames + 255) // 256 * 8


def _bits(like, rows, frames, stride=None):
    """An output buffer for bit frames.  The operators write whole words up to the last frame; padding words, if there are any, are cleared."""
    words = (frames + 31) // 32
    stride = bit_stride(frames) if stride is None else stride
    return _n.empty_i32(like, rows, stride) if stride == words else torch.zeros((rows, stride), dtype=torch.int32, device=like.device)


# ------------------------------------------------------------------------------------------ StochasticLut6
def stochastic_lut6_forward(x, idx, W, frames, y=None, binary=False, lut_binarize=False, bias=BIAS, bit_output=False):
    """fp32 or bit-packed x -> fp32 y (clip to [0,1]) or, with bit_output (bit x only), bit-packed y = lut > 0.5."""
    O = idx.shape[0]
    _chk(idx, torch.int32, "idx"); _chk(W, torch.float32, "W")
    if x.dtype == torch.float32:
        _chk(x, torch.float32, "x")
        if y is None:
            y = _n.empty_f32(x, O, x.shape[1])
        _n.bbcu_fp32_StochasticLut6_Forward(x, y, idx, W, O, frames, x.shape[1], int(binary), int(lut_binarize), bias)
    elif bit_output:
        _chk(x, torch.int32, "x")
        if y is None:
            y = _bits(x, O, frames, x.shape[1])
        _n.bbcu_bit_bit_fp32_StochasticLut6_Forward(x, y, idx, W, O, frames, x.shape[1], int(lut_binarize), bias)
    else:
        _chk(x, torch.int32, "x")
        if y is None:
            y = _n.empty_f32(x, O, fp32_stride(frames))
        _n.bbcu_bit_fp32_StochasticLut6_Forward(x, y, idx, W, O, frames, y.shape[1], x.shape[1], int(lut_binarize), bias)
    return y


def stochastic_lut6_backward(x, dy, idx, W, dW, n_in, frames, dx=None, binary=False, lut_binarize=False, bias=BIAS, dx_tmp=None):
    """dx is overwritten, dW accumulated into.  dx_tmp: optional fp32 scratch [6 * nodes, tmp_stride] as the reference's callers pass it."""
    O = idx.shape[0]
    _chk(dy, torch.float32, "dy"); _chk(dW, torch.float32, "dW")
    if dx is None:
        dx = _n.empty_f32(dy, n_in, dy.shape[1])
    if x.dtype == torch.float32:
        assert x.shape[1] == dy.shape[1], "x, dy and dx share one frame stride"
        _n.bbcu_fp32_StochasticLut6_Backward(x, dy, dx, dx_tmp, idx, 0, W, dW, 0, n_in, O, frames, dy.shape[1],
                                             0 if dx_tmp is None else dx_tmp.shape[1], 0 if dx_tmp is None else dx_tmp.shape[1], int(binary),
                                             int(lut_binarize), bias)
    else:
        _chk(x, torch.int32, "x")
        _n.bbcu_bit_fp32_StochasticLut6_Backward(x, dy, dx, 0, idx, 0, W, dW, 0, n_in, O, frames, dy.shape[1], x.shape[1], 0, 0, int(lut_binarize),
                                                 bias)
    return dx


# ------------------------------------------------------------------------------------------ DifferentiableLut6
def differentiable_lut6_forward_training(x, idx, W, running_mean, running_var, frames, y=None, gamma=0.3, beta=0.5, momentum=0.9,
                                         bias=BIAS, lut_binarize=False, binary=True, mean=None, rstd=None):
    """Returns (y, mean, rstd), in `mean` and `rstd` where they are given; running_mean / running_var are updated in place.  Bit x gives bit y."""
    if x.dtype == torch.float32:
        return _n.train_forward(x, y, idx, W, mean, rstd, running_mean, running_var, gamma, beta, momentum, bias, frames, lut_binarize, binary)
    _chk(x, torch.int32, "x")
    O = idx.shape[0]
    mean = _n.vector_f32(x, O) if mean is None else mean
    rstd = _n.vector_f32(x, O) if rstd is None else rstd
    if y is None:
        y = _bits(x, O, frames, x.shape[1])
    _n.bbcu_bit_fp32_DifferentiableLut6_ForwardTraining(x, y, idx, W, mean, rstd, running_mean, running_var, gamma, beta, momentum, bias, O, frames,
                                                        x.shape[1], int(lut_binarize))
    return y, mean, rstd


def differentiable_lut6_forward_inference(x, idx, W, running_mean, running_var, frames, y=None, gamma=0.3, beta=0.5, bias=BIAS,
                                          lut_binarize=False, binary=True):
    O = idx.shape[0]
    if x.dtype == torch.float32:
        if y is None:
            y = _n.empty_f32(x, O, x.shape[1])
        _n.bbcu_fp32_DifferentiableLut6_ForwardInference(x, y, idx, W, running_mean, running_var, gamma, beta, bias, O, frames, x.shape[1],
                                                         int(lut_binarize), int(binary))
    else:
        if y is None:
            y = _bits(x, O, frames, x.shape[1])
        _n.bbcu_bit_fp32_DifferentiableLut6_ForwardInference(x, y, idx, W, running_mean, running_var, gamma, beta, bias, O, frames, x.shape[1],
                                                             int(lut_binarize))
    return y


def differentiable_lut6_backward(x, dy, idx, W, dW, mean, rstd, n_in, frames, dx=None, gamma=0.3, beta=0.5, bias=BIAS, lut_binarize=False,
                                 binary=True, dx_tmp=None):
    if dx_tmp is None and x.dtype == torch.float32:
        return _n.train_backward(x, dy, dx, idx, W, dW, mean, rstd, gamma, beta, bias, n_in, frames, lut_binarize, binary)
    O = idx.shape[0]
    if dx is None:
        dx = _n.empty_f32(dy, n_in, dy.shape[1])
    scratch = _n.vector_f32(dy, 2 * O)
    dmean = scratch.data_ptr()
    dvar = dmean + 4 * O
    if x.dtype == torch.float32:
        assert x.shape[1] == dy.shape[1]
        _n.bbcu_fp32_DifferentiableLut6_Backward(x, dy, dx, dx_tmp, idx, 0, W, dW, mean, rstd, dmean, dvar, gamma, beta, bias, 0, n_in, O, frames,
                                                 dy.shape[1], dx_tmp.shape[1], dx_tmp.shape[1], int(lut_binarize), int(binary))
    else:
        _n.bbcu_bit_fp32_DifferentiableLut6_Backward(x, dy, dx, 0, idx, 0, W, dW, mean, rstd, dmean, dvar, gamma, beta, bias, 0, n_in, O, frames,
                                                     dy.shape[1], x.shape[1], 0, 0, int(lut_binarize))
    return dx


# ------------------------------------------------------------------------------------------ StochasticBatchNormalization
def stochastic_bn_forward_training(x, running_mean, running_var, frames, gamma=0.2, beta=0.5, momentum=0.9):
    O = x.shape[0]
    y = torch.empty_like(x)
    mean, rstd = _n.vector_f32(x, O), _n.vector_f32(x, O)
    _n.bbcu_fp32_StochasticBatchNormalization_ForwardTraining(x, y, mean, rstd, running_mean, running_var, gamma, beta, momentum, O, frames,
                                                              x.shape[1])
    return y, mean, rstd


def stochastic_bn_reforward(x, mean, rstd, frames, gamma=0.2, beta=0.5):
    y = torch.empty_like(x)
    _n.bbcu_fp32_StochasticBatchNormalization_ReForward(x, y, mean, rstd, gamma, beta, x.shape[0], frames, x.shape[1])
    return y


def stochastic_bn_forward_inference(x, running_mean, running_var, frames, gamma=0.2, beta=0.5):
    y = torch.empty_like(x)
    _n.bbcu_fp32_StochasticBatchNormalization_ForwardInference(x, y, running_mean, running_var, gamma, beta, x.shape[0], frames, x.shape[1])
    return y


def stochastic_bn_backward(x, dy, mean, rstd, frames, gamma=0.2):
    dx = torch.empty_like(dy)
    _n.bbcu_fp32_StochasticBatchNormalization_Backward(x, dy, dx, mean, rstd, gamma, 1.0 / frames, dy.shape[0], frames, dy.shape[1], x.shape[1])
    return dx


# ------------------------------------------------------------------------------------------ BinaryLut6
def binary_lut6_forward(x, idx, table, frames, y=None, lop3_immediate=False):
    """Bit-packed inference forward; ``table`` is [nodes, 2] int32 (64-entry truth table per node).
    lop3_immediate: evaluate through the truth-table-immediate kernel (same results; aligned rows only)."""
    _chk(x, torch.int32, "x"); _chk(idx, torch.int32, "idx"); _chk(table, torch.int32, "table")
    O = idx.shape[0]
    if y is None:
        y = _n.empty_i32(x, O, x.shape[1])
    (_n.bbcu_bit_BinaryLut6_Forward_Lop3Immediate if lop3_immediate else _n.bbcu_bit_BinaryLut6_Forward)(x, y, idx, table, O, frames, x.shape[1])
    return y


def binary_lut6_forward_host(x, idx, table, frames, y=None):
    """BinaryLut6 forward on HOST tensors (int32, ideally pinned): chunked upload / kernel / download overlapped inside the library."""
    for t, n in ((x, "x"), (idx, "idx"), (table, "table")):
        if t.is_cuda or t.dtype != torch.int32 or not t.is_contiguous():
            raise ValueError(f"{n}: expected a contiguous int32 host tensor")
    O = idx.shape[0]
    if y is None:
        y = torch.empty((O, x.shape[1]), dtype=torch.int32).pin_memory()
    _n.bbcu_host_bit_BinaryLut6_Forward(x, y, idx, table, x.shape[0], O, frames, x.shape[1])
    return y


# ------------------------------------------------------------------------------------------ per-step neighbours
def clamp_(t, lo=0.0, hi=1.0):
    _n.bbcu_fp32_Vector_clamp(t, t, lo, hi, t.numel())
    return t


def softmax_cross_entropy(y, t, frames, pix_size=1):
    """bb::LossSoftmaxCrossEntropy::CalculateLoss: returns (dy, loss) with loss = -sum(loss_buf) / t_sum (the mean over frames)."""
    rows, stride = y.shape
    dy, loss = _n.empty_f32(y, rows, stride), _n.scalar_f64(y)
    _n.bbcu_fp32_LossSoftmaxCrossEntropyMean(y, t, dy, loss, pix_size, rows // pix_size, frames, stride)
    return dy, loss


def mean_squared_error(y, t, frames, batch_size=None, loss_buf=None, dy=None):
    """bb::LossMeanSquaredError::CalculateLoss (mean reduction): returns (dy, loss_buf); loss = loss_buf.sum() / frames seen."""
    nodes = y.shape[0]
    batch_size = frames if batch_size is None else batch_size
    if dy is None:
        dy = torch.empty_like(y)
    if loss_buf is None:
        loss_buf = torch.zeros(1024, dtype=torch.float64, device=y.device)
    _n.bbcu_fp32_LossMeanSquaredError(y, t, dy, loss_buf, loss_buf.numel(), nodes, frames, y.shape[1], 2.0 / (nodes * batch_size), 1.0 / nodes)
    return dy, loss_buf


def reduce_forward(x, out_nodes, frames, y=None):
    """bb::Reduce forward: y[o] = mean_i x[out_nodes * i + o]."""
    rows, stride = x.shape
    if y is None:
        y = _n.empty_f32(x, out_nodes, stride)
    _n.bbcu_fp32_Reduce_Forward(x, y, rows, out_nodes, frames, stride, y.shape[1])
    return y


def reduce_backward(dy, in_nodes, frames, dx=None):
    rows, stride = dy.shape
    if dx is None:
        dx = _n.empty_f32(dy, in_nodes, stride)
    _n.bbcu_fp32_Reduce_Backward(dy, dx, in_nodes, rows, frames, stride, dx.shape[1])
    return dx


def real_to_binary(x, frames, frame_mod=1, depth_mod=1, lo=0.0, hi=1.0, thresholds=None, point_size=None):
    """bb::RealToBinary forward to bit frames: [nodes, frames] fp32 -> [nodes * depth_mod, frames * frame_mod] bits.
    thresholds: optional fp32 [nodes, >= frames * frame_mod] (what a seeded value generator supplies in the reference)."""
    nodes = x.shape[0]
    point_size = nodes if point_size is None else point_size
    out_frames = frames * frame_mod
    y = _bits(x, nodes * depth_mod, out_frames)
    _n.bbcu_bit_fp32_RealToBinary_Forward(x, y, thresholds, 0 if thresholds is None else thresholds.shape[1], depth_mod, frame_mod, lo, hi,
                                          point_size, nodes // point_size, frames, x.shape[1], y.shape[1])
    return y


def binary_to_real(x, x_nodes, y_nodes, y_frames, frame_mux=1):
    """bb::BinaryToReal forward: bit (int32) or fp32 frames -> fp32 [y_nodes, y_frames], averaging node_mux x frame_mux inputs."""
    y = _n.empty_f32(x, y_nodes, fp32_stride(y_frames))
    forward = _n.bbcu_bit_fp32_BinaryToReal_Forward if x.dtype == torch.int32 else _n.bbcu_fp32_BinaryToReal_Forward
    forward(x, y, x_nodes // y_nodes, frame_mux, y_nodes, x.shape[1], y_frames, y.shape[1])
    return y


def binary_to_real_backward(dy, x_nodes, y_frames, frame_mux=1):
    y_nodes = dy.shape[0]
    dx = _n.empty_f32(dy, x_nodes, fp32_stride(y_frames * frame_mux))
    _n.bbcu_fp32_BinaryToReal_Backward(dy, dx, x_nodes // y_nodes, frame_mux, y_nodes, dx.shape[1], y_frames, dy.shape[1])
    return dx


BORDER_MODES = {"constant": 0, "reflect": 1, "reflect_101": 2, "replicate": 3, "wrap": 4}


def im2col_geometry(h, w, fh, fw, y_stride=1, x_stride=1, padding="valid"):
    """(out_h, out_w, y_offset, x_offset) of bb::ConvolutionIm2Col (include/bb/ConvolutionIm2Col.h:200-215)."""
    if padding == "valid":
        return ((h - fh + 1) + (y_stride - 1)) // y_stride, ((w - fw + 1) + (x_stride - 1)) // x_stride, 0, 0
    if padding == "same":
        return (h + y_stride - 1) // y_stride, (w + x_stride - 1) // x_stride, (fh - 1) // 2, (fw - 1) // 2
    raise ValueError(f"unknown padding {padding!r}")


def im2col_forward(x, frames, c, h, w, fh, fw, y_stride=1, x_stride=1, padding="valid", border_mode="reflect_101", border_value=0.0, y=None):
    """bb::ConvolutionIm2Col forward: [c*h*w, frames] (fp32, or int32 bit words) -> [c*fh*fw, frames*oh*ow].  `y`: an output buffer of
    that shape to write into (every word up to the last frame is written; nothing needs clearing)."""
    oh, ow, yo, xo = im2col_geometry(h, w, fh, fw, y_stride, x_stride, padding)
    of = frames * oh * ow
    if x.dtype == torch.int32:
        if y is None:
            y = _bits(x, c * fh * fw, of)
        _n.bbcu_bit_Im2Col_Forward(x, y, x_stride, y_stride, xo, yo, frames, x.shape[1], w, h, c, ow, oh, y.shape[1], fw, fh, BORDER_MODES[border_mode])
    else:
        if y is None:
            y = _n.empty_f32(x, c * fh * fw, fp32_stride(of))
        _n.bbcu_fp32_Im2Col_Forward(x, y, x_stride, y_stride, xo, yo, frames, x.shape[1], w, h, c, ow, oh, y.shape[1], fw, fh,
                                    BORDER_MODES[border_mode], border_value)
    return y


def im2col_backward(dy, frames, c, h, w, fh, fw, y_stride=1, x_stride=1, padding="valid"):
    oh, ow, yo, xo = im2col_geometry(h, w, fh, fw, y_stride, x_stride, padding)
    dx = _n.empty_f32(dy, c * h * w, fp32_stride(frames))
    _n.bbcu_fp32_Im2Col_Backward(dy, dx, x_stride, y_stride, xo, yo, frames, dx.shape[1], w, h, c, ow, oh, dy.shape[1], fw, fh)
    return dx


def col2im_forward(x, c, h, w, out_frames):
    """bb::ConvolutionCol2Im forward: [c, out_frames*h*w] -> [c*h*w, out_frames] (fp32, or int32 bit words)."""
    if x.dtype == torch.int32:
        y = _bits(x, c * h * w, out_frames)
        _n.bbcu_bit_Col2Im_Forward(x, y, w, h, c, x.shape[1], out_frames, y.shape[1])
    else:
        y = _n.empty_f32(x, c * h * w, fp32_stride(out_frames))
        _n.bbcu_fp32_Col2Im_Forward(x, y, w, h, c, x.shape[1], out_frames, y.shape[1])
    return y


def col2im_backward(dy, c, h, w, out_frames):
    dx = _n.empty_f32(dy, c, fp32_stride(out_frames * h * w))
    _n.bbcu_fp32_Col2Im_Backward(dy, dx, w, h, c, dx.shape[1], out_frames, dy.shape[1])
    return dx


def maxpool_forward(x, frames, c, h, w, fh, fw, want_argmax=True):
    """bb::MaxPooling forward.  fp32: returns (y, argmax or None); int32 bit words: returns y."""
    oh, ow = (h + fh - 1) // fh, (w + fw - 1) // fw
    if x.dtype == torch.int32:
        y = _bits(x, c * oh * ow, frames, x.shape[1])
        _n.bbcu_bit_MaxPooling_Forward(x, y, fh, fw, w, h, ow, oh, c, frames, x.shape[1])
        return y
    y = _n.empty_f32(x, c * oh * ow, x.shape[1])
    am = _n.empty_i32(x, c * oh * ow, x.shape[1]) if want_argmax else None
    _n.bbcu_fp32_MaxPooling_Forward(x, y, am, fh, fw, w, h, ow, oh, c, frames, x.shape[1])
    return y, am


def maxpool_backward(sel, dy, frames, c, h, w, fh, fw, bit_input=False):
    """sel: the forward's argmax (fp32 layer) or, with bit_input=True, the forward's bit-packed input."""
    oh, ow = (h + fh - 1) // fh, (w + fw - 1) // fw
    dx = _n.empty_f32(dy, c * h * w, dy.shape[1])
    if bit_input:
        _n.bbcu_bit_fp32_MaxPooling_Backward(sel, dy, dx, fh, fw, w, h, ow, oh, c, frames, sel.shape[1], dy.shape[1])
    else:
        _n.bbcu_fp32_MaxPooling_Backward(sel, dy, dx, fh, fw, w, h, ow, oh, c, frames, dy.shape[1])
    return dx


class Adam:
    """bb::OptimizerAdam over a list of (param, grad) CUDA tensors (include/bb/OptimizerAdam.h:142-184)."""

    def __init__(self, params, grads, lr=0.001, beta1=0.9, beta2=0.999):
        self.params, self.grads = list(params), list(grads)
        self.m = [torch.zeros_like(p) for p in self.params]
        self.v = [torch.zeros_like(p) for p in self.params]
        dev = self.params[0].device
        self._sizes = torch.tensor([p.numel() for p in self.params], dtype=torch.int32, device=dev)
        mk = lambda ts: torch.tensor([t.data_ptr() for t in ts], dtype=torch.int64, device=dev)
        self._tabs = [mk(self.params), mk(self.grads), mk(self.m), mk(self.v)]
        self.lr, self.beta1, self.beta2 = lr, beta1, beta2
        self.b1, self.b2 = beta1, beta2

    def _step(self, operator):
        lr_t = self.lr * (1.0 - self.b2) ** 0.5 / (1.0 - self.b1)
        operator(len(self.params), self._sizes, *self._tabs, lr_t, self.beta1, self.beta2)
        self.b1 *= self.beta1
        self.b2 *= self.beta2

    def step(self):
        self._step(_n.bbcu_fp32_OptimizerAdam)

    def zero_grad(self):
        for g in self.grads:
            g.zero_()

    def update(self):          # Optimizer::Update = Step + ZeroGrad (include/bb/Optimizer.h:29-33), one pass over the tables
        self._step(_n.bbcu_fp32_OptimizerAdamUpdate)


# ------------------------------------------------------------------------------------------ frame-sharded halves
def dl6_forward_stats(x, idx, W, frames, y, sums, bias=BIAS, lut_binarize=False, binary=True):
    """Pass 1 of the training forward on this rank's frames: raw LUT values into y, per-node (sum y, sum y^2) into sums [O,2] fp64."""
    _n.bbcu_fp32_DifferentiableLut6_ForwardStats(x, y, idx, W, sums, bias, idx.shape[0], frames, x.shape[1], int(lut_binarize), int(binary))


def dl6_forward_normalize(y, sums, mean, rstd, running_mean, running_var, frames, total_frames, gamma=0.3, beta=0.5, momentum=0.9, binary=True):
    """Pass 2: statistics from the (all-reduced) sums over total_frames, then normalise y in place."""
    _n.bbcu_fp32_DifferentiableLut6_ForwardNormalize(y, sums, mean, rstd, running_mean, running_var, gamma, beta, momentum, y.shape[0], frames,
                                                     y.shape[1], int(total_frames), int(binary))


def dl6_backward_stats(x, dy, idx, W, mean, rstd, frames, sums, gamma=0.3, beta=0.5, bias=BIAS, lut_binarize=False, binary=True):
    _n.bbcu_fp32_DifferentiableLut6_BackwardStats(x, dy, idx, W, mean, rstd, sums, gamma, beta, bias, idx.shape[0], frames, x.shape[1],
                                                  int(lut_binarize), int(binary))


def dl6_backward_stats_from_output(y, dy, rstd, frames, sums, gamma=0.3, beta=0.5):
    """The sums of dl6_backward_stats from the layer's training output y (non-binary mode): no second LUT evaluation."""
    _n.bbcu_fp32_DifferentiableLut6_BackwardStatsFromOutput(y, dy, rstd, sums, gamma, beta, y.shape[0], frames, y.shape[1], 0)


def dl6_backward_apply(x, dy, dx, idx, W, dW, mean, rstd, sums, n_in, frames, total_frames, gamma=0.3, beta=0.5, bias=BIAS, lut_binarize=False,
                       binary=True):
    O = idx.shape[0]
    dmean, dvar = _n.vector_f32(dy, O), _n.vector_f32(dy, O)
    _n.bbcu_fp32_DifferentiableLut6_BackwardApply(x, dy, dx, idx, W, dW, mean, rstd, sums, dmean, dvar, gamma, beta, bias, n_in, O, frames,
                                                  dy.shape[1], int(total_frames), int(lut_binarize), int(binary))
    return dx
