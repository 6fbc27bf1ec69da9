"""binarybrain_b200._native, the operators on torch tensors: which memory of a tensor an operator gets."""
import os

import pytest


@pytest.fixture(scope="module")
def native():
    from binarybrain_b200 import abi
    if not os.path.exists(abi.LIB_PATH):
        pytest.skip("library not built")
    import torch  # noqa: F401  (the module needs torch's libraries loaded)
    from binarybrain_b200 import _native
    return _native


def test_written_tensors_get_memory_of_their_own_and_read_ones_do_not(native):
    """An operator that writes into a lazily cloned tensor must not reach the tensor that it was cloned from; one that reads needs no copy."""
    import torch
    from binarybrain_b200 import abi
    written, read = torch._lazy_clone(torch.zeros(64)), torch._lazy_clone(torch.ones(64))
    with pytest.raises(abi.BbcuError):                                   # the arguments are taken, the size is refused: nothing runs
        native.bbcu_fp32_Vector_clamp(written, read, 0.0, 1.0, -1, 0)
    assert not torch._C._is_cow_tensor(written) and torch._C._is_cow_tensor(read)


def test_a_tensor_without_memory_is_an_error(native):
    import torch
    for args in ((torch.eye(3).to_sparse(), torch.ones(9)), (torch.ones(9), torch.eye(3).to_sparse())):
        with pytest.raises(RuntimeError, match="storage"):
            native.bbcu_fp32_Vector_clamp(*args, 0.0, 1.0, 0, 0)


def test_the_small_layer_limits_are_those_of_the_library(native):
    from binarybrain_b200 import ops
    assert (ops.SMALL_NODE_FRAMES, ops.SMALL_FRAMES) == (native.SMALL_NODE_FRAMES, native.SMALL_FRAMES) == (1 << 21, 4096)
    assert "SMALL_FRAMES" in vars(ops)                                   # looked up once
    with pytest.raises(AttributeError):
        ops.SMALL_LAYERS


class _Step:
    """The training step of a layer of three nodes on fp32 frames, with the arguments that a call gives in another form."""

    def __init__(self, frames, device):
        import torch
        from binarybrain_b200 import ops
        g = torch.Generator().manual_seed(1)
        self.ops, self.frames = ops, frames
        self.x, self.dy, self.W = (torch.rand(s, generator=g).to(device) for s in ((7, 8), (3, 8), (3, 64)))
        self.idx = torch.tensor([[0, 1, 2, 3, 4, 5], [6, 5, 4, 3, 2, 1], [0, 2, 4, 6, 1, 3]], dtype=torch.int32).to(device)
        self.new = lambda *s: torch.zeros(s, device=device)

    def forward(self, x=None, **kw):
        return self.ops.differentiable_lut6_forward_training(self.x if x is None else x, self.idx, self.W, self.new(3), self.new(3) + 1, self.frames, **kw)

    def backward(self, x=None, dy=None, **kw):
        dW = self.new(3, 64)
        dx = self.ops.differentiable_lut6_backward(self.x if x is None else x, self.dy if dy is None else dy, self.idx, self.W, dW, self.new(3) + 0.5, self.new(3) + 2,
                                                   7, self.frames, **kw)
        return dx, dW


def test_the_training_step_takes_what_its_operators_take(native):
    """Flags that int() takes, addresses as outputs, tensors of more dimensions.  A negative number of frames: the arguments are taken, nothing runs."""
    import numpy as np
    import torch
    step, buffer = _Step(-1, "cpu"), torch.zeros(64)
    address = buffer.data_ptr()
    taken = [{}] + [{name: flag} for name in ("binary", "lut_binarize") for flag in (True, np.bool_(True), 1.0, torch.tensor(0.0), np.int64(1))]
    for kw in taken + [{"y": address}, {"mean": address}, {"rstd": address}, {"x": step.x[:, :, None]}]:
        with pytest.raises(RuntimeError):                                # from the library, or for want of a device
            step.forward(**kw)
    for kw in taken + [{"dx": address}, {"x": step.x[:, :, None]}]:
        with pytest.raises(RuntimeError):
            step.backward(**kw)


def test_the_training_step_refuses_what_its_operators_refuse(native):
    step = _Step(-1, "cpu")
    for kw in ({"binary": None}, {"lut_binarize": [1]}, {"y": "y"}, {"mean": [0.0]}, {"rstd": 0.5}):
        with pytest.raises(TypeError):
            step.forward(**kw)
    for kw in ({"binary": None}, {"lut_binarize": [1]}, {"dx": "dx"}):
        with pytest.raises(TypeError):
            step.backward(**kw)
    with pytest.raises(OverflowError):
        step.forward(binary=1 << 40)
    with pytest.raises(IndexError):
        step.forward(x=step.x[0])
    with pytest.raises(AssertionError):
        step.backward(dy=step.dy[:, :4])


@pytest.mark.gpu
def test_the_training_step_with_other_forms_of_its_arguments():
    import numpy as np
    import torch
    step = _Step(8, "cuda")
    for binary in (False, True):
        want, (dx_w, dW_w) = step.forward(binary=binary), step.backward(binary=binary)
        out = [step.new(3, 8), step.new(3), step.new(3)]
        got = step.forward(binary=np.bool_(binary), lut_binarize=0.0, **{k: t.data_ptr() for k, t in zip(("y", "mean", "rstd"), out)})
        assert [int(p) for p in got] == [t.data_ptr() for t in out]
        assert all(torch.equal(a, b) for a, b in zip(out, want))
        dx = step.new(7, 8)
        address, dW = step.backward(binary=float(binary), lut_binarize=np.bool_(False), dx=dx.data_ptr())
        assert address == dx.data_ptr() and torch.allclose(dx, dx_w, rtol=0, atol=1e-5) and torch.allclose(dW, dW_w, rtol=0, atol=1e-5)


@pytest.mark.gpu
def test_a_lazily_cloned_output_leaves_its_twin_alone():
    import torch
    from binarybrain_b200 import ops
    base = torch.full((1000,), 3.0, device="cuda")
    twin = torch._lazy_clone(base)
    ops.clamp_(twin)
    assert (twin == 1.0).all() and (base == 3.0).all()
