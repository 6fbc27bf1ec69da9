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


@pytest.mark.gpu
def test_a_lazily_cloned_output_leaves_its_twin_alone():
    import torch
    from binarybrain_b200 import ops
    base = torch.full((1000,), 3.0, device="cuda")
    twin = torch._lazy_clone(base)
    ops.clamp_(twin)
    assert (twin == 1.0).all() and (base == 3.0).all()
