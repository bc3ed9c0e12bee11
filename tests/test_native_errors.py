"""Errors of the native host path: arguments that it refuses before anything reaches a GPU raise, with the type torch or Python
gives them, and never end the process."""
import pytest
import torch

from nectarml_b200 import ops, train


@pytest.fixture(autouse=True)
def _built(lib):
    pass


def _bn(x):
    p, ws = torch.zeros(8), ops.Workspace()
    return ops._native.bn_forward(x, None, p, p, 1, 0.2, 1e-5, None, False, ws)


def test_tensor_without_channels():
    empty = torch.zeros(4, 0, dtype=torch.float16)
    for call in (lambda: _bn(empty), lambda: ops._native.act_forward(empty, 1, 0.0, False),
                 lambda: ops._native.act_backward(empty, None, empty, 1, 0.0)):
        with pytest.raises(AssertionError, match="without channels"):
            call()


def test_torch_errors_keep_their_type():
    with pytest.raises(IndexError):
        _bn(torch.zeros((), dtype=torch.float16))


def test_unsupported_tensors():
    w = torch.zeros(8, 8)
    with pytest.raises(_error(), match="CUDA device"):
        ops.linear_forward(torch.zeros(2, 8), w)
    with pytest.raises(_error(), match="float32 and float16"):
        ops.linear_forward(torch.zeros(2, 8, dtype=torch.float64), w)
    with pytest.raises(AssertionError):
        ops.linear_forward(torch.zeros(2, 7), w)


def _error():
    from nectarml_b200 import _lib
    return _lib.NectarB200Error


def test_layers_refuse_forward_mode():
    """A layer without a forward-mode derivative says so, as an autograd function without one does; it must not return a value
    whose tangent is missing."""
    import torch.autograd.forward_ad as fwd
    store = train.ParamStore("cpu")
    conv, bn = train.Conv(store, 8, 8, 3, 1, 1), train.BatchNormAct(store, 8)
    store.finalize(1)
    x, token = torch.zeros(1, 4, 4, 8, dtype=torch.float16), torch.zeros((), requires_grad=True)
    with fwd.dual_level():
        dual = fwd.make_dual(x, torch.ones_like(x))
        for call in (lambda: conv(dual, token), lambda: bn(dual, token), lambda: bn(x, token, residual=dual),
                     lambda: bn(x, token, join=dual)):
            with pytest.raises(NotImplementedError):
                call()
