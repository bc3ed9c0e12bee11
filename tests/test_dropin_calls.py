"""The drop-in's native calls: what they take, what they refuse and with which error, as the ctypes binding of the same entry points.  Every
call here is refused before anything reaches a GPU."""
import ctypes as C
import inspect

import pytest

from nectarml_b200 import _lib, _nectarml

CONV, F32 = _nectarml.tensor.conv, _nectarml.DType.Float32


@pytest.fixture(autouse=True)
def _built(lib):
    pass


def _calls():
    for name, fn in vars(type(CONV)).items():
        if not name.startswith("_"):
            fn = getattr(CONV, name)
            yield name, fn, len(inspect.signature(fn).parameters)


@pytest.mark.parametrize("name,fn,n", list(_calls()))
def test_every_convolution_call(name, fn, n):
    names = list(inspect.signature(fn).parameters)
    args = [0] * n
    args[names.index("dtype")] = F32
    with pytest.raises(RuntimeError, match="nectarml_b200: "):  # zero sizes: refused by the entry point itself
        fn(*args)
    with pytest.raises(RuntimeError, match="nectarml_b200: "):
        fn(**dict(zip(names, args)))
    for bad in (1.0, None, "1"):
        at = names.index("B")
        with pytest.raises(C.ArgumentError, match="cannot be interpreted as an integer"):
            fn(*args[:at], bad, *args[at + 1:])
    args[names.index("dtype")] = _nectarml.DType.Int32
    with pytest.raises(RuntimeError, match="only support float32 and float16"):
        fn(*args)


def test_integers_are_cut_to_the_width_of_the_parameter():
    # -1 as an unsigned pointer, 2^32 as an int of 0: taken, and refused for the sizes alone
    with pytest.raises(RuntimeError, match="invalid argument"):
        _nectarml.tensor.matmul(-1, 1 << 70, (1 << 32, 4), (4, 4), F32)


class _Stands:
    def __init__(self, v):
        self._as_parameter_ = v


@pytest.mark.parametrize("wrap", [lambda t, v: v, lambda t, v: t(v), lambda t, v: _Stands(v), lambda t, v: _Stands(t(v)), lambda t, v: _Stands(_Stands(v))],
                         ids=["int", "ctypes", "as_parameter", "as_parameter_ctypes", "as_parameter_twice"])
def test_what_ctypes_takes_for_an_integer(wrap):
    """The value arrives as well: two groups are refused in another way than one group of no channels."""
    def call(groups):
        names = list(inspect.signature(CONV.conv2d).parameters)
        args = dict.fromkeys(names, wrap(C.c_int, 1))
        args.update({n: wrap(C.c_size_t, 16) for n in names if n.endswith("_ptr") or n.endswith("_size")})
        args.update(C_in=wrap(C.c_int, 0), groups=wrap(C.c_int, groups), dtype=F32, half_precision=False)
        with pytest.raises(RuntimeError) as e:
            CONV.conv2d(**args)
        return str(e.value)
    assert "invalid argument" in call(1) and call(1) != call(2)
    with pytest.raises(RuntimeError, match="invalid argument"):
        _nectarml.tensor.matmul(wrap(C.c_size_t, 0), wrap(C.c_size_t, 0), (2, 0), (0, 2), F32)


@pytest.mark.parametrize("bad", [_Stands("1"), _Stands(_Stands(None)), C.c_short(1), C.c_size_t(1)])
def test_what_ctypes_refuses_for_an_int(bad):
    names = list(inspect.signature(CONV.conv2d).parameters)
    args = dict.fromkeys(names, 0)
    args.update(B=bad, dtype=F32)
    with pytest.raises(C.ArgumentError):
        CONV.conv2d(**args)


@pytest.mark.parametrize("a,b,error", [((2, 0), (0, 2), RuntimeError), ((2, 3), (4, 2), RuntimeError), ((2,), (2, 2), RuntimeError), (3, (2, 2), TypeError),
                                       (iter((2, 2)), (2, 2), TypeError), ((2, "x"), (2, 2), ValueError), ((2, None), (2, 2), TypeError)])
def test_matmul_shapes(a, b, error):
    with pytest.raises(error):
        _nectarml.tensor.matmul(0, 0, a, b, F32)


def test_a_shape_that_changes_while_it_is_read():
    """The sizes are those of the moment of the call."""
    class Clears:
        def __int__(self):
            dims.clear()
            return 1 << 31  # (as an int: negative, refused)
    dims = [Clears()] + [2] * 1000
    with pytest.raises(RuntimeError, match="invalid argument"):
        _nectarml.tensor.matmul(0, 0, dims, (2, 2), F32)
    assert dims == []


def test_matmul_pointers():
    with pytest.raises(C.ArgumentError):
        _nectarml.tensor.matmul(None, 0, (2, 2), (2, 2), F32)
    with pytest.raises(C.ArgumentError):
        _nectarml.free_cuda(1.5)


def test_the_binding_has_every_entry_point(lib):
    from nectarml_b200 import _dropin
    assert {n[len("nml_ref_"):] for n in _lib.SYMBOLS if n.startswith("nml_ref_")} == {n for n in vars(_dropin) if not n.startswith("_")}
