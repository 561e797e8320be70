"""The native view of the launchers (csrc/py_calls.cpp): how arguments are taken. No GPU: every call here ends before
a kernel would be launched."""
import pytest

from hipml_b200 import _lib


class _Tensor:
    """What the module asks of a tensor, with a count of the questions."""

    def __init__(self, fails=False):
        self.asked, self.fails = 0, fails

    def data_ptr(self):
        self.asked += 1
        if self.fails:
            raise RuntimeError("no storage")
        return 256


@pytest.mark.parametrize("bad", [0, 2, 4])
def test_nothing_is_converted_after_an_argument_has_failed(bad):
    args = [_Tensor(fails=i == bad) for i in range(5)]
    with pytest.raises(RuntimeError, match="no storage"):
        _lib.calls().kv_append_f32(*args, 1024)
    assert [a.asked for a in args] == [1] * (bad + 1) + [0] * (4 - bad)


def test_what_is_not_a_whole_number_is_a_type_error():
    args = [_Tensor() for _ in range(5)]
    with pytest.raises(TypeError):
        _lib.calls().kv_append_f32(*args, 1.5)
    with pytest.raises(TypeError, match="5 arguments given, 6 wanted"):
        _lib.calls().kv_append_f32(*args)
