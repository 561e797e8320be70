"""The native view of the launchers (csrc/py_calls.cpp): how arguments are taken. No GPU: every call here ends before
a kernel would be launched."""
import numpy as np
import pytest
import torch

from hipml_b200 import _lib, api


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


@pytest.mark.parametrize("sections", [None, [], [11, 11, 10], (11, 11, 10, 0), [11.0, 11.0, 10.0, 0.0],
                                      np.array([11, 11, 10, 0]), torch.tensor([11, 11, 10, 0])], ids=str)
def test_sections_may_be_any_sequence_of_up_to_four_numbers(sections):
    t = [_Tensor() for _ in range(9)]
    with pytest.raises(TypeError, match="real number"):   # of eps, the last argument: all before it were taken
        api.attn_front_append_q8(*t, 24, 4, 256, 64, 1e7, None, sections=sections, stride=8)


@pytest.mark.parametrize("sections,error", [([1, 2, 3, 4, 5], IndexError), (7, TypeError), (["x"], ValueError)], ids=str)
def test_other_sections_are_refused(sections, error):
    t = [_Tensor() for _ in range(9)]
    with pytest.raises(error):
        api.attn_front_append_q8(*t, 24, 4, 256, 64, 1e7, 1e-6, sections=sections, stride=8)
