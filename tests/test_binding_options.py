"""Options of a call are read on that call: whatever was passed before, and whatever the passed
objects do later."""
import math

import pytest

from libsdca_b200 import binding


class Radius:
    """A number kept in an object that changes in place, as a 0-d tensor does."""

    def __init__(self, value):
        self.value = value

    def __float__(self):
        return float(self.value)

    __int__ = __index__ = lambda self: int(self.value)


@pytest.mark.parametrize("name", ["lo", "hi", "rhs", "rho", "alpha"])
def test_options_that_change_in_place_are_read_again(name):
    import torch
    for box, change in ((Radius(1.0), lambda b: setattr(b, "value", 4.0)),
                        (torch.tensor(1.0), lambda b: b.fill_(4.0))):
        assert getattr(binding._call_opts({name: box}), name) == 1.0
        change(box)
        assert getattr(binding._call_opts({name: box}), name) == 4.0


def test_integers_that_change_in_place_are_read_again():
    k = Radius(2)
    assert binding._call_opts({"k": k}).k == 2
    k.value = 7
    assert binding._call_opts({"k": k}).k == 7


def test_equal_options_that_are_not_the_same():
    for first, then in ((0.0, -0.0), (-0.0, 0.0)):
        binding._call_opts({"lo": first})
        assert math.copysign(1.0, binding._call_opts({"lo": then}).lo) == math.copysign(1.0, then)


def test_options_agree_with_a_fresh_struct():
    for opts in ({}, dict(k=5), dict(k=True), dict(k=5.0), dict(rhs=2, rho=0.5), dict(precision="single"),
                 dict(accurate_math=True), dict(accurate_math=0), dict(lo=0, hi=float("inf"))):
        got, want = binding._call_opts(opts), binding.make_opts(**opts)
        assert bytes(got) == bytes(want), opts
    for bad in (dict(precision="long double"), dict(precision="half")):
        with pytest.raises(binding.SdcabError):
            binding._call_opts(bad)
    with pytest.raises(TypeError):
        binding._call_opts(dict(no_such_option=1))
