"""The drop-in modules' resident graphs are found by the contents of the caller's arrays."""
import numpy as np
import pytest

from gde import dropin


@pytest.mark.parametrize("which", [0, 1, 2])
def test_every_byte_shape_and_type_counts(which):
    arrays = [np.arange(5, dtype=np.int64), np.arange(7, dtype=np.int32), np.arange(4, dtype=np.float64)]
    kept = dropin._Contents(arrays, False)
    assert kept.equal(dropin._arrays(*arrays), False)
    assert not kept.equal(dropin._arrays(*arrays), True)
    for change in (lambda a: a[:-1], lambda a: a.astype(np.int16), lambda a: np.where(np.arange(a.size) == 2, 9, a)):
        other = list(arrays)
        other[which] = change(arrays[which])
        assert not kept.equal(dropin._arrays(*other), False)
    other = list(arrays)
    other[which] = np.repeat(arrays[which], 2)[::2]  # the same values in a strided array
    assert kept.equal(dropin._arrays(*other), False)
    arrays[which][-1] += 1  # an edit in place
    assert not kept.equal(dropin._arrays(*arrays), False)


def test_no_degree_is_not_some_degree():
    a = [np.arange(5), np.arange(7)]
    assert dropin._Contents([*a, None], False).equal(dropin._arrays(*a, None), False)
    assert not dropin._Contents([*a, None], False).equal(dropin._arrays(*a, np.ones(4)), False)
