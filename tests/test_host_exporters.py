"""Addresses are taken only of objects that hold their values themselves: a buffer that another object provides for the
occasion is gone when the call that read its address returns."""
import sys

import numpy as np
import pytest

import relxill_gb300 as R

E = np.exp(np.linspace(np.log(0.5), np.log(20.0), 9))


class Lent:
    """Hands out a buffer of its own making on each request."""

    def __buffer__(self, flags):
        return memoryview(E.copy())

    def __len__(self):
        return len(E)


@pytest.mark.skipif(sys.version_info < (3, 12), reason="classes cannot export buffers")
def test_lent_buffers():
    assert R._host().arrays([E, Lent()]) is None
    assert R._host().arrays([E, E[1:]]) is not None  # a view holds what it is a view of
