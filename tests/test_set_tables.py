"""ICGenerator.set_tables against a recording stand-in for the library: what the
plan is given follows the caller's table whatever the caller did to it."""

import numpy as np
import pytest
import torch

from aarambam_gb300 import _lib
from aarambam_gb300.ic import ICGenerator


class Recorder:
    """aar_set_tables alone: keeps the tables as the plan would."""

    def __init__(self, rc=0):
        self.given, self.rc = [], rc

    def aar_set_tables(self, h, alpha, x0, M):
        if self.rc == 0:
            self.given.append((np.ctypeslib.as_array(alpha, (M, M, M)).copy(), np.ctypeslib.as_array(x0, (M,)).copy()))
        return self.rc

    def aar_last_error(self, h):
        return b"refused"


def generator(alpha, x0):
    g = ICGenerator.__new__(ICGenerator)
    g.L, g.h = Recorder(), None
    g._alpha, g._x0 = np.zeros((0, 0, 0)), np.zeros(0)
    g.set_tables(alpha, x0)
    return g


@pytest.mark.parametrize("make", [np.array, lambda a: torch.tensor(a).numpy()])
def test_a_table_changed_in_place_is_set_again(make):
    alpha, x0 = make(np.ones((2, 2, 2))), make(np.array([1.0, 0.5]))
    g = generator(alpha, x0)
    alpha[0, 0, 1] = 7.0
    g.set_tables(alpha)
    x0[1] = 0.25
    g.set_tables(alpha, x0)
    g.set_tables(alpha.copy(), x0.copy())  # unchanged: not set again
    assert len(g.L.given) == 3
    assert g.L.given[1][0][0, 0, 1] == 7.0 and g.L.given[1][1][1] == 0.5 and g.L.given[2][1][1] == 0.25


def test_a_refused_table_is_not_taken_for_the_plan_s():
    alpha, x0 = np.ones((2, 2, 2)), np.array([1.0, 0.5])
    g = generator(alpha, x0)
    g.L.rc = 1
    with pytest.raises(_lib.AarError):
        g.set_tables(2 * alpha)
    g.L.rc = 0
    g.set_tables(2 * alpha)
    assert len(g.L.given) == 2 and g.L.given[1][0][0, 0, 0] == 2.0


@pytest.mark.parametrize("alpha,x0", [(np.ones((3, 3, 3)), None), (np.ones((3, 3, 2)), np.ones(3)), (np.ones((2, 2)), None)])
def test_tables_that_are_too_short_are_refused(alpha, x0):
    """Before the library reads past their end: x0 of two modes beside an alpha
    of three, an alpha that is not a cube."""
    g = generator(np.ones((2, 2, 2)), np.array([1.0, 0.5]))
    with pytest.raises(ValueError):
        g.set_tables(alpha, x0)
    assert len(g.L.given) == 1 and g.n_modes == 2
