"""Pickles of QubitOperator made when its terms were a plain list load as operators
that can be changed (no GPU)."""

import copy
import pickle

import pytest

import qforte_b200 as qb


def _terms():
    c = qb.Circuit()
    c.add(qb.gate("X", 0, 0))
    c.add(qb.gate("Z", 2, 2))
    return [[0.5 + 0.25j, c], [2.0 + 0j, qb.Circuit()]]


@pytest.mark.parametrize("protocol", range(2, pickle.HIGHEST_PROTOCOL + 1))
def test_pickle_of_a_plain_list_loads(protocol):
    old = qb.QubitOperator()
    old._t = _terms()
    got = pickle.loads(pickle.dumps(old, protocol))
    got.mult_coeffs(2.0)
    got.add(1.0, qb.Circuit())
    assert [c for c, _ in got.terms()] == [1.0 + 0.5j, 4.0, 1.0]
    assert got.terms()[0][1] == _terms()[0][1]


def test_copies_share_and_separate_terms():
    qo = qb.QubitOperator()
    for c, circ in _terms():
        qo.add(c, circ)
    shallow, deep = copy.copy(qo), copy.deepcopy(qo)
    qo.mult_coeffs(3.0)
    assert shallow.terms()[1][0] == 6.0 and deep.terms()[1][0] == 2.0
