"""QubitOperator's kept device sum: one made from equal terms is reused until the
operator or one of its circuits changes, by any method, and copies and pickles
do not carry it (no GPU: the device sum is replaced by the term list)."""

import copy
import pickle

import pytest

import qforte_b200 as qb
from qforte_b200 import device


@pytest.fixture
def calls(monkeypatch):
    made = []

    def fake(terms, segments=None, nsegment=1):
        made.append(list(terms))
        return made[-1]

    monkeypatch.setattr(device, "sum_from_terms", fake)
    return made


def _operator():
    qo = qb.QubitOperator()
    for q, lab in ((0, "Z"), (1, "X"), (2, "Y")):
        c = qb.Circuit()
        c.add(qb.gate(lab, q, q))
        c.add(qb.gate("Z", q + 1, q + 1))
        qo.add(0.5 + q, c)
    qo.simplify()
    return qo


CHANGES = {
    "add": lambda qo: qo.add(0.25, qb.Circuit()),
    "add_op": lambda qo: qo.add(_operator()),
    "set_coeffs": lambda qo: qo.set_coeffs([1.0, 2.0, 3.0]),
    "mult_coeffs": lambda qo: qo.mult_coeffs(2.0),
    "simplify": lambda qo: (qo.add(0.25, qo.terms()[0][1]), qo.simplify()),
    "operator_product": lambda qo: qo.operator_product(_operator()),
    "circuit add": lambda qo: qo.terms()[1][1].add(qb.gate("X", 0, 0)),
    "circuit add_circuit": lambda qo: qo.terms()[1][1].add(qo.terms()[0][1]),
    "circuit insert_gate": lambda qo: qo.terms()[1][1].insert_gate(0, qb.gate("X", 0, 0)),
    "circuit remove_gate": lambda qo: qo.terms()[1][1].remove_gate(0),
    "circuit swap_gates": lambda qo: qo.terms()[0][1].swap_gates(0, 1),
}


@pytest.mark.parametrize("change", CHANGES)
def test_changed_operators_are_gathered_again(calls, change):
    qo = _operator()
    first = qo._device_sum()
    assert qo._device_sum() is first and len(calls) == 1
    CHANGES[change](qo)
    assert qo._device_sum() == qo._pauli_terms(applied=True)
    assert len(calls) == 2


def test_gate_lists_are_gathered_on_each_call(calls):
    qo = qb.QubitOperator()
    c = qb.Circuit()
    c.add(qb.gate("X", 0, 0))
    qo.add(1.0, c)
    qo._device_sum()
    c.add(qb.gate("Z", 1, 1))
    assert qo._device_sum() == qo._pauli_terms(applied=True) and len(calls) == 2


@pytest.mark.parametrize("how", [copy.copy, copy.deepcopy, lambda x: pickle.loads(pickle.dumps(x))])
def test_copies(calls, how):
    qo = _operator()
    first = qo._device_sum()
    other = how(qo)
    assert other._pauli_terms() == qo._pauli_terms()
    other.mult_coeffs(3.0)
    assert other._device_sum() == other._pauli_terms()
    assert qo._device_sum() == qo._pauli_terms()
    assert first is not other._device_sum()
