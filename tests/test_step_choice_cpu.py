"""CPU: which captured steps are cut at all, and which are one chain of whole calls (pure host logic of ``lethe_b200.ops``)."""
import pytest

from lethe_b200 import ops

B200_SMS = 148


@pytest.mark.parametrize("gate,delta,NT,BH,cut", [
    (ops.GATE_SCALAR, True, 32, 16, True), (ops.GATE_CHANNEL, True, 32, 16, True), (ops.GATE_CHANNEL, True, 37, 8, True),
    (ops.GATE_CHANNEL, True, 36, 8, False), (ops.GATE_NONE, False, 32, 16, False), (ops.GATE_SCALAR, False, 64, 64, True),
    (ops.GATE_CHANNEL, False, 63, 64, False)])
def test_which_steps_are_cut(gate, delta, NT, BH, cut):
    assert ops.step_is_cut(gate, delta, NT, BH, B200_SMS) == cut


@pytest.mark.parametrize("gate,V,delta,BH,chain", [
    (ops.GATE_SCALAR, 128, True, 64, False), (ops.GATE_CHANNEL, 128, True, 16, False), (ops.GATE_CHANNEL, 128, True, 19, True),
    (ops.GATE_CHANNEL, 64, True, 37, False), (ops.GATE_CHANNEL, 64, True, 38, True), (ops.GATE_CHANNEL, 64, False, 88, False),
    (ops.GATE_CHANNEL, 64, False, 89, True), (ops.GATE_CHANNEL, 128, False, 80, False)])
def test_which_steps_are_one_chain(gate, V, delta, BH, chain):
    assert ops.step_is_chain(gate, V, delta, BH, B200_SMS) == chain
