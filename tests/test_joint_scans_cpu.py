"""CPU: which scans the library launches with the kernel beside them in one, and that a captured step is planned by what it says
(``lethe_gdn_joint_scans``)."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

from lethe_b200 import native, ops

B200_SMS = 148


def joint(gate, V, delta, BH, NT=64, lean=1, sms=B200_SMS):
    return native.lib().lethe_gdn_joint_scans(ctypes.byref(ops._Dims(1, BH, 64 * NT, 128, V, gate, delta)), lean, sms)


@pytest.mark.parametrize("V", [64, 128])
@pytest.mark.parametrize("gate,delta", [(ops.GATE_SCALAR, 1), (ops.GATE_NONE, 0), (ops.GATE_CHANNEL, 0), (ops.GATE_CHANNEL, 1), (ops.GATE_CHANNEL, 2)])
def test_a_captured_step_is_one_chain_where_both_scans_are_joint(monkeypatch, gate, delta, V):
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda dev: SimpleNamespace(multi_processor_count=B200_SMS))
    for NT in (1, 2, 4, 8, 64):
        for BH in list(range(1, 200)) + [256, 512, 1024]:
            bits = joint(gate, V, delta, BH, NT)
            assert ops.step_is_chain(gate, V, delta != 0, BH, B200_SMS, NT) == (bits == 3 and NT >= 8)      # (shorter ones are never cut)
            buf = SimpleNamespace(dims=SimpleNamespace(gate=gate, V=V, delta=delta))
            assert ops.GdnStepGraph._joint_scans(buf, BH, NT, None) == bits
            if gate != ops.GATE_CHANNEL:
                assert bits == 0


def test_none_for_a_call_that_leaves_every_record_or_for_bad_sizes():
    assert joint(ops.GATE_CHANNEL, 128, 1, 64) == 3
    assert joint(ops.GATE_CHANNEL, 128, 1, 64, lean=0) == 0
    assert joint(ops.GATE_CHANNEL, 96, 1, 64) == 0
    assert native.lib().lethe_gdn_joint_scans(None, 1, B200_SMS) == 0


F, A = 1, 2      # forward, adjoint


@pytest.mark.parametrize("V,delta,BH,NT,lean,bits", [
    # one CTA per SM: short sequences of many pairs are a row of rounds that are all start
    (128, 0, 1024, 1, 1, 0), (128, 0, 256, 2, 1, 0), (128, 0, 256, 3, 1, A), (128, 0, 256, 5, 1, A), (128, 0, 256, 6, 1, F | A),
    (64, 0, 512, 7, 1, A), (64, 0, 512, 8, 1, F | A), (64, 0, 512, 5, 2, A), (64, 0, 512, 6, 2, F | A), (128, 0, 256, 2, 2, 0),
    (128, 0, 256, 3, 2, F | A), (128, 1, 1024, 1, 1, A), (128, 1, 1024, 2, 1, F | A), (128, 2, 149, 1, 1, A),
    # one round (with the delta term, or in the adjoint: two) at any length
    (128, 0, 64, 1, 1, F | A), (64, 0, 128, 1, 1, F | A), (128, 0, 128, 1, 1, A), (128, 1, 148, 1, 1, F | A), (64, 1, 38, 1, 1, F | A)])
def test_short_sequences_of_many_pairs(V, delta, BH, NT, lean, bits):
    assert joint(ops.GATE_CHANNEL, V, delta, BH, NT, lean) == bits


@pytest.mark.parametrize("BH,NT,cut", [(1, 39, False), (1, 40, True), (2, 128, True), (4, 40, True), (4, 64, True), (5, 48, False), (8, 32, False), (5, 60, True)])
def test_few_long_sequences_with_the_channel_gate_are_cut(BH, NT, cut):
    assert ops.step_is_cut(ops.GATE_CHANNEL, True, NT, BH, B200_SMS) == cut
    assert not ops.step_is_cut(ops.GATE_CHANNEL, False, NT, BH, B200_SMS)
