"""Choices by a device's SMs are by the current device's, with several devices of different sizes in a process."""
from types import SimpleNamespace

import torch


def test_every_device_has_its_own_count(monkeypatch):
    from oracle_engine_b200.csrc import ops, ops_tc
    now = [1]
    monkeypatch.setattr(torch.cuda, "current_device", lambda: now[0])
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: SimpleNamespace(multi_processor_count={1: 148, 2: 20}[d]))
    monkeypatch.setattr(ops, "_sms", {})
    seen = []
    for now[0] in (1, 2, 1):
        seen.append((ops.sm_count(), ops_tc.prompt_cluster(256, 1, 3, 8, 1)))
    assert seen == [(148, 2), (20, 1), (148, 2)]
