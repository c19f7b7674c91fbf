"""Dispatch rules that speak of waves ask the device for its SM count."""
from __future__ import annotations

import pytest

from test_programmatic_loads import CSRC, source


@pytest.mark.parametrize("unit", ["ip_launch_t.cuh", "adjoint.cu"])
def test_wave_rules_ask_the_device(unit):
    text = source(CSRC / unit)
    assert "148" not in text and "device_sms()" in text
