"""The byte model of the sharded join's roofline (CPU)."""
from __future__ import annotations

import importlib.util
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def bench():
    spec = importlib.util.spec_from_file_location("bench", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


# 100 own rows split at 24 B when there are ranks to split over; 90 received
# rows joined at 8 B (direct) or histogram 8 + keys 12 + 8 + build/probe 4
@pytest.mark.parametrize("world,partitioned,expect", [(1, False, 8 * 90), (1, True, 32 * 90), (4, False, 2400 + 8 * 90),
                                                      (4, True, 2400 + 32 * 90)])
def test_sharded_bytes(world, partitioned, expect):
    assert bench().sharded_bytes(100, 90, world, partitioned)[0] == expect
