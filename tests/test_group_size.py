"""Units per group when the caller leaves it to the library."""

from types import SimpleNamespace

import pytest

from gl_engine import api


@pytest.mark.parametrize("n, max_units, per_unit, want", [
    (1, None, 1 << 20, 1), (8, None, 1 << 30, 8),        # up to eight units: one group, whatever they need
    (9, None, 1 << 20, 9), (16, None, 1 << 27, 16),      # within the workspace limit: up to sixteen
    (40, None, 1 << 20, 16),
    (9, None, 1 << 28, 8), (16, None, (1 << 27) + 1, 8),  # beyond it: eight
    (40, 5, 1 << 30, 5), (3, 12, 1 << 20, 12),           # the caller's own choice stands
])
def test_units_per_group(monkeypatch, n, max_units, per_unit, want):
    monkeypatch.setattr(api, "get_plan", lambda max_units: SimpleNamespace(
        units=max_units, workspace_bytes=max_units * per_unit))
    assert api._plan_for(n, max_units).units == want
