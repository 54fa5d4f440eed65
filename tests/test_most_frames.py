"""Frame count over task descriptors: an array of them and a list give the same
count, and the same refusal of times that are not finite (CPU)."""
import math

import pytest

from pincosimulator_gb300 import twmc


def tasks(spans, store=0):
    arr = (twmc.TaskDesc * len(spans))()
    for t, s in zip(arr, spans):
        t.t_start, t.t_end, t.store_initial = 0.5, 0.5 + s, store
    return arr


def outcome(t, dt):
    try:
        return twmc._most_frames(t, dt)
    except (ValueError, OverflowError) as e:
        return type(e)


@pytest.mark.parametrize("store", [0, 1])
@pytest.mark.parametrize("spans", [
    [1.0], [1.0, 2.0, 0.3], [0.05, 0.15, 0.25], [-3.0, -1.0], [0.0], [1e6, 1e-9], [1e300, 1.0],
    [math.nan], [1.0, math.nan], [math.nan, 1.0], [math.inf], [1.0, math.inf], [-math.inf, 1.0], [math.nan, math.inf]])
def test_array_and_list_agree(spans, store):
    t = tasks(spans, store)
    assert outcome(t, 0.1) == outcome(list(t), 0.1)
