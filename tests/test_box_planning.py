"""Planning of copies of many small blocks: boxes are not planned where they would not be launched (a copy
of fewer than about a million elements in boxes beside blocks that go by tiles or units)."""
import numpy as np

from yastn_gb300 import _plans as P


def _plan(shapes, order):
    tasks, at = [], 0
    for shape in shapes:
        st = P.row_major_strides(shape)
        dims = [shape[o] for o in order]
        tasks.append((at, at, dims, [st[o] for o in order], P.row_major_strides(dims)))
        at += int(np.prod(shape))
    return P.CopyPlan(tasks, at, at)


def test_no_boxes_are_planned_in_vain(monkeypatch):
    calls, task = [], P._box_task
    monkeypatch.setattr(P, '_box_task', lambda *a: calls.append(1) or task(*a))
    small = [(5, 6, 5, 7)] * 300
    plan = _plan(small + [(5, 6, 5, 2)], (3, 2, 1, 0))  # the last one goes unit by unit
    tasks, items, boxes, *_ = plan.packed_with_boxes(True, 8)
    assert len(tasks) == 301 and len(boxes) == 0 and not calls
    # alone they all go by boxes, as do those of a large copy beside others
    plan = _plan(small, (3, 2, 1, 0))
    assert len(plan.packed_with_boxes(True, 8)[2]) == 300
    plan = _plan([(15, 14, 13, 13, 12)] * 3 + [(5, 6, 5, 7, 2)], (4, 3, 2, 1, 0))
    tasks, items, boxes, *_ = plan.packed_with_boxes(True, 8)
    assert len(tasks) == 1 and len(boxes) == 3
