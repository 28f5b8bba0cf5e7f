"""The record of the last plan is a plain dict."""

import json

from torch_neuronx_b200 import ops


def test_last_plan_is_a_dict():
    assert type(ops.last_plan) is dict
    json.dumps(ops.last_plan)
    assert ops.last_plan.copy() == ops.last_plan
