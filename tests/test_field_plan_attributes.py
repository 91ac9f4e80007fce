"""What a caller could set on a plan can be set (CPU only)."""
from temgymcore_gb300.gaussian import FieldPlan


def test_the_method_can_be_set():
    plan = object.__new__(FieldPlan)
    plan.method = "direct"
    assert plan.method == "direct"
    plan.method = "fp64"
    assert plan.method == "fp64"
