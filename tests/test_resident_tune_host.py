"""The tunings a context gives queries whose caller names none (no GPU)."""
import pytest

from gpudbmetalcodegen_b200 import engine


@pytest.mark.parametrize("rows", [0, 1, (1 << 25) - 1, 1 << 25, 120_000_000])
def test_every_resident_tuning_plans_and_compiles(rows):
    for name in engine.templates():
        spec = f"template={name}" + (";table=dim;col=b_key" if name == "colmax" else "")
        tune = engine.resident_tune(spec, rows)
        q = engine.Query(spec, tune)
        assert "phase 0" in q.plan
        assert all(kv in q.plan for kv in tune.split(";") if kv)


def test_the_streaming_sum_changes_form_at_two_to_the_25_rows():
    assert engine.resident_tune("template=q6", (1 << 25) - 1) != engine.resident_tune("template=q6", 1 << 25)
    assert engine.resident_tune("template=q6", 0) == engine.resident_tune("template=q6", 1 << 25)


def test_unknown_specs_have_no_tuning():
    assert engine.resident_tune("template=nope") == "" and engine.resident_tune("garbage") == ""
