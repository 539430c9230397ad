"""bench.py's accuracy keys: a comparison that did not run has no mismatch count and
is not among those that within_tolerance speaks for."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402


def _ran(mx=1e-6, mismatches=0):
    return {"pairs": 10, "cells": 100, "max": mx, "mean": mx / 2,
            "non_finite_mismatches": mismatches}


class _Engine:
    def batch(self, b):
        import oracle
        return oracle.batch_log10(b, oracle.SCALED)


def test_skipped_reference_is_not_counted(monkeypatch):
    import oracle
    monkeypatch.setattr(oracle, "ref_available", lambda: False)
    monkeypatch.setattr(bench, "ACCURACY_SAMPLES", [("C1", "tiny", 1.0, 1.0)])
    rows = bench.accuracy_per_config(_Engine())
    assert rows[0]["vs_reference"]["non_finite_mismatches"] is None
    assert rows[0]["vs_fp64_oracle"]["non_finite_mismatches"] == 0
    out, worst = bench.accuracy_fields(rows)
    assert out["C1_reference_non_finite_mismatches"] is None
    assert out["within_tolerance"] is True and out["within_tolerance_vs"] == "vs_fp64_oracle"
    assert worst == {"vs_fp64_oracle": 0.0, "vs_reference": None}


def test_tolerance_is_of_the_comparisons_that_ran():
    none = {"pairs": 0, "cells": 0, "max": None, "mean": None, "non_finite_mismatches": None}

    def fields(*rows):
        return bench.accuracy_fields([{"config": f"C{k}", "vs_fp64_oracle": o, "vs_reference": r}
                                      for k, (o, r) in enumerate(rows)])[0]

    both = fields((_ran(), _ran()))
    assert both["within_tolerance"] and both["within_tolerance_vs"] == "vs_fp64_oracle vs_reference"
    assert not fields((_ran(mismatches=1), none))["within_tolerance"]
    assert not fields((_ran(), _ran(mx=1.0)))["within_tolerance"]
    partly = fields((_ran(), _ran()), (_ran(), none))
    assert partly["within_tolerance"] and partly["within_tolerance_vs"] == "vs_fp64_oracle"
    assert not fields((_ran(), _ran(mismatches=2)), (_ran(), none))["within_tolerance"]
    assert fields((none, none))["within_tolerance"] is None
