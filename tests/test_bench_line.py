"""The benchmark's JSON line stays short: the served leg reports its jobs by
kind, not one by one."""
import json

import bench


def test_served_jobs_by_kind():
    recs = [{"kind": "dam_break" if i % 3 else "ring_inlet", "cells": 1000 + i, "n_solid": 1 + i % 3,
             "steps": 500 + i, "tts_s": 0.1 * i} for i in range(200)]
    out = bench.served_by_kind(recs)
    assert out["dam_break"]["requests"] + out["ring_inlet"]["requests"] == 200
    assert sum(v["cells"] for v in out.values()) == sum(r["cells"] for r in recs)
    assert out["ring_inlet"]["p50_s"] <= out["ring_inlet"]["p99_s"] <= 0.1 * 199
    assert len(json.dumps(out)) < 500
