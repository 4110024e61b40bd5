"""The oracle's restated profile defaults equal those the compiled reference
gave for the golden fixtures, and stand in for it where it is not built."""
import glob
import json
import os

import numpy as np
import pytest

from conftest import ROOT

GOLDEN = sorted(glob.glob(os.path.join(ROOT, "tests", "golden", "*.npz")))


@pytest.mark.parametrize("path", GOLDEN, ids=lambda p: os.path.basename(p))
def test_defaults_equal_golden(oracle_mod, path):
    prm = json.loads(str(np.load(path)["params"]))
    for key, wiener in (("basic", False), ("final", True)):
        want = prm[key]
        assert oracle_mod.stage_default(prm["profile"], wiener, want["sigma"]) == want


def test_golden_covers_every_profile():
    found = {json.loads(str(np.load(p)["params"]))["profile"] for p in GOLDEN}
    assert found == {"fast", "lc", "np", "high", "vn"}


def test_defaults_without_the_reference(oracle_mod, monkeypatch):
    monkeypatch.setattr(oracle_mod, "reference_available", lambda: False)
    got = oracle_mod.reference_stage_default("np", True, (17.0, 9.0, 4.0))
    assert got == oracle_mod.stage_default("np", True, (17.0, 9.0, 4.0))
