"""The autotuner measures the launch shapes of a kernel on scenes that launch it (no GPU):
plain scenes up to a size take the passes with a group of lanes per particle, which have
no shapes, so that what is measured there would be one kernel's noise."""
import json
import re
from pathlib import Path

import pytest

from particles4all_b200 import autotune

PACKAGE = Path(autotune.__file__).parent


def test_limit_is_the_library_s():
    assert autotune.GROUPED == int(re.search(r"kGroup8 = (\d+)", (PACKAGE / "csrc" / "api.cu").read_text()).group(1))


def test_buckets_and_committed_table():
    for bound, n in autotune.BUCKETS:
        assert n <= bound and (n > autotune.GROUPED) == (bound > autotune.GROUPED)
    table = json.loads(Path(autotune.DEFAULT_PATH).read_text())
    for name in ("lambda", "delta", "xsph_normals"):
        sizes = [int(n) for n, per in table["measured"].items() if not n.startswith("batch") and name in per]
        assert sizes and min(sizes) > autotune.GROUPED, name
        best = [table["measured"][str(n)][name]["best"] for n in sizes]
        assert [v for _, v in table["kernels"][name]] == best, name


def test_a_bucket_of_other_passes_is_refused(monkeypatch):
    monkeypatch.setattr(autotune, "_scene_sim", lambda n: pytest.fail("measured"))
    with pytest.raises(ValueError):
        autotune.tune(buckets=[(24_000, 12_000)], path=None, batch_buckets=None)
