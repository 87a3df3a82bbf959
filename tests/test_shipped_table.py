"""The shipped schedule table (CPU only): every entry's choice follows from the
times it carries. "ms" is its fastest candidate's; the choice is that candidate,
or the library's own (tile 0) with a "library_ms" within 2 % of it, or the one of
least geometric mean in the entry's "sustained" times."""
import json
import math

import pytest

from hb_hammerbench_b200 import autotune

TABLE = json.load(open(autotune.SHIPPED_PATH))


@pytest.mark.parametrize("key", sorted(TABLE))
def test_choice_follows_from_the_entry(key):
    e = TABLE[key]
    best = min((c for c in e["candidates"] if "ms" in c), key=lambda c: c["ms"])
    assert e["ms"] == best["ms"]
    if "sustained" in e:
        assert len(e["sustained_shapes"]) > 1
        for m, n, k in e["sustained_shapes"]:
            assert autotune.shape_key(m, n, k, key.split(":")[0]) == key
        mean = {}
        for s in e["sustained"]:
            assert len(s["ms"]) == len(e["sustained_shapes"])
            mean[json.dumps(s["config"], sort_keys=True)] = math.fsum(map(math.log, s["ms"]))
        assert min(mean, key=mean.get) == json.dumps(e["config"], sort_keys=True)
    elif e["config"] != best["config"]:
        assert e["config"]["tile"] == 0 and e["library_ms"] <= 1.02 * e["ms"]
