"""Saved tuning tables of an earlier tensor-core engine: their bit-plane settings
apply, their tensor-core settings, which count other units, do not."""
import json

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def ctx():
    from hammingdist_gb300 import abi

    c = abi.Context(0)
    yield c
    c.close()


def _table(**top):
    entries = [{"n_bucket": nb, "L_bucket": lb, "dtype": dt, "tile": 64, "stages": 4,
                "mma_band": 32, "mma_rows": 1}
               for nb in range(7) for lb in range(4) for dt in (1, 2)]
    return {"device": "NVIDIA GB300", **top, "mma_min_items": [7, 1, 1, 1], "entries": entries}


@pytest.mark.parametrize("top,mma", [({"sm_count": 152}, (16, 2, 48)),
                                     ({"sm_count": 152, "mma_engine": 1}, (16, 2, 48)),
                                     ({"sm_count": 152, "mma_engine": 2}, (32, 1, 7)),
                                     ({}, (32, 1, 7))])  # written by hand
def test_engine_of_a_table(ctx, tmp_path, top, mma):
    path = str(tmp_path / "t.json")
    with open(path, "w") as f:
        json.dump(_table(**top), f)
    ctx.tune_load(path)
    assert ctx.tune_lookup(300, 1000, np.uint8) == (64, 4)
    assert ctx.tune_lookup_mma(300, 1000, np.uint8) == mma


def test_saved_and_shipped_tables_are_of_this_engine(ctx, tmp_path):
    import hammingdist_gb300 as hd
    import os

    path = str(tmp_path / "t.json")
    ctx.tune_save(path)
    engine = json.load(open(path))["mma_engine"]
    shipped = os.path.join(os.path.dirname(hd.__file__), "tuning", "gb300.json")
    assert json.load(open(shipped))["mma_engine"] == engine
    ctx.tune_load(path)
