"""The one-launch backward regression loop against one launch per date."""
from __future__ import annotations

from dataclasses import replace

import pytest
import torch

pytestmark = pytest.mark.gpu


# drop: every date's last basis functions left out, so that no date has a
# table the kernels know
@pytest.mark.parametrize("model,P,drop", [("c2", 1, 0), ("c2", 31, 0), ("c2", 4099, 0),
                                          ("c3", 513, 0), ("c3", 60001, 0), ("c3", 8192, 1),
                                          ("c2", 5001, 1), ("c5", 2049, 0), ("c5", 50003, 0)])
@pytest.mark.parametrize("normalise", [True, False])
def test_regression_loop_equals_dates(cuda, model, P, drop, normalise):
    """The one-launch backward loop against one launch per date (the sharded
    protocol with one shard): the same sums in the same order."""
    from useful_code_b200 import market as mk
    from useful_code_b200.pricer import Pipeline
    from useful_code_b200.sharded import regress_sharded

    cfg = mk.make_config(model)
    pipe = Pipeline(mk.build_market(replace(cfg, normalise=normalise)))
    pipe._nbasis[:] = (pipe._nbasis - drop).clip(1)
    ls = pipe.first_pass(P, 31)
    one = pipe.regress(ls)
    dates = regress_sharded(pipe, ls, P)
    # the dates divide their sums by the paths in another kernel: the same
    # FP64 operations, so equal bits
    assert torch.equal(one.beta, dates.beta)
    assert int(one.status) == int(dates.status)
    assert abs(float(one.price) - float(dates.price)) <= 1e-12 * abs(float(dates.price))
