"""The configuration that the autotuner picks for the radix path, run and held
against the oracle at a size that a default plan joins directly."""
import numpy as np
import pytest
import torch

import oracle
from pageflow_b200 import datagen
from pageflow_b200.join_aggregate import JoinAggregate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shrink", [200, 2000])
def test_the_tuned_radix_configuration_matches_the_oracle(tmp_path, monkeypatch, shrink):
    monkeypatch.setenv("PAGEFLOW_TUNE_CACHE", str(tmp_path / "tune.json"))
    for v in ("PF_JOIN_PATH", "PF_SJ_FP", "PF_SJ_TARGET", "PF_COUNTED"):
        monkeypatch.delenv(v, raising=False)
    w = datagen.scaled(datagen.SCALE, 1 / shrink)
    cols = [*datagen.gen_build(w, "cuda"), *datagen.gen_probe(w, "cuda")]
    s, c, matched, _ = oracle.join_aggregate(*[t.cpu().numpy() for t in cols], 100, 0, w.n_groups,
                                             B=16)
    here = np.nonzero(c)[0]

    def check(plan):
        keys, sums, counts = plan.run(*cols)
        assert np.array_equal(keys.cpu().numpy(), here)
        assert np.array_equal(sums.cpu().numpy(), s[here])
        assert np.array_equal(counts.cpu().numpy(), c[here])
        assert plan.read_stats().matched == matched

    for cached in (False, True):
        plan = JoinAggregate(w.n_build, w.n_probe, 0, w.n_groups, "cuda")
        assert plan.autotune and plan.direct
        plan.direct = False
        check(plan)
        assert plan.tuning.cached == cached
        t = plan.tuning.choice
        assert plan.B == t.B and plan.knobs.table == t.table and plan.knobs.sub_rows == t.sub_rows
    check(JoinAggregate(w.n_build, w.n_probe, 0, w.n_groups, "cuda", B=t.B,
                        knobs=dict(path=0, table=t.table, sub_rows=t.sub_rows, counted=t.counted)))
