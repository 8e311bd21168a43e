"""The shard's rows are dealt to the expander CTAs in turn: few and many CTAs, shares of several slices, rows left over."""

import pytest
import torch

from tests.cases import ROUNDTRIP_CASES, Case
from tests.harness import assert_within_ulp, check_dispatch_records, expected_combine, run_round_trip

# one CTA lists 2048 rows of its share at a time; senders with one CTA take tokens two at a time, also the last odd one
CASES = [c for c in ROUNDTRIP_CASES if c.name in ("rt_softmax_wide", "rt_zipf", "rt_single_expert")] + [
    Case("several_slices", S=1301, K=3, epn=4, H=64, num_sms=1, B=2, token_padding=32, routing="zipf"),
]


@pytest.mark.gpu
@pytest.mark.parametrize("ctas", [1, 3, 140])
@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
def test_round_trip_with_so_many_expander_ctas(case, ctas, monkeypatch):
    monkeypatch.setenv("MOONEP_NUM_SMS_DEDUP", str(ctas))
    R = 2
    recs = run_round_trip(case, R, "cuda")
    _, dst_pos, _, _ = check_dispatch_records(case, R, recs)
    want = expected_combine(case, R, recs, dst_pos)
    for r in range(R):
        assert_within_ulp(recs[r]["out"], want[r], max_ulps=1, what=f"rank {r} combine")
        assert torch.equal(recs[r]["weights_back"], recs[r]["w"])
