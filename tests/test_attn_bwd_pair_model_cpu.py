"""Happens-before check of the CTA-pair attention backward's barrier protocol (host-side model, no GPU)."""

import pytest

from teletron_b200.utils.pair_pipeline_model import Variant, check


@pytest.mark.parametrize("chunks", [1, 2, 3, 4, 7])
def test_pair_protocol_orders_every_buffer(chunks):
    """One and two chunks (no S ahead, no dQ read-out before the next), and enough that every barrier has gone through both parities
    several times."""
    assert check(chunks) == []


@pytest.mark.parametrize("variant,needle", [
    (Variant(cluster_fence=False), "('dSown', 1, 0) at cluster scope"),
    (Variant(cluster_acquire=False), "('dSown', 1, 1) at cluster scope"),
    (Variant(wait_last_dq_read=False), "are not ordered on ('T1.4', 0)"),
    (Variant(wait_quad_read=False), "are not ordered on ('T1.1', 0)"),
    (Variant(wait_dq_before_ds=False), "are not ordered on ('out', 0, 0)"),
])
def test_model_sees_each_hazard(variant, needle):
    found = check(4, variant)
    assert any(needle in v for v in found), found[:5]
