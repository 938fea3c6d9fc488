"""Routing metadata at the edges of the one-launch kernel: cluster sizes, ids per lane, and the row count above which the
chip-wide kernels take over.  Integer work, compared bit for bit."""
import pytest
import torch

from test_routing_gpu import _check_against_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,E", [(1, 1), (1, 1024), (31, 5), (1024, 7), (1025, 64), (2049, 1024), (16384, 60), (16385, 3),
                                    (65537, 256), (131072, 64), (131073, 64)])
def test_row_counts_at_the_edges(rows, E, native):
    g = torch.Generator().manual_seed(rows)
    idx = torch.randint(0, E, (rows, 1), generator=g)
    idx[rows // 2:] = torch.where(torch.rand(rows - rows // 2, 1, generator=g) < 0.5, E // 2, idx[rows // 2:])   # one hot expert
    plan = _check_against_oracle(idx, E)
    n = int(plan.num_mtiles[0])
    if rows <= native.ROUTE_ONE_LAUNCH_ROWS:
        assert bool((plan.row_src[n * 128:] == -1).all())   # the tail of the row map is marked as padding too


def test_no_rows(native):
    from moe_explore.routing_plan import build_routing_plan

    plan = build_routing_plan(torch.empty(0, 2, dtype=torch.int64, device="cuda"), 9, 2)
    assert plan.group_indices.tolist() == [0] * 10 and plan.num_mtiles.tolist()[:2] == [0, 0]
    assert bool((plan.row_src == -1).all())


def test_one_launch_up_to_the_largest_cluster_the_device_takes(native):
    """A whole B200 takes clusters of 16 CTAs for any number of experts (a device that does not: fewer rows per launch, and the
    chip-wide form beyond); the largest tables (155 KB of shared memory in every CTA) at the full row count."""
    lib = native.load()
    for E in (1, 256, 257, 1024):
        assert lib.moe_routing_one_launch_rows(E) == native.ROUTE_ONE_LAUNCH_ROWS
        assert native.routing_launches(131072, E) == 1 and native.routing_launches(131073, E) == native.ROUTE_CHIP_WIDE_LAUNCHES
    assert lib.moe_routing_one_launch_rows(0) == lib.moe_routing_one_launch_rows(5000) == 8192   # what one CTA holds
    g = torch.Generator().manual_seed(1)
    for rows in (131072, 131071, 65535, 8193):
        _check_against_oracle(torch.randint(0, 1024, (rows, 1), generator=g), 1024)
