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


@pytest.mark.parametrize("rows,experts", [(1000, 3), (1000, 40), (40000, 1024)])
def test_prefix_that_runs_back_and_forth_stays_inside_the_maps(rows, experts, native):
    """0, R, 0, R, ...: every other group has all the rows, together many times what the maps hold.  Status 5, no map entry
    past the bound, and the functional GEMM on such groups computes the groups that were kept."""
    from moe_explore.routing_plan import device_status, plan_from_groups
    from moe_explore.triton_kernels.m_grouped_gemm import MGroupedGEMMParams, m_grouped_gemm

    groups = torch.tensor([0, rows] * ((experts + 1) // 2) + ([rows] if experts % 2 == 0 else []), dtype=torch.int32)[:experts + 1]
    bound = native.mtiles_bound(rows, experts)
    tiles = (rows + 127) // 128
    kept = min(bound // tiles, (experts + 1) // 2)
    assert (experts + 1) // 2 * tiles > bound   # what the maps would have to hold
    native.read_status(device_status(), reset=True)
    plan = plan_from_groups(groups.cuda(), rows)
    assert native.read_status(plan.status, reset=True) == 5
    assert plan.num_mtiles.tolist() == [kept * tiles, kept * ((tiles + 1) // 2), bound, 0]
    assert int(plan.pad_offsets.max()) == int(plan.pad_offsets[-1]) == kept * tiles * 128
    assert plan.mtile_expert[: kept * tiles].tolist() == [2 * (m // tiles) for m in range(kept * tiles)]
    assert int(plan.row_src.max()) < rows and int(plan.dst_row.max()) < plan.padded_rows
    assert int(plan.tile_pairs[bound + experts]) == kept * ((tiles + 1) // 2)
    x = torch.randn(rows, 64, device="cuda").bfloat16()
    w = torch.zeros(experts, 64, 72, device="cuda").bfloat16()
    out = m_grouped_gemm(x, MGroupedGEMMParams(w, groups.cuda(), torch.arange(rows, device="cuda"), True, True, rows, 1))
    torch.cuda.synchronize()
    assert not out.any() and native.read_status(device_status(), reset=True) == 5
