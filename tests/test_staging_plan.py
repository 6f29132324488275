"""CPU test: the cached pager plan of a layer follows the projections' own views."""
import types

import pytest
import torch


def _manager(tm, staging):
    man = staging.GroupedQGmapCPUStagingManager([], mode="bitmap")
    man.slot_tables = [{p: torch.zeros((4,), dtype=torch.int32) for p in ("gate", "down")}]
    for proj in staging.PROJECTIONS:
        host = {"q_gmap_sparse": torch.zeros((4, 2, 8), dtype=torch.int32)}
        view = tm._native.TrisProjView()
        view.out_features, view.output_scale = 8, 4096
        man.entries[(0, proj)] = types.SimpleNamespace(payload={"_tris_prepared": True, "_tris_view": view}, host=host, block_bytes={"q_gmap_sparse": 64})
        man.buffers[(0, proj, "q_gmap_sparse")] = torch.zeros((64,), dtype=torch.uint8)
    return man


@pytest.mark.parametrize("proj", ["gate", "up", "down"])
def test_plan_follows_a_view_that_is_rebuilt_or_edited(proj):
    import trismoe_b200 as tm
    from trismoe_b200 import staging

    man = _manager(tm, staging)
    launches, views = man._plan(0, 0)
    again = man._plan(0, 0)
    assert again[0] is launches and again[1] is views and views[proj].output_scale == 4096
    payload = man.entries[(0, proj)].payload
    payload["_tris_view"].output_scale = 8192  # in place
    assert man._plan(0, 0)[1][proj].output_scale == 8192
    # rebuilt until an address comes back that an earlier, freed view had
    seen = {id(payload["_tris_view"])}
    for i in range(1, 2000):
        payload["_tris_view"] = None
        view = tm._native.TrisProjView()
        view.out_features, view.output_scale = 8, 4096 * (2 + i)
        payload["_tris_view"] = view
        assert man._plan(0, 0)[1][proj].output_scale == 4096 * (2 + i)
        if id(view) in seen:
            break
        seen.add(id(view))
    else:
        pytest.skip("no address was used twice")
