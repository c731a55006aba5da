"""Tilings built from the grid and by searching the neighbour table give the same lists."""
import pytest

pytestmark = pytest.mark.gpu


def lists(tl, side, rings):
    """Per tile its counts, ids, neighbour indices and edge lengths (what lies beyond the counts is not written)."""
    import torch
    cnt = tl.counts.view(tl.ntiles, rings + 1)
    ids, group = tl.ids.view(tl.ntiles, tl.nmax), (tl.ntiles, tl.cmax // 32, 3, 32, -1)
    lnbr = tl.lnbr[: tl.ntiles * tl.cmax * 6].view(group).transpose(2, 3).reshape(tl.ntiles, tl.cmax, 6)
    ledge = tl.ledge.view(group).transpose(2, 3).reshape(tl.ntiles, tl.cmax, 12)
    n, c = cnt.sum(1), cnt.sum(1) - cnt[:, rings]
    seen = torch.arange(tl.nmax, device="cuda") < n[:, None]
    upd = torch.arange(tl.cmax, device="cuda") < c[:, None]
    return cnt, torch.where(seen, ids, -1), torch.where(upd[..., None], lnbr, 0), torch.where(upd[..., None], ledge, 0.0)


@pytest.mark.parametrize("k,side,rings", [(2, 2, 1), (9, 2, 8), (40, 8, 2), (47, 16, 4), (100, 32, 4), (131, 20, 5), (200, 33, 3)])
def test_grid_and_search_agree(k, side, rings):
    import torch
    from nixis_gb300 import mesh
    m = mesh.PlanetMesh(k)
    one = m.tiling(side, rings)
    # 8 bytes off the 16-byte boundary the build searches every tile
    buf = torch.empty(m.edge.numel() + 2, dtype=torch.float32, device="cuda")
    off = buf[2:].view(m.edge.shape)
    off.copy_(m.edge)
    assert off.data_ptr() % 16 == 8
    m2 = mesh.PlanetMesh(k)
    m2.edge = off
    two = m2.tiling(side, rings)
    assert (one.maxnl, one.maxc) == (two.maxnl, two.maxc)
    for a, b in zip(lists(one, side, rings), lists(two, side, rings)):
        assert torch.equal(a, b)
    members = torch.cat([i[:c] for i, c in zip(one.ids.view(one.ntiles, one.nmax), one.counts.view(one.ntiles, -1)[:, 0])])
    assert torch.equal(members.sort().values, torch.arange(m.n, device="cuda", dtype=torch.int32))


def test_another_neighbour_table_is_searched():
    import torch
    from nixis_gb300 import mesh
    m = mesh.PlanetMesh(60)
    v = m.n - 1200                                     # a face-interior vertex, its ring turned by one slot
    m.nbr[v] = m.nbr[v].roll(1)
    m.edge, _ = mesh.edge_lengths(m.xyz, m.nbr)
    tl = m.tiling(16, 4)
    assert tl.maxnl > 0
    cnt, ids, lnbr, ledge = lists(tl, 16, 4)
    t, q = torch.nonzero(ids == v, as_tuple=True)
    hit = q < (cnt.sum(1) - cnt[:, 4])[t]
    assert hit.any()
    for a, b in zip(t[hit].tolist(), q[hit].tolist()):
        assert torch.equal(ids[a][lnbr[a, b].long()], m.nbr[v]) and torch.equal(ledge[a, b], m.edge[v].reshape(-1))
