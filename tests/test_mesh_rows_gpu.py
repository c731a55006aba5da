"""The icosphere's vertices, neighbour rows and edge lengths made directly, bit for bit against the general functions
(adjacency of its triangles) and the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 7, 33, 64, 129])
def test_rows_equal_the_adjacency_of_the_triangles(k):
    import torch
    from nixis_gb300 import mesh
    m = mesh.PlanetMesh(k)
    xyz, tris = mesh.icosphere(k)
    nbr = mesh.sort_adjacency(mesh.build_adjacency(tris))
    assert torch.equal(m.xyz.view(torch.int64), xyz.view(torch.int64))
    assert torch.equal(m.nbr, nbr)
    edge, err = mesh.edge_lengths(xyz, nbr)
    assert int(err.item()) == 0 and torch.equal(m.edge, edge)


@pytest.mark.parametrize("k", [257, 640])
def test_large_meshes_equal_the_oracle(k):
    from nixis_gb300 import mesh
    m = mesh.PlanetMesh(k)
    pts, tris = O.icosphere(k)
    adj = O.build_adjacency(tris)
    O.sort_adjacency(adj)
    assert np.array_equal(m.xyz.cpu().numpy().view(np.uint64), pts.view(np.uint64))
    assert np.array_equal(m.nbr.cpu().numpy(), adj)
    e = pts[adj.clip(0)] - pts[:, None, :]
    d = np.sqrt((e[..., 0] * e[..., 0] + e[..., 1] * e[..., 1]) + e[..., 2] * e[..., 2]) * (adj >= 0)
    hi = d.astype(np.float32)
    got = m.edge.cpu().numpy()
    assert np.array_equal(got[..., 0], hi) and np.array_equal(got[..., 1], (d - hi).astype(np.float32))


def test_scaled_and_shuffled_vertices_have_exact_lengths():
    """Edge lengths of radii and orders that no icosphere here has: the binary64 lengths' pairs exactly."""
    import torch
    from nixis_gb300 import mesh
    rng = np.random.default_rng(4)
    m = mesh.PlanetMesh(24)
    for radius in (6378100.0, 1e-7, 3e11, 1e25):
        perm = torch.from_numpy(rng.permutation(m.n)).cuda()
        inv = torch.empty_like(perm)
        inv[perm] = torch.arange(m.n, device="cuda")
        xyz = (m.xyz * radius)[perm]
        nbr = torch.where(m.nbr[perm] >= 0, inv[m.nbr[perm].clamp(min=0).long()].int(), m.nbr[perm]).int()
        e = xyz[nbr.clamp(min=0).long()] - xyz[:, None, :]
        d = torch.sqrt((e[..., 0] * e[..., 0] + e[..., 1] * e[..., 1]) + e[..., 2] * e[..., 2]) * (nbr >= 0)
        edge, _ = mesh.edge_lengths(xyz, nbr)
        hi = d.float()
        assert torch.equal(edge[..., 0], hi) and torch.equal(edge[..., 1], (d - hi.double()).float())


@pytest.mark.parametrize("k", [2, 3, 17, 64])
def test_edge_rows_of_any_alignment(k):
    """Rows 8 bytes off a 16-byte boundary: the same pairs, nothing beside them."""
    import torch
    from nixis_gb300 import _dev, mesh
    from nixis_gb300._lib import call
    m = mesh.PlanetMesh(k)
    buf = torch.full((m.edge.numel() + 4,), 7.0, dtype=torch.float32, device="cuda")
    call("nx_icosphere_edges", k, _dev.ptr(m.xyz), _dev.ptr(m.nbr), _dev.ptr(buf[2:]), None, _dev.stream_handle())
    assert torch.equal(buf[2:-2].view(m.edge.shape), m.edge)
    assert torch.equal(m.edge, mesh.edge_lengths(m.xyz, m.nbr)[0])
    assert (buf[:2] == 7.0).all() and (buf[-2:] == 7.0).all()


def test_the_longest_edge_counts_what_border_rows_leave_out(monkeypatch):
    """A far vertex of a face's border that only face-interior rows name, in the slots that compute no other distance."""
    import torch
    from nixis_gb300 import erosion, mesh
    monkeypatch.setattr(erosion, "BLOCKED_WORK", 1)
    k = 40
    m = mesh.PlanetMesh(k)
    inner = 12 + 30 * (k - 1)
    slots = {}
    for slot in range(6):
        for v in m.nbr[inner:, slot][m.nbr[inner:, slot] < inner].unique().tolist():
            slots.setdefault(v, set()).add(slot)
    v = next(v for v in sorted(slots) if v >= 12 and slots[v] <= {0, 1, 5})
    nbr, xyz = m.nbr.clone(), m.xyz.clone()
    nbr[:inner][nbr[:inner] == v] = -1
    nbr[v] = -1
    assert erosion.ErosionRun(xyz, nbr, iters=9).k == k
    xyz[v] *= 9.0                                # 8 from its neighbours: too long for blocked passes
    assert erosion.ErosionRun(xyz, nbr, iters=9).k is None
