"""Blocked passes: state rows off a 32-byte boundary, every pass length, every variant that shares the tables' layout."""
import pytest

pytestmark = pytest.mark.gpu


def run(m, h, iters, cfg, shift):
    """Heights, water and sediment after `iters` iterations; state rows `shift` floats off a 512-byte boundary."""
    import torch
    from nixis_gb300 import autotune, erosion
    was = autotune.current()
    try:
        if cfg is not None:
            autotune.use(cfg)
        r = erosion.ErosionRun(m.xyz, m.nbr, m.edge, iters=iters)
        r.k = m.k
        for name in ("st", "st_tmp"):
            t = getattr(r, name)
            setattr(r, name, torch.zeros(t.numel() + 8, dtype=t.dtype, device="cuda")[shift:shift + t.numel()].view(t.shape))
        r.load(h)
        if cfg is None:
            r.steps(iters, rain=0.01)
        else:
            assert r.blocked(iters, 0.01)
        out = [torch.empty(m.n, dtype=torch.float64, device="cuda") for _ in range(3)]
        r.store(*out)
        return out
    finally:
        autotune.use(was)


@pytest.mark.parametrize("iters", [1, 4, 5, 7, 16, 33])
@pytest.mark.parametrize("shift", [0, 4])
def test_rows_of_any_alignment(shift, iters):
    import torch
    from nixis_gb300 import autotune, mesh
    m = mesh.PlanetMesh(67)
    g = torch.Generator().manual_seed(iters)
    h = torch.rand(m.n, dtype=torch.float64, generator=g).cuda() * 100.0
    for a, b in zip(run(m, h, iters, None, 0), run(m, h, iters, autotune.current(), shift)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("side, rings, threads, variant", [(32, 4, 384, 4), (16, 2, 256, 0), (20, 3, 384, 1), (24, 8, 512, 0), (33, 1, 320, 4)])
def test_rows_of_any_order(side, rings, threads, variant):
    import torch
    from nixis_gb300 import autotune, mesh
    m = mesh.PlanetMesh(90)
    h = torch.rand(m.n, dtype=torch.float64, generator=torch.Generator().manual_seed(side)).cuda()
    cfg = autotune.TbConfig(side, rings, threads, variant)
    for a, b in zip(run(m, h, 13, None, 0), run(m, h, 13, cfg, 0)):
        assert torch.equal(a, b)


def test_passes_of_another_setting_are_refused():
    """The buffer a state starts in follows from the rings, so a run for other rings than the setting's does nothing."""
    import ctypes
    import torch
    from nixis_gb300 import _dev, _lib, autotune, erosion, mesh
    m = mesh.PlanetMesh(40)
    tb = autotune.current()
    tl = m.tiling(tb.tile_side, tb.rings)
    r = erosion.ErosionRun(m.xyz, m.nbr, m.edge)
    r.load(torch.rand(m.n, dtype=torch.float64, device="cuda"))
    was = r.st.clone()
    autotune.apply(tb)
    d = _lib.ErosionPlanet(0, m.n, m.nbr.data_ptr(), m.edge.data_ptr(), 7, 0.0, 0, 0, tl.dev.data_ptr(), tl.ntiles, tl.maxnl, tl.maxc)
    ws = torch.zeros(int(_lib.lib().nx_erosion_workspace_size(max(m.n, 256 * tl.ntiles), 1)), dtype=torch.uint8, device="cuda")
    for rings in (tb.rings + 1, 0):
        with pytest.raises(_lib.NxError):
            _lib.call("nx_erosion_run", _dev.ptr(r.planet), ctypes.byref(d), 1, rings, _dev.ptr(r.st), _dev.ptr(r.st_tmp), _dev.ptr(ws),
                      ws.numel(), _dev.stream_handle())
    assert torch.equal(r.st, was)


@pytest.mark.parametrize("turned", [False, True])
def test_a_run_on_its_own_stream_reads_its_own_checks(turned, monkeypatch):
    """The table's comparison and the edges' flag are read behind the run's kernels, which a busy stream delays."""
    import torch
    from nixis_gb300 import erosion, mesh
    monkeypatch.setattr(erosion, "BLOCKED_WORK", 1)
    m = mesh.PlanetMesh(50)
    nbr = m.nbr.clone()
    if turned:
        nbr[-900] = nbr[-900].roll(1)
    h = torch.rand(m.n, dtype=torch.float64, generator=torch.Generator().manual_seed(1)).cuda()
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    out = []
    for stream in (None, s):
        if stream is not None:
            with torch.cuda.stream(stream):
                torch.cuda._sleep(20_000_000)
        r = erosion.ErosionRun(m.xyz, nbr, stream=stream, iters=9)
        assert (r.k is None) == turned
        torch.cuda.synchronize()
        r.load(h)
        torch.cuda.synchronize()
        assert r.blocked(9, 0.01) != turned
        if turned:
            r.steps(9, rain=0.01)
        assert r.error() == 0
        torch.cuda.synchronize()
        out.append(torch.empty_like(h))
        r.store(out[-1])
        torch.cuda.synchronize()
    assert torch.equal(out[0], out[1])


def test_a_run_leaves_the_setting_of_others_alone(monkeypatch):
    """A drop-in run takes its setting with it: batches and servers on other threads go on with the one they applied."""
    import ctypes
    import torch
    from nixis_gb300 import _lib, autotune, erosion, mesh
    monkeypatch.setattr(erosion, "BLOCKED_WORK", 1)
    m = mesh.PlanetMesh(50)
    h = torch.rand(m.n, dtype=torch.float64, generator=torch.Generator().manual_seed(4)).cuda()
    was = autotune.current()
    run = erosion.ErosionRun(m.xyz, m.nbr, iters=9).load(h)
    try:
        autotune.apply(autotune.TbConfig(16, 2, 256, 0))
        assert run.blocked(9, erosion.RAIN)
        assert _lib.lib().nx_erosion_npass(8) == 4
    finally:
        autotune.apply(was)
    got = torch.empty_like(h)
    run.store(got)
    one = erosion.ErosionRun(m.xyz, m.nbr).load(h)
    one.steps(9, rain=erosion.RAIN)
    want = torch.empty_like(h)
    one.store(want)
    assert run.error() == 0 and torch.equal(got, want)
    d = _lib.ErosionPlanet()
    for rings, threads, variant in ((0, 256, 0), (9, 256, 0), (4, 384, 0), (4, 256, 7)):
        with pytest.raises(_lib.NxError):
            _lib.call("nx_erosion_run_as", None, ctypes.byref(d), 1, rings, threads, variant, None, None, None, 0, None)
