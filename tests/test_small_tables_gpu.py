"""Host tables as kernel arguments, schedules by one native call, and results written straight into host arrays.

Everything here is copied or computed by the same operations as on the general path, so every comparison is exact."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from nixis_gb300 import _dev, _lib, climate, mesh, util  # noqa: E402

gpu = pytest.mark.gpu


@pytest.mark.parametrize("axial, year, days", [(23.44, 365, 365), (-7.5, 88.25, 1), (0, 3, 40), (97, -12.5, 700)])
def test_seasonal_tilts_are_the_reference_sums(axial, year, days):
    want = [climate.calculate_seasonal_tilt(axial, climate.day2deg(year, d)) for d in range(days)]
    assert climate.annual_schedule(axial, year, days, 24)[1] == want


@pytest.mark.parametrize("axial, year", [(np.float32(23.44), 365), (23.44, np.int64(12)), (23.44, 1e-300)])
def test_other_number_types_keep_pythons_arithmetic(axial, year):
    want = [climate.calculate_seasonal_tilt(axial, climate.day2deg(year, d)) for d in range(1)]
    assert climate.annual_schedule(axial, year, 1, 2)[1] == want
    with pytest.raises(ZeroDivisionError):
        climate.annual_schedule(23.44, 0, 2, 2)


@gpu
@pytest.mark.parametrize("off", [0, 1, 4])
@pytest.mark.parametrize("n", [0, 1, 3, 4, 255, 3999, 4000, 4001, 8000, 15999, 16000])
def test_upload_sizes_and_alignments(n, off):
    src = np.random.default_rng(n).integers(0, 256, n, np.uint8)
    want = src.copy()
    dst = torch.full((n + 16,), 77, dtype=torch.uint8, device="cuda")
    torch.cuda._sleep(1000)
    _lib.call("nx_upload", ctypes.c_void_p(dst.data_ptr() + off), ctypes.c_void_p(src.ctypes.data), n, _dev.stream_handle())
    src[:] = 0                                   # the bytes were taken by the call
    got = dst.cpu().numpy()
    assert np.array_equal(got[off:off + n], want)
    assert (got[:off] == 77).all() and (got[off + n:] == 77).all()
    with pytest.raises(_lib.NxError):
        _lib.call("nx_upload", ctypes.c_void_p(dst.data_ptr()), ctypes.c_void_p(got.ctypes.data), 16001, None)


@gpu
@pytest.mark.parametrize("n", [1999, 2000, 2001, 2500])
def test_arrays_around_the_upload_limit(n):
    a = np.random.default_rng(n).random(2 * n)[::2]          # strided
    b = a.copy()
    t = _dev.to_device(a, np.float64)
    a[:] = 0.0
    assert np.array_equal(t.cpu().numpy(), b)
    for out in (np.zeros(n), np.zeros(2 * n)[::2], np.zeros(n, np.float32), np.zeros(2 * n)[::-2]):
        _dev.to_host(out, t)
        assert np.array_equal(out, b.astype(out.dtype))
    ro = np.zeros(n)
    ro.flags.writeable = False
    with pytest.raises(ValueError):
        _dev.to_host(ro, t)


@gpu
@pytest.mark.parametrize("n_rot, n_tilt", [(24, 365), (7, 3), (0, 4), (1600, 400), (1601, 400)])
def test_schedules_by_arguments_and_by_table(n_rot, n_tilt):
    m = mesh.PlanetMesh(9)
    rot, tilt = [-180.0 + 360.0 / max(n_rot, 1) * i for i in range(n_rot)], list(np.linspace(-30.0, 31.0, n_tilt))
    tab, nre, pairs = climate._plan(rot, tilt)
    tdev = torch.from_numpy(tab).cuda()
    want = torch.empty(m.n, dtype=torch.float32, device="cuda")
    _lib.call("nx_insolation", _dev.ptr(m.xyz), m.n, 1.0, _dev.ptr(tdev), nre, pairs, n_tilt, _dev.ptr(want), 0,
              _dev.stream_handle())
    assert torch.equal(climate.insolation_sum(m.xyz, 1.0, rot, tilt), want)
    assert torch.equal(climate._sum(m.xyz, 1.0, rot, tilt, None, False, torch.cuda.current_stream(), 1361.0 / 77), want * (1361.0 / 77))
    out = want.clone()
    climate.insolation_sum(m.xyz, 1.0, rot, tilt, out=out, accumulate=True)
    assert torch.equal(out, want + want)


@gpu
def test_mapped_files_go_through_staging(tmp_path):
    """The same bytes from and into a memory-mapped file, also behind a plain view of it."""
    a = np.random.default_rng(1).random(9000)
    f = np.memmap(tmp_path / "x", np.float64, "w+", shape=a.shape)
    f[:] = a
    assert not _dev._in_memory(f) and not _dev._in_memory(np.asarray(f)[10:]) and _dev._in_memory(a[10:])
    for src in (f, np.asarray(f)):
        t = _dev.to_device(src, np.float64)
        assert np.array_equal(t.cpu().numpy(), a)
    out = np.memmap(tmp_path / "y", np.float64, "w+", shape=a.shape)
    _dev.to_host(out, t)
    assert np.array_equal(out, a)


@gpu
@pytest.mark.parametrize("busy", ["its own", "the caller's"])
@pytest.mark.parametrize("days, hours", [(2000, 24), (6, 2400), (300, 24)])
def test_a_schedule_on_another_stream(days, hours, busy):
    """Table, sums and their scaling are in the order of the stream that was given, whichever of the two is held back."""
    m = mesh.PlanetMesh(12)
    want = climate.annual_insolation(m.xyz, 1.0, days=days, hours=hours, mean_wm2=True)
    host = m.xyz.cpu().numpy()
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s if busy == "its own" else torch.cuda.current_stream()):
        torch.cuda._sleep(200_000_000)
    got = [climate.annual_insolation(v, 1.0, days=days, hours=hours, mean_wm2=True, stream=s) for v in (m.xyz, host)]
    s.synchronize()
    with torch.cuda.stream(s):
        kept = [g.clone() for g in got]
    torch.cuda.synchronize()
    assert torch.equal(kept[0], want) and torch.equal(kept[1], want)


@gpu
def test_bytes_of_a_mapping_go_through_staging(tmp_path):
    """Arrays made of a mapping's buffer, past the size of an upload, in both directions."""
    import mmap
    a = np.random.default_rng(1).random(9000)
    (tmp_path / "x").write_bytes(a.tobytes())
    with open(tmp_path / "x", "r+b") as f:
        mm = mmap.mmap(f.fileno(), 0)
    for src in (np.frombuffer(mm), np.asarray(memoryview(mm)).view(np.float64)):
        t = _dev.to_device(src, np.float64)
        assert np.array_equal(t.cpu().numpy(), a)
    _dev.to_host(np.frombuffer(mm), t + 1.0)
    assert np.array_equal(np.frombuffer(mm), a + 1.0)
    points, _ = util.create_mesh(10)             # (the library's own results need none)
    assert _dev._in_memory(points)


@gpu
def test_a_large_array_does_not_wait_for_a_busy_stream():
    a = np.random.default_rng(2).random(300_000)
    want = a.copy()
    for _ in range(2):                           # (the first makes the page-locked buffer)
        torch.cuda.synchronize()
        torch.cuda._sleep(400_000_000)
        t = _dev.to_device(a, np.float64)
        busy = not torch.cuda.current_stream().query()
    a[:] = 0.0
    assert busy
    assert np.array_equal(t.cpu().numpy(), want)


@gpu
def test_a_call_on_an_idle_stream_stages_nothing(monkeypatch):
    """Host fields of a drop-in erosion are copied before the run's own work is on the stream."""
    from nixis_gb300 import erosion
    points, cells = util.create_mesh(20)
    nbr = util.build_adjacency(cells)
    util.sort_adjacency(nbr)
    staged = []
    pin = torch.Tensor.pin_memory
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda t, *a: staged.append(t.shape) or pin(t, *a))
    torch.cuda.synchronize()
    height = points[:, 2] * 100.0
    erosion.erode_terrain3(points, nbr, height, num_iter=3)
    assert staged == []


@gpu
def test_the_question_whether_a_stream_is_idle_leaves_captures_whole():
    """Asked while another thread captures, of a busy stream, and of the captured one."""
    import threading
    idle = _lib.lib().nx_stream_idle
    x, got = torch.zeros(8, device="cuda"), []
    graph, s, busy = torch.cuda.CUDAGraph(), torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=s):
        x.add_(1.0)
        other = threading.Thread(target=lambda: got.append(idle(None)))
        other.start()
        other.join()
        got.append(idle(s.cuda_stream))
    assert got == [1, 0]
    graph.replay()
    torch.cuda.synchronize()
    assert x.eq(1.0).all()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(100_000_000)
    assert idle(busy.cuda_stream) == 0
    busy.synchronize()
    assert idle(busy.cuda_stream) == 1


@gpu
def test_the_handle_is_the_current_streams():
    s = torch.cuda.Stream()
    for _ in range(2):
        assert _dev.stream_handle().value == (torch.cuda.current_stream().cuda_stream or None)
        with torch.cuda.stream(s):
            assert _dev.stream_handle().value == s.cuda_stream
    assert _dev.stream_handle(s).value == s.cuda_stream
