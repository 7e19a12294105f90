"""Monitor npz I/O in the reference's format (beamz/devices/monitors.py:569-589: keys
fields, power_history, power_timestamps, monitor_info) and CustomMaterial rasterisation
on the host restatement, against files the reference itself wrote (tests/golden/)."""
import numpy as np
import pytest

import designs as D
from oracle import fdtd2d, raster2d


def _monitor_case(bz):
    d = D.wg_design(bz)
    t = D.time_axis(bz, 40)
    d += bz.GaussianSource(position=(1.0 * D.UM, 1.0 * D.UM), width=0.1 * D.UM, signal=D.gauss_signal(bz, t))
    mon = bz.Monitor(design=d, start=(1.6 * D.UM, 0.6 * D.UM), end=(1.6 * D.UM, 1.4 * D.UM), name="m",
                     record_interval=2)
    d += mon
    return d, t, mon


def test_load_reference_saved_monitor(bz, tmp_path):
    """A file written by the reference's Monitor.save_data loads into this Monitor, holds
    the oracle's records of the same run, and survives a save/load round trip with the
    same keys."""
    d, t, mon = _monitor_case(bz)
    mon.load_data(str(D.HERE / "monitor_saved.npz"))
    assert set(mon.fields) == {"Ez", "Hx", "Hy", "t"} and len(mon.fields["Ez"]) == 20
    eps, sig = raster2d.rasterize(d, D.RES)
    ref = fdtd2d.run(eps, sig, D.RES, D.RES, t[1] - t[0], len(t), d.sources, [mon], record=True)
    rec = ref["records"][0]
    for k in ("Ez", "Hx", "Hy"):
        np.testing.assert_array_equal(np.array(mon.fields[k]), rec[k])
    np.testing.assert_array_equal(np.array(mon.fields["t"]), rec["t"])
    np.testing.assert_array_equal(np.array(mon.power_history), rec["power"])
    out = tmp_path / "again.npz"
    mon.save_data(str(out))
    a = np.load(out, allow_pickle=True)
    assert sorted(a.files) == ["fields", "monitor_info", "power_history", "power_timestamps"]
    assert a["monitor_info"].item() == {"type": "line", "is_3d": False}
    for k in ("Ez", "Hx", "Hy", "t"):
        np.testing.assert_array_equal(np.array(a["fields"].item()[k]), np.array(mon.fields[k]))
    np.testing.assert_array_equal(a["power_history"], np.array(mon.power_history))
    with pytest.raises(ValueError):
        mon.save_data(str(tmp_path / "x.h5"), format="hdf5")


def test_custom_material_raster_oracle_matches_reference(bz, golden):
    g = golden("raster_custom")
    eps, mu, sig = raster2d.rasterize_all(D.raster_custom(bz), D.RES)
    np.testing.assert_array_equal(eps, g["eps"])
    np.testing.assert_array_equal(mu, g["mu"])
    np.testing.assert_array_equal(sig, g["sigma"])
    assert len(np.unique(g["eps"])) > 50  # the functions and the grid really vary


class _RecordingEngine:
    """Stand-in for the 2D engine after `step_index` steps: point p of the row of step n
    holds n + p / 10 for Ez, 100 more for Hx, 200 more for Hy. ``drained``: rows have left
    the device before the end, as with a full record buffer."""
    n_comp, d2h_bytes = 1, 0

    def __init__(self, monitors, drained):
        from types import SimpleNamespace

        self.step_index, self._taken, self._drained = 0, 0, drained
        self.mp = SimpleNamespace(monitors=monitors, slices=[slice(0, 3)] * len(monitors), valid=[True] * len(monitors))

    def _rows(self):
        n = np.arange(self._taken, self.step_index, dtype=float)[:, None]
        self._taken = self.step_index
        ez = n + np.arange(3) / 10.0
        return np.stack([ez, ez + 100.0, ez + 200.0], axis=-1)[:, None, None]  # [steps][design][comp][points][3]

    def take_records_device(self):
        import torch

        return None if self._drained or self._taken == self.step_index else torch.as_tensor(self._rows())

    def take_records(self):
        return self._rows()

    def check_divergence(self):
        pass

    def dft_fields(self):
        return None


@pytest.mark.parametrize("drained", [False, True])
@pytest.mark.parametrize("interval", [1, 3])
@pytest.mark.parametrize("parts", [(20,), (10, 10), (4, 5, 11), (7, 0, 13), (1, 1, 18)])
def test_finalising_between_steps_keeps_rows_and_times_together(bz, monkeypatch, parts, interval, drained):
    """A run that is finalised, continued and finalised again hands its monitors every row
    once, at its own step's time, as one finalise at the end does."""
    from beamz_b200.simulation import fdtd

    monkeypatch.setattr(fdtd, "to_host", lambda t: t.numpy())
    sim = fdtd.FDTD.__new__(fdtd.FDTD)
    mon = bz.Monitor(start=(0.0, 0.0), end=(0.0, 1e-6), record_interval=interval)
    sim.monitors, sim.results, sim.accumulate_power, sim.dt = [mon], {}, False, 0.25
    sim.engine = _RecordingEngine([mon], drained)
    for n in parts:
        sim.engine.step_index += n
        sim.finalize_simulation()
    steps = np.arange(20)[interval - 1::interval]
    ez = steps[:, None] + np.arange(3) / 10.0
    np.testing.assert_array_equal(np.array(mon.fields["Ez"]), ez)
    np.testing.assert_array_equal(np.array(mon.fields["Hx"]), ez + 100.0)
    np.testing.assert_array_equal(np.array(mon.fields["Hy"]), ez + 200.0)
    np.testing.assert_array_equal(np.array(mon.fields["t"]), steps * 0.25)
    np.testing.assert_array_equal(np.array(mon.power_timestamps), steps * 0.25)
    mag = ez * np.sqrt((ez + 200.0) ** 2 + (ez + 100.0) ** 2)
    np.testing.assert_allclose(np.array(mon.power_history), mag.sum(axis=1), rtol=1e-13)
    np.testing.assert_allclose(mon.power_accumulated, mag.sum(axis=0), rtol=1e-13)
    assert mon.power_accumulation_count == len(steps) and mon.last_record_step == steps[-1]


@pytest.mark.parametrize("limit,pinned", [(2 * 3 * 3 * 8, True), (2 * 3 * 3 * 8 - 1, False)])
def test_page_locked_memory_takes_records_up_to_its_limit(bz, monkeypatch, limit, pinned):
    """Samples above PINNED_RECORD_BYTES a monitor reach it through pageable memory."""
    from beamz_b200.simulation import fdtd

    calls = []
    monkeypatch.setattr(fdtd, "to_host", lambda t: calls.append(t.nbytes) or t.numpy())
    monkeypatch.setattr(fdtd, "PINNED_RECORD_BYTES", limit)
    sim = fdtd.FDTD.__new__(fdtd.FDTD)
    mon = bz.Monitor(start=(0.0, 0.0), end=(0.0, 1e-6))
    sim.monitors, sim.results, sim.accumulate_power, sim.dt = [mon], {}, False, 0.25
    sim.engine = _RecordingEngine([mon], False)
    sim.engine.step_index = 2
    sim.finalize_simulation()
    assert bool(calls) == pinned
    np.testing.assert_array_equal(np.array(mon.fields["Hy"]), np.arange(2)[:, None] + np.arange(3) / 10.0 + 200.0)
