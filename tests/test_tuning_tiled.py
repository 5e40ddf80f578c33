"""Stored schedules of grids past one 128 x 128 tile: entries that count the adjoint's items in depths keep
their forward part only, entries of the tensor-core adjoint (layers) are used whole."""
import types

import pytest

from conftest import load_pkg


def _plan(pb, nx, ny, nsx, nsy, precision):
    f = pb._lib.Field(nx=nx, ny=ny, nz=64, n_sx=nsx, n_sy=nsy, n_layers=20)
    return types.SimpleNamespace(field=f, precision=precision, active_pairs=lambda: 900)


@pytest.mark.parametrize("nx, ny, nsx, nsy, precision, tiled", [
    (128, 128, 64, 64, 5, False), (129, 128, 64, 64, 5, True), (128, 129, 64, 64, 1, True),
    (300, 256, 64, 64, 4, True), (300, 257, 64, 64, 5, False), (200, 200, 65, 64, 5, False),
    (200, 200, 64, 65, 5, False), (200, 200, 61, 61, 0, False)])
def test_entries_in_depths_are_not_read_as_layers(monkeypatch, tmp_path, nx, ny, nsx, nsy, precision, tiled):
    pb = load_pkg()
    tun = pb.tuning
    monkeypatch.setenv("PBD_TUNING_CACHE", str(tmp_path / "tuning.json"))
    plan = _plan(pb, nx, ny, nsx, nsy, precision)
    old = f"loss_grad|{nx}x{ny}x64|{nsx}x{nsy}x20|p{precision}|a900"
    tun._store({old: {"schedule": [24, 8], "ms": 1.0}})
    assert tun.lookup(plan, "loss_grad") == ((24, 0) if tiled else (24, 8))
    tun._store({old: {"schedule": [24, 8], "ms": 1.0}, tun.geometry_key(plan, "loss_grad"): {"schedule": [12, 4], "ms": 1.0}})
    assert tun.lookup(plan, "loss_grad") == (12, 4)
    assert tun.lookup(plan, "forward") is None
