"""The tuner's cache key and candidates (no GPU)."""
import types

import pytest
import torch

from ddfacet_b200 import autotune, device as D


def _workload(**kw):
    vs = types.SimpleNamespace(nblocks=1000, vis=torch.zeros((10, 8, 4), dtype=torch.complex64), single_vis_blocks=1,
                               large_blocks=None, uvw_dt=kw.get("uvw_dt"))
    f = types.SimpleNamespace(grid=torch.zeros((1, 1, 5, 5)), cf=types.SimpleNamespace(max_support=7), grid_acc=None)
    pol = D.make_pol(kw.get("corr", [9, 10, 11, 12]), kw.get("stokes", [1]))
    jones = kw.get("jones", D.JonesData(mode=1, kms=torch.zeros(1), apply_amp=1, apply_phase=1))
    return vs, [f], pol, jones


OTHER = {
    "circular": dict(corr=[5, 6, 7, 8]), "stokes q": dict(stokes=[2]), "smearing": dict(uvw_dt=torch.zeros(1)),
    "no jones": dict(jones=None),
    "beam": dict(jones=D.JonesData(mode=1, kms=torch.zeros(1), beam=torch.zeros(1), apply_amp=1, apply_phase=1)),
    "interpolated": dict(jones=D.JonesData(mode=1, kms=torch.zeros(1), interp_mode=1, apply_amp=1, apply_phase=1)),
    "phases": dict(jones=D.JonesData(mode=1, kms=torch.zeros(1), apply_amp=0, apply_phase=1)),
}


@pytest.mark.parametrize("what", list(OTHER))
def test_key_tells_kernels_apart(what, monkeypatch):
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda d: "gpu")
    key = autotune.workload_key(*_workload())
    assert key == autotune.workload_key(*_workload())
    assert key != autotune.workload_key(*_workload(**OTHER[what]))


def test_key_tells_schedulers_apart(monkeypatch):
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda d: "gpu")
    key = autotune.workload_key(*_workload())
    monkeypatch.setattr(autotune, "SCHEDULE", autotune.SCHEDULE + 1)
    assert key != autotune.workload_key(*_workload())


@pytest.mark.parametrize("grid", [True, False])
@pytest.mark.parametrize("single,own", [(True, 64), (False, 16)])
def test_candidates_are_different_schedules(single, own, grid):
    """The library's own chunk (0) is 64 stripes for single visibilities and 16 for averaged blocks."""
    c = [(x["facets_per_pack"], x["stripes_per_item"] or own) for x in autotune.candidates(single, grid)]
    assert len(set(c)) == len(c) == 6
