"""Calls at the edges of what the kernels are launched with: many facets of several Stokes planes, facets
with an FP64 accumulator in the backward pass, values that are not finite, streams of the caller's,
coherent sums, and grids of more than 2^31 cells."""
import ctypes as C
import dataclasses

import numpy as np
import pytest
import torch

import cases
from ddfacet_b200 import _abi, bda, device as D

pytestmark = pytest.mark.gpu


def _rms(a, b):
    return float((a - b).abs().pow(2).mean().sqrt() / b.abs().pow(2).mean().sqrt())


def _randn(shape, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.view_as_complex(torch.randn((*shape, 2), generator=gen, device="cuda"))


@pytest.mark.parametrize("kw", [dict(), dict(bda_mode=1, dphi=0.6)], ids=["single", "bda"])
@pytest.mark.parametrize("stokes", [(1, 2, 3), (1, 2, 3, 4)], ids=["iqu", "iquv"])
@pytest.mark.parametrize("n", [117, 118, 121, 128])
def test_degrid_planes_times_facets(n, stokes, kw):
    """A launch of up to 128 facets with three or four planes: the descriptors and the gather's buffers
    together pass 48 KB of shared memory.  Against launches of eight facets: up to sixteen more
    roundings of a visibility, 3e-8 relative each, adding as their root -- 1e-6."""
    c = cases.make_case(seed=61, nant=6, ntimes=6, nchan=6, ncorr=4, npix=63, cell_arcsec=8.0, nw=2,
                        stokes_ids=stokes, **kw)
    vs, fg, _ = cases._gpu_objs(c)
    fs = [dataclasses.replace(fg, grid=_randn(fg.grid.shape, i), l0=1e-4 * i) for i in range(n)]
    pol = D.make_pol(c.corr_ids, c.stokes_ids)
    out = []
    for batch in (D.Batch.create(facets_per_pack=8), D.Batch.create(), None):
        v = dataclasses.replace(vs, vis=torch.zeros_like(vs.vis))
        D.degrid(v, fs, pol, batch=batch)
        out.append(v.vis)
    assert _rms(out[1], out[0]) < 1e-6
    assert _rms(out[2], out[0]) < 1e-6


ADJ = {"stokes_i": dict(), "iquv": dict(stokes_ids=(1, 2, 3, 4)), "bda": dict(bda_mode=1, dphi=0.6),
       "wide": dict(sup=11, stokes_ids=(1, 2))}


@pytest.mark.parametrize("form", list(ADJ))
def test_adjoint_leaves_the_accumulator_alone(form):
    """ddfg_degrid_adjoint adds to ``grid``; an FP64 accumulator belongs to the gridding calls."""
    c = cases.make_case(seed=62, nant=7, ntimes=8, nchan=8, ncorr=4, npix=127, cell_arcsec=5.0, nw=2, **ADJ[form])
    cases.add_jones(c, nt=2, nd=2, mode=1)
    vs, fg, jd = cases._gpu_objs(c)
    pol = D.make_pol(c.corr_ids, c.stokes_ids)
    lib, vss, js = _abi.lib(), vs.struct(), jd.struct()
    got = []
    for acc in (None, torch.zeros(fg.grid.shape, dtype=torch.complex128, device="cuda")):
        g = dataclasses.replace(fg, grid=torch.zeros_like(fg.grid))
        s = g.struct(degrid=True)
        s.grid_acc = None if acc is None else acc.data_ptr()
        _abi.check(lib.ddfg_degrid_adjoint(C.byref(vss), C.byref(js), C.byref(pol), C.byref(s), 1, D._stream_ptr()))
        got.append(g.grid)
    assert torch.count_nonzero(torch.view_as_real(acc)) == 0
    assert torch.count_nonzero(torch.view_as_real(got[0])) > 0
    assert _rms(got[1], got[0]) < 1e-6  # float32 additions in another order
