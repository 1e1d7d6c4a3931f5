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
