"""The tap loops and the Stokes I kernels where they can go wrong.

* Supports at the edges of the tap slots and of the gridder's tile (5, 7: two taps a lane; 9 ... 25:
  several rounds; 33: wider than the tile, laid down tap by tap), maps in order and shuffled (a
  stripe's records then do not fit one tile), float32 and FP64 sums, against the FP64 restatement:
  1e-6 relative RMS.  Terms carry some ten FP32 roundings (3e-7 at 2^-24 each, adding as their root);
  the grid's own FP32 additions are as many as a cell has terms, a few hundred here, also adding as
  the root of their number.
* The Stokes I kernels (no smearing, Jones terms as stored) against the general ones, which the same
  inputs reach when smearing is switched on with both of its factors off: visibilities and grids
  within 1e-6 relative RMS (another order of the same FP32 products), weight sums 1e-12 and Jones
  sums 1e-9 relative (the same FP32 weights, FP64 sums in another order), over correlations, maps,
  Jones channels, bands, channel counts on both sides of the shared per-channel sums, and lists of
  large blocks.
"""
import dataclasses

import numpy as np
import pytest
import torch

import cases
from ddfacet_b200 import device as D
from ddfacet_b200.autograd import PredictSetup, predict

pytestmark = pytest.mark.gpu


def _rms(a, b):
    return float((a - b).abs().pow(2).mean().sqrt() / b.abs().pow(2).mean().sqrt())


@pytest.mark.parametrize("sup", [5, 7, 9, 11, 15, 17, 23, 25, 33])
@pytest.mark.parametrize("kw", [dict(), dict(bda_mode=1, dphi=0.5), dict(stokes_ids=(1, 2, 3, 4))],
                         ids=["single", "bda", "iquv"])
def test_supports_against_fp64(sup, kw):
    c = cases.make_case(seed=41, nant=7, ntimes=12, nchan=9, ncorr=4, npix=243, cell_arcsec=4.0, nw=3, sup=sup,
                        flag_frac=0.1, nband=2, **kw)
    want = cases.run_fp64_grid(c)["grid"]
    vis = cases.run_fp64_degrid(c, want.astype(np.complex64))
    vs, fg, _ = cases._gpu_objs(c)
    pol = D.make_pol(c.corr_ids, c.stokes_ids)
    order = torch.randperm(vs.nblocks, generator=torch.Generator().manual_seed(3)).cuda()
    for v in (vs, vs.with_block_order(order)):
        for fp64 in (False, True):
            g = dataclasses.replace(fg, grid=torch.zeros_like(fg.grid), grid_acc=None)
            if fp64:
                g.with_fp64_accumulation()
            D.grid(v, [g], pol, batch=D.Batch.create())
            assert cases.rel_rms(g.grid.cpu().numpy(), want) < 1e-6
        m = dataclasses.replace(fg, grid=torch.from_numpy(want.astype(np.complex64)).cuda())
        out = dataclasses.replace(v, vis=torch.zeros_like(v.vis))
        D.degrid(out, [m], pol, batch=D.Batch.create())
        assert cases.rel_rms(out.vis.cpu().numpy(), vis) < 1e-6


FORMS = {
    "single": dict(), "single_wide": dict(sup=11), "bda1": dict(bda_mode=1, dphi=0.6),
    "bda2": dict(bda_mode=2, dphi=0.6), "large": dict(bda_mode=1, dphi=2.5),
}


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("ncorr,nchan,nch", [(4, 9, 0), (4, 37, 1), (4, 130, 5), (2, 9, 3), (2, 5, 0), (1, 9, 1)])
def test_stokes_i_kernels_against_general(form, ncorr, nchan, nch):
    args = dict(seed=43, nant=7, ntimes=10, nchan=nchan, ncorr=ncorr, npix=255, cell_arcsec=5.0, nw=3, flag_frac=0.15,
                nband=2, f_lo=1.0e9, f_hi=1.6e9)
    c = cases.make_case(**{**args, **FORMS[form]})
    if nch:
        cases.add_jones(c, nt=3, nd=3, nch=nch, mode=1)
    vs, fg, jd = cases._gpu_objs(c)
    if form == "large":
        vs = vs.with_large_blocks(16)
        assert vs.large_blocks is not None
    off = dataclasses.replace(vs, uvw_dt=torch.zeros_like(vs.uvw), dt=1.0, dnu=1.0, do_tsmear=0, do_fsmear=0)
    pol = D.make_pol(c.corr_ids, [1])
    gen = torch.Generator(device="cuda").manual_seed(5)
    model = torch.view_as_complex(torch.randn((*fg.grid.shape, 2), generator=gen, device="cuda"))
    for batch in (None, D.Batch.create()):
        got = []
        for v in (vs, off):
            z = {k: torch.zeros_like(getattr(fg, k)) for k in ("grid", "sumwt", "sumjones", "sumjones_chan")}
            g = dataclasses.replace(fg, **z).with_fp64_accumulation()
            D.grid(v, [g, dataclasses.replace(g, grid=torch.zeros_like(fg.grid), grid_acc=None, l0=0.003)], pol, jd,
                   batch=batch)
            d = dataclasses.replace(v, vis=torch.zeros_like(v.vis))
            m = dataclasses.replace(fg, grid=model)
            D.degrid(d, [m, dataclasses.replace(m, l0=0.003, cu=m.cu * 1.1)], pol, jd, batch=batch)
            got.append((g, d.vis))
        (g, d), (g0, d0) = got
        assert _rms(g.grid, g0.grid) < 1e-6
        assert _rms(d, d0) < 1e-6
        torch.testing.assert_close(g.sumwt, g0.sumwt, rtol=1e-12, atol=0)
        if nch:
            torch.testing.assert_close(g.sumjones, g0.sumjones, rtol=1e-9, atol=0)
            torch.testing.assert_close(g.sumjones_chan, g0.sumjones_chan, rtol=1e-9, atol=0)
    if nch:
        grads = []
        for v in (vs, off):
            kms = jd.kms.clone().requires_grad_()
            grid = model.clone().requires_grad_()
            p = predict(PredictSetup(vs=v, facets=[fg], pol=pol, jones=jd), [grid], kms)
            grads.append(torch.autograd.grad(p, [grid, kms], grad_outputs=vs.vis))
        for a, b in zip(*grads):
            assert _rms(a, b) < 1e-6


@pytest.mark.parametrize("kw", [dict(nchan=160, nband=150), dict(nchan=3000, nband=2, bda_mode=1, dphi=0.5)],
                         ids=["bands", "channels"])
def test_sums_that_fill_shared_memory(kw):
    """One facet's weight sums (150 bands, eight warps) or per-channel Jones sums (3000 channels) beside
    the wide tiles: more shared memory than two or three CTAs an SM leave each other."""
    c = cases.make_case(seed=47, nant=4, ntimes=4, ncorr=4, npix=125, cell_arcsec=5.0, nw=2, sup=11, **kw)
    cases.add_jones(c, nt=2, nd=2, mode=1)
    want = cases.run_fp64_grid(c)
    got = cases.run_gpu_grid(c, batched=True, fp64_acc=True)
    assert cases.rel_rms(got["grid"], want["grid"]) < 1e-6
    np.testing.assert_allclose(got["sumwt"], want["sumwt"], rtol=1e-12)
    np.testing.assert_allclose(got["sumjones_chan"], want["sumjones_chan"], rtol=1e-5)


@pytest.mark.parametrize("ncorr", [1, 4])
@pytest.mark.parametrize("ntimes", [19, 20, 39, 41])
def test_few_stripes_a_warp(ntimes, ncorr):
    """At one CTA an SM of 148: 1129 stripes (less than one a warp: spread), 1188 and 2316 (one or two:
    neighbours for each CTA), 2435 (chunks).  Every visibility is predicted once, as in a launch of all
    the CTAs that fit (another grouping of the same FP32 sums: 1e-6 relative RMS, and none left out)."""
    c = cases.make_case(seed=53, nant=20, ntimes=ntimes, nchan=10, ncorr=ncorr, npix=125, cell_arcsec=5.0, nw=2)
    cases.add_jones(c, nt=3, nd=2, mode=1)
    vs, fg, jd = cases._gpu_objs(c)
    gen = torch.Generator(device="cuda").manual_seed(7)
    model = torch.view_as_complex(torch.randn((*fg.grid.shape, 2), generator=gen, device="cuda"))
    out = []
    for ctas in (0, 1):
        d = dataclasses.replace(vs, vis=torch.zeros_like(vs.vis))
        D.degrid(d, [dataclasses.replace(fg, grid=model)], D.make_pol(c.corr_ids, [1]), jd,
                 batch=D.Batch.create(ctas_per_sm=ctas))
        out.append(d.vis)
    assert _rms(out[1], out[0]) < 1e-6
    assert torch.equal(out[1] != 0, out[0] != 0)
