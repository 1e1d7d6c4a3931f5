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


def _geometry(c, vs, fg, degrid=False):
    """D.block_geometry of a map of single visibilities as [nrow, nchan, 8]."""
    at = c.bda[2 + vs.nblocks:].reshape(-1, 3)
    out = np.zeros((c.nrow, c.nchan, 8), np.int32)
    out[at[:, 2], at[:, 0]] = D.block_geometry(vs, fg, degrid=degrid).cpu().numpy()
    return out


def test_gradients_of_values_that_are_not_finite():
    """Upstream gradients of NaN and Inf at visibilities that miss the facet (beyond wmax) take no part in
    the Jones gradient, in the Stokes I kernel as in the general one (reached with smearing switched on and
    both of its factors off)."""
    c = cases.make_case(seed=63, nant=7, ntimes=8, nchan=8, ncorr=4, npix=127, cell_arcsec=5.0, nw=3)
    cases.add_jones(c, nt=2, nd=2, mode=1)
    vs, fg, jd = cases._gpu_objs(c)
    fg.cf = dataclasses.replace(fg.cf, wmax=fg.cf.wmax * 0.4)
    fg = dataclasses.replace(fg, grid=_randn(fg.grid.shape, 3))
    pol = D.make_pol(c.corr_ids, [1])
    miss = torch.from_numpy(_geometry(c, vs, fg, degrid=True)[:, :, 0] != 1).cuda()
    at = torch.nonzero(miss)
    assert 0.05 * miss.numel() < at.shape[0] < 0.95 * miss.numel()
    good = vs.vis.clone()
    good[miss] = 0
    bad = good.clone()
    bad[at[::2, 0], at[::2, 1]] = complex(float("nan"), 0.0)
    bad[at[1::2, 0], at[1::2, 1]] = complex(float("inf"), float("-inf"))
    lib = _abi.lib()
    out = []
    for vis, smear in ((good, False), (bad, False), (bad, True)):
        v = dataclasses.replace(vs, vis=vis)
        if smear:
            v = dataclasses.replace(v, uvw_dt=torch.zeros_like(vs.uvw), dt=1.0, dnu=1.0, do_tsmear=0, do_fsmear=0)
        kms = torch.zeros_like(jd.kms)
        vss, js, s = v.struct(), jd.struct(), fg.struct(degrid=True)
        _abi.check(lib.ddfg_degrid_jones_grad(C.byref(vss), C.byref(js), C.byref(pol), C.byref(s), 1, kms.data_ptr(),
                                              D._stream_ptr()))
        out.append(kms)
    assert torch.isfinite(torch.view_as_real(out[0])).all()
    for k in out[1:]:
        assert torch.isfinite(torch.view_as_real(k)).all()
        assert _rms(k, out[0]) < 1e-6


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("kw", [dict(), dict(stokes_ids=(1, 2, 3, 4)), dict(sup=11)], ids=["i", "iquv", "wide"])
def test_gridding_values_that_are_not_finite(kw, fp64):
    """A NaN and an Inf reach the cells of their own footprints and no others; rows with NaN coordinates
    reach none."""
    c = cases.make_case(seed=64, nant=7, ntimes=10, nchan=8, ncorr=4, npix=127, cell_arcsec=5.0, nw=2, **kw)
    c.uvw = c.uvw.copy()
    c.uvw[5, 2] = np.nan
    c.uvw[9, 0] = np.nan
    vs, fg, _ = cases._gpu_objs(c)
    geo = _geometry(c, vs, fg)
    assert (geo[5, :, 0] != 1).all() and (geo[9, :, 0] != 1).all()
    pick = [(r, ch) for r, ch in ((40, 2), (90, 5)) if geo[r, ch, 0] == 1]
    assert len(pick) == 2
    vs.vis[pick[0]] = complex(float("nan"), 0.0)
    vs.vis[pick[1]] = complex(float("inf"), 0.0)
    want = np.ones((c.npix, c.npix), bool)
    for r, ch in pick:
        sup = int(fg.cf.sup[geo[r, ch, 2]])
        x, y = geo[r, ch, 3] - (sup - 1) // 2, geo[r, ch, 4] - (sup - 1) // 2
        want[y:y + sup, x:x + sup] = False
    g = dataclasses.replace(fg, grid=torch.zeros_like(fg.grid), grid_acc=None)
    if fp64:
        g.with_fp64_accumulation()
    D.grid(vs, [g], D.make_pol(c.corr_ids, c.stokes_ids), batch=D.Batch.create())
    ok = torch.isfinite(torch.view_as_real(g.grid)).all(-1).cpu().numpy()
    for p in range(c.npol):
        assert np.array_equal(ok[0, p], want)
    if fp64:
        assert torch.count_nonzero(torch.view_as_real(g.grid_acc)) == 0


def test_images_on_a_stream_of_the_callers():
    """The image is zeroed on the stream that adds to it, however busy the current one is."""
    from ddfacet_b200.facetmachine import FacetMachine

    fm = FacetMachine(300, 6.0, 2, np.linspace(1.3e9, 1.45e9, 4), nw=2, wmax=500.0)
    for i, f in enumerate(fm.facets):
        f.grid.sumwt.fill_(3.0)
        f.model.grid.copy_(_randn(f.model.grid.shape, 20 + i))
    grids = [_randn(f.grid.grid.shape, i) for i, f in enumerate(fm.facets)]
    grads = [f.model.grid for f in fm.facets]

    def images(stream):
        for f, g in zip(fm.facets, grids):
            f.grid.grid.copy_(g)
        torch.cuda.synchronize()
        if stream is not None:
            torch.cuda._sleep(200_000_000)  # a tenth of a second
        out = fm.facets_to_image(stream=stream), fm.image_to_facets_adjoint(grads, stream=stream)
        torch.cuda.synchronize()
        return out

    want = images(None)
    got = images(torch.cuda.Stream())
    for a, b in zip(got, want):
        assert torch.count_nonzero(b) > 0
        assert torch.equal(a, b)


@pytest.mark.parametrize("nch", [0, 1, 6])
def test_sums_of_stripes_with_one_band_and_two(nch):
    """96 channels in two bands of 48: of a row's three stripes the outer two add up in one lane and the
    middle one with atomics, to the same slots.  FP64 sums of FP32 weights: 1e-12, times FP32 Jones
    weights: 1e-6."""
    c = cases.make_case(seed=66, nant=10, ntimes=20, nchan=96, ncorr=4, npix=127, cell_arcsec=5.0, nw=2, nband=2,
                        flag_frac=0.05)
    if nch:
        cases.add_jones(c, nt=2, nd=2, mode=1, nch=nch)
    want = cases.run_fp64_grid(c)
    got = cases.run_gpu_grid(c, batched=True)
    np.testing.assert_allclose(got["sumwt"], want["sumwt"], rtol=1e-12)
    if nch:
        np.testing.assert_allclose(got["sumjones"], want["sumjones"], rtol=1e-6)
        np.testing.assert_allclose(got["sumjones_chan"], want["sumjones_chan"], rtol=1e-6)


def _coherent(nant, ntimes, **kw):
    c = cases.make_case(seed=65, nant=nant, ntimes=ntimes, nchan=32, ncorr=4, npix=127, cell_arcsec=5.0, nw=2, **kw)
    rng = np.random.default_rng(6)
    c.vis[:] = (1 + 1e-3 * rng.standard_normal(c.vis.shape[:2]))[:, :, None]
    return c


def _grid_error(c, vs, fg):
    g = dataclasses.replace(fg, grid=torch.zeros_like(fg.grid)).with_fp64_accumulation()
    D.grid(vs, [g], D.make_pol(c.corr_ids, c.stokes_ids), batch=D.Batch.create())
    return cases.rel_rms(g.grid.cpu().numpy(), cases.run_fp64_grid(c)["grid"])


def test_long_blocks_of_coherent_visibilities():
    """Blocks of 2048 visibilities that add up in phase, at the phase centre (the phasor is 1).  A sum in
    FP32 loses 6e-7 of it; one in FP64 leaves the FP32 roundings of the block's value, of its product
    with a tap and of the grid cell, 3e-8 each: 5e-8, with room to 1e-7."""
    c = _coherent(5, 64, bda_mode=1, dphi=50.0)
    vs, fg, _ = cases._gpu_objs(c)
    assert vs.nblocks == 10 and not vs.single_vis_blocks
    assert _grid_error(c, vs, fg) < 1e-7


@pytest.mark.parametrize("kw", [dict(sup=17), dict(sup=23), dict(sup=19, stokes_ids=(1, 2, 3, 4)),
                                dict(sup=7, stokes_ids=(1, 2, 3, 4), blocks=True),
                                dict(sup=11, stokes_ids=(1, 2), blocks=True), dict(sup=7, blocks=True)],
                         ids=["i17", "i23", "iquv19", "iquv_blocks", "iq11_blocks", "i_blocks"])
def test_runs_reach_the_accumulator_in_fp64(kw):
    """One baseline's 32 channels on one cell, FP64 sums: the products add up in FP64 where supports are
    wide or blocks averaged.  Of a cell's own value, RMS over the cells: the cell's rounding at the end
    2.6e-8, those of 32 products (3.5e-8 each, independent) and of the 32 values 6e-9 each: 2.8e-8, with
    room to 4e-8; a sum of 32 in FP32 has 8e-8."""
    kw = dict(kw)
    blocks = kw.pop("blocks", False)
    c = _coherent(2, 2 if blocks else 1, f_lo=1.4e9, f_hi=1.4001e9, **kw)
    if blocks:  # the second row in one block, which makes the map an averaged one; it is flagged
        blk = [[ch, ch + 1, 0] for ch in range(c.nchan)] + [[0, c.nchan, 1]]
        c.bda = np.concatenate([bda._header(len(blk)), [len(b) for b in blk], *blk]).astype(np.int32)
        c.flags[1] = True
    vs, fg, _ = cases._gpu_objs(c)
    assert bool(vs.single_vis_blocks) != blocks
    g = dataclasses.replace(fg, grid=torch.zeros_like(fg.grid)).with_fp64_accumulation()
    D.grid(vs, [g], D.make_pol(c.corr_ids, c.stokes_ids), batch=D.Batch.create())
    want = cases.run_fp64_grid(c)["grid"]
    on = want != 0
    got = g.grid.cpu().numpy().astype(np.complex128)[on]
    assert np.sqrt(np.mean(np.abs(got / want[on] - 1) ** 2)) < 4e-8


@pytest.mark.parametrize("stokes", [(1,), (1, 2)], ids=["i", "iq"])
@pytest.mark.parametrize("kw", [dict(nchan=600, nband=600), dict(nchan=1600, nband=1500),
                                dict(nchan=5000, bda_mode=1, dphi=0.5), dict(nchan=7000, bda_mode=1, dphi=0.5)],
                         ids=["600bands", "1500bands", "5000ch", "7000ch"])
def test_sums_of_many_bands_and_channels(kw, stokes):
    """Weight sums in one copy that the warps of a CTA share, and per-channel Jones sums beside the tiles of
    twelve warps.  FP64 sums of FP32 weights: 1e-12, times FP32 Jones weights: 1e-6."""
    c = cases.make_case(seed=67, nant=4, ntimes=3, ncorr=4, npix=63, cell_arcsec=8.0, nw=2, flag_frac=0.1,
                        stokes_ids=stokes, **kw)
    cases.add_jones(c, nt=2, nd=2, mode=1)
    want = cases.run_fp64_grid(c)
    vs, fg, jd = cases._gpu_objs(c)
    pol = D.make_pol(c.corr_ids, c.stokes_ids)
    fs = [dataclasses.replace(fg, **{k: torch.zeros_like(getattr(fg, k)) for k in
                                     ("grid", "sumwt", "sumjones", "sumjones_chan")}) for _ in range(3)]
    D.grid(vs, fs, pol, jd, batch=D.Batch.create())
    for f in fs:
        assert cases.rel_rms(f.grid.cpu().numpy(), want["grid"]) < 1e-6
        np.testing.assert_allclose(f.sumwt.cpu().numpy(), want["sumwt"], rtol=1e-12)
        np.testing.assert_allclose(f.sumjones.cpu().numpy(), want["sumjones"], rtol=1e-6)
        np.testing.assert_allclose(f.sumjones_chan.cpu().numpy(), want["sumjones_chan"], rtol=1e-6)


def test_phasor_rounding():
    """A model of ones seven cells apart: every 7 x 7 footprint holds one, so a prediction is one tap times
    the phasor.  Of a prediction's own value, RMS: the product and the phasor's own sine and cosine in FP32
    leave 4.1e-8 to 4.4e-8; a phase rounded to FP32 before them 5.5e-8 to 5.8e-8."""
    c = cases.make_case(seed=68, nant=12, ntimes=20, nchan=8, ncorr=1, npix=255, cell_arcsec=3.0, nw=1, sup=7,
                        lm=(0.012, -0.009))
    vs, fg, _ = cases._gpu_objs(c)
    assert set(fg.cf.sup.tolist()) == {7}
    model = np.zeros((1, 1, c.npix, c.npix), np.complex64)
    model[:, :, ::7, ::7] = 1
    got = cases.run_gpu_degrid(c, model).astype(np.complex128)
    want = cases.run_fp64_degrid(c, model)
    on = want != 0
    assert on.mean() > 0.9
    assert np.sqrt(np.mean(np.abs(got[on] / want[on] - 1) ** 2)) < 5e-8


@pytest.mark.parametrize("stokes,n", [((1,), 33000), ((1, 2), 23200)], ids=["i", "iq"])
def test_bands_beyond_two_billion_cells(stokes, n):
    """Two bands of a grid of more than 2^31 cells: the second is gridded and degridded as the only band of
    a grid of half the size is (float32 grids: another order of the additions, 1e-6)."""
    c = cases.make_case(seed=69, nant=7, ntimes=6, nchan=8, ncorr=4, npix=127, cell_arcsec=5.0, nw=2, stokes_ids=stokes)
    vs, fg, _ = cases._gpu_objs(c)
    incr = tuple(x * c.npix / n for x in c.incr)  # the same footprints about the middle of the grid
    pol = D.make_pol(c.corr_ids, c.stokes_ids)
    npol, lo, hi = len(stokes), n // 2 - 100, n // 2 + 100
    model = _randn((npol, hi - lo, hi - lo), 5)
    got = {}
    for nband in (1, 2):
        v = dataclasses.replace(vs, chan_map=torch.full_like(vs.chan_map, nband - 1))
        grid = torch.zeros((nband, npol, n, n), dtype=torch.complex64, device="cuda")
        f = dataclasses.replace(fg, grid=grid, incr=incr, sumwt=None, sumjones=None, sumjones_chan=None, grid_acc=None)
        out = []
        for acc in (None, torch.zeros(grid.shape, dtype=torch.complex128, device="cuda")):
            D.grid(v, [dataclasses.replace(f, grid_acc=acc)], pol)
            out.append(grid[-1, :, lo:hi, lo:hi].clone())
            grid[-1, :, lo:hi, lo:hi] = 0
            assert not torch.view_as_real(grid).any()  # nothing elsewhere
            del acc
        grid[-1, :, lo:hi, lo:hi] = model
        d = dataclasses.replace(v, vis=torch.zeros_like(v.vis))
        D.degrid(d, [f], pol)
        got[nband] = [*out, d.vis]
        del f, grid
        torch.cuda.empty_cache()
    for a, b in zip(got[2], got[1]):
        assert torch.count_nonzero(torch.view_as_real(b)) > 0
        assert _rms(a, b) < 1e-6


@pytest.mark.parametrize("kw", [dict(), dict(bda_mode=1, dphi=0.6), dict(nchan=130)], ids=["single", "bda", "130ch"])
def test_one_correlation_against_fp64(kw):
    """One correlation goes to the general gridding kernels and to the Stokes I degridder.  Grids and
    predictions carry some ten FP32 roundings, 3e-7 at most together: 1e-6; weight sums 1e-12, sums with
    FP32 Jones weights 1e-6."""
    c = cases.make_case(**{**dict(seed=70, nant=7, ntimes=10, nchan=9, ncorr=1, npix=127, cell_arcsec=5.0, nw=3, nband=2,
                                  flag_frac=0.1), **kw})
    cases.add_jones(c, nt=2, nd=2, mode=1, nch=2)
    want = cases.run_fp64_grid(c)
    got = cases.run_gpu_grid(c, batched=True, fp64_acc=True)
    assert cases.rel_rms(got["grid"], want["grid"]) < 1e-6
    np.testing.assert_allclose(got["sumwt"], want["sumwt"], rtol=1e-12)
    np.testing.assert_allclose(got["sumjones"], want["sumjones"], rtol=1e-6)
    np.testing.assert_allclose(got["sumjones_chan"], want["sumjones_chan"], rtol=1e-6)
    model = want["grid"].astype(np.complex64)
    assert cases.rel_rms(cases.run_gpu_degrid(c, model, batched=True), cases.run_fp64_degrid(c, model)) < 1e-6
