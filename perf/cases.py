"""The work that users of this framework have it do, as cases that can be timed and checked.

A case is a dict of plain values.  ``kind`` says which public call it makes:

* ``grid``    -- ``device.grid``: visibilities onto every facet's residual grid, as
                 ``FacetMachine.grid_all_facets`` and the major cycle call it;
* ``degrid``  -- ``device.degrid``: every facet's model prediction subtracted from the
                 visibilities;
* ``predict`` -- ``autograd.predict`` and its backward pass for every facet's model grid and the
                 Jones terms;
* ``worker``  -- ``ClassDDEGridMachine.put`` and ``get`` of one facet on numpy arrays, as one of
                 DDFacet's facet workers calls them;
* ``images``  -- ``FacetMachine.facets_to_image`` and ``image_to_facets``.

The other fields are the observation (``nant`` antennas in a disk of ``radius`` metres, or
log-radial with ``lograd``, ``ntimes`` dumps of ``dump`` seconds, ``nchan`` channels, ``ncorr``
correlations), the image (``npix`` pixels of ``cell`` arcsec in ``side`` x ``side`` facets, or in
a Voronoi tessellation of ``nfacets`` directions with ``side`` 0; ``nfacets`` of the facets are
taken), the W planes ``nw``, frequency bands ``nband``, ``stokes``, the flagged fraction ``flag``,
per-facet Jones terms (``jones``), FP64 grid sums (``fp64``), block averaging at a decorrelation
(``average``, 0: one visibility a block) and the schedule handed to the batched calls (``pack``
facets per pack and ``items`` stripes per item, 0: the library's own; ``pack`` -1: the plain call).
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

from ddfacet_b200 import autograd, bda, configs, device as D, facetmachine, geometry, gridmachine, synth

C = 299792458.0
OVERS = 11
PADDING = 1.7
OMEGA = 7.2921150e-5  # rad/s


# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------
def _case(kind, name=None, nant=27, ntimes=30, dump=10.0, nchan=16, ncorr=4, radius=4000.0, lograd=False, npix=1024,
          cell=1.5, side=1, nfacets=1, nw=8, nband=1, stokes="I", flag=0.05, jones=True, fp64=False, average=0.0,
          pack=0, items=0):
    c = dict(kind=kind, nant=nant, ntimes=ntimes, dump=dump, nchan=nchan, ncorr=ncorr, radius=radius, lograd=lograd,
             npix=npix, cell=cell, side=side, nfacets=nfacets, nw=nw, nband=nband, stokes=stokes, flag=flag,
             jones=jones, fp64=fp64, average=average, pack=pack, items=items)
    return dict(c, name=name) if name else c


def listed():
    # one DDFacet facet worker's chunk of the single-facet Stokes-I case (27 antennas, 16 channels)
    plain = dict(nant=27, ntimes=60, nchan=16, npix=1024, cell=1.0, nw=8)
    # a few dumps of the 4096^2, 9 x 9 facet direction-dependent imaging run (735^2 padded grids)
    multi = dict(nant=64, ntimes=20, dump=8.0, nchan=64, npix=4096, cell=1.5, side=9, nfacets=25, nw=32)
    # a few dumps of the 10000^2, 11 x 11 facet, 256-channel run (1485^2 padded grids)
    scale = dict(nant=64, ntimes=24, dump=8.0, nchan=256, npix=10000, cell=1.0, side=11, nfacets=25, nw=64, flag=0.0)
    # the uneven Voronoi facets with baseline-dependent averaging, twenty minutes of a smaller field
    uneven = dict(nant=48, ntimes=300, dump=4.0, nchan=64, radius=12000.0, lograd=True, npix=3000, cell=1.0, side=0,
                  nfacets=9, nw=32, average=0.02)
    return [
        _case("worker", "worker_put_get", **plain),
        # the smallest calls: a single facet and a short, narrow chunk, where launches and latency count
        _case("grid", "grid_small", nant=10, ntimes=30, nchan=8, ncorr=1, radius=2000.0, npix=255, cell=3.0, nw=4,
              jones=False, pack=-1),
        _case("degrid", "degrid_small", nant=10, ntimes=30, nchan=8, ncorr=1, radius=2000.0, npix=255, cell=3.0, nw=4,
              jones=False, pack=-1),
        # the major cycle over many facets, forward and backward
        _case("grid", "grid_facets", fp64=True, **multi),
        _case("degrid", "degrid_facets", **multi),
        # the same at the largest configuration, the degridder with the schedule its tuner picks
        _case("grid", "grid_at_scale", fp64=True, **scale),
        _case("degrid", "degrid_at_scale", pack=16, items=64, **scale),
        # averaged blocks on facets of very different sizes
        _case("grid", "grid_averaged", fp64=True, **uneven),
        _case("degrid", "degrid_averaged", **uneven),
        # full polarisation in two bands over a wide field: four Stokes planes, supports of 7 to 23, the
        # plain call with float32 sums that a FacetMachine makes
        _case("grid", "grid_iquv_wide", nant=27, ntimes=40, nchan=32, radius=3500.0, npix=3000, cell=2.5, side=2,
              nfacets=4, nw=16, nband=2, stokes="IQUV", flag=0.1, pack=-1),
        # calibration and imaging by gradient: the prediction and its derivatives
        _case("predict", "predict_gradient", nant=64, ntimes=6, dump=8.0, nchan=64, npix=4096, cell=1.5, side=9,
              nfacets=9, nw=32),
        # residual grids to the image, the model image back to facet grids
        _case("images", "facet_images", npix=3000, cell=1.5, side=3, nfacets=9, nband=2, nw=2),
    ]


def _cost(c):
    """Taps of a pass, roughly: supports grow with the facets' field, averaging leaves fewer blocks."""
    s2 = 49 if c["npix"] / (c["side"] or 2) * c["cell"] < 1000 else 225
    per = {"grid": 1, "degrid": 1, "predict": 5, "worker": 2, "images": 0}[c["kind"]] * (0.5 if c["average"] else 1)
    return per * c["nfacets"] * c["ntimes"] * c["nant"] * (c["nant"] - 1) // 2 * c["nchan"] * s2 * len(c["stokes"])


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    while True:
        kind = rng.choice(["grid"] * 4 + ["degrid"] * 4 + ["predict", "worker", "images"])
        if kind == "images":
            side = rng.randint(1, 4)
            return _case("images", npix=log(700, 900 * side + 100), cell=rng.choice([1.0, 1.5]), side=side,
                         nfacets=side * side, nband=rng.randint(1, 3), nw=2, stokes=rng.choice(["I", "I", "IQUV"]))
        c = _case(kind, nant=log(7, 64), ntimes=log(4, 120), dump=rng.choice([4.0, 8.0, 10.0]), nchan=log(4, 256),
                  ncorr=rng.choice([1, 2, 4, 4, 4]), radius=float(log(2000, 6000)), npix=log(1500, 6000),
                  cell=rng.choice([1.0, 1.5]), side=rng.choice([4, 7, 9]), nfacets=log(1, 32), nw=log(4, 64),
                  nband=rng.choice([1, 1, 1, 2]), flag=rng.choice([0.0, 0.05, 0.3]),
                  jones=rng.random() < 0.75, fp64=rng.random() < 0.6, pack=rng.choice([0, 0, 0, -1, 8, 16]),
                  items=rng.choice([0, 0, 64]))
        if kind in ("worker", "predict"):
            c.update(jones=True, fp64=False, nfacets=1 if kind == "worker" else min(12, c["nfacets"]))
        else:
            shape = rng.random()
            if shape < 0.3:  # averaged blocks, uneven facets
                c.update(side=0, npix=log(1500, 3000), nfacets=rng.randint(3, 12), lograd=True, radius=12000.0,
                         average=rng.choice([0.01, 0.02, 0.05]), ntimes=max(20, c["ntimes"]))
            elif shape < 0.5:  # full polarisation, wide field
                c.update(ncorr=4, stokes="IQUV", side=2, nfacets=rng.randint(1, 4), npix=log(1500, 3000), cell=2.5,
                         radius=3500.0, nw=log(4, 24))
        if c["nfacets"] > c["side"] ** 2 > 0:
            c["nfacets"] = c["side"] ** 2
        if _cost(c) <= 1.2e10:  # no more than the largest listed case
            return c


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")


@functools.lru_cache(maxsize=8)
def _baselines(nant, radius, lograd):
    """Baseline vectors (equatorial XYZ, metres) and antenna pairs of the fixed array."""
    rng = np.random.default_rng(1005)
    e, n, _ = synth.antenna_layout(rng, nant, radius, "lograd" if lograd else "disk")
    lat = np.deg2rad(34.0)
    xyz = np.stack([-np.sin(lat) * n, e, np.cos(lat) * n])
    a0, a1 = np.triu_indices(nant, 1)
    return xyz[:, a1] - xyz[:, a0], a0.astype(np.int32), a1.astype(np.int32)


def _uvw(hour_angles, b):
    d = np.deg2rad(40.0)
    s, c = np.sin(hour_angles)[:, None], np.cos(hour_angles)[:, None]
    u = s * b[0] + c * b[1]
    v = -np.sin(d) * c * b[0] + np.sin(d) * s * b[1] + np.cos(d) * b[2]
    w = np.cos(d) * c * b[0] - np.cos(d) * s * b[1] + np.sin(d) * b[2]
    return np.ascontiguousarray(np.stack([u.ravel(), v.ravel(), w.ravel()], axis=1))


def _freqs(c):
    return np.linspace(0.90e9, 1.67e9, c["nchan"])


@functools.lru_cache(maxsize=4)
def _plain_map(nant, ntimes, nchan):
    _, a0, a1 = _baselines(nant, 1000.0, False)
    return bda.plain_map(np.tile(a0, ntimes), np.tile(a1, ntimes), nchan)


@functools.lru_cache(maxsize=4)
def _field(npix, cell, side, nfacets, nw, nchan, nant, radius, lograd):
    """The facets and their W tables: they belong to the field and the array, and a program computes
    them once for all its chunks (DDFacet keeps them in its cache on disk)."""
    if side:
        every = geometry.regular_facets(npix, side, cell, PADDING).facets
        pick = np.unique(np.linspace(0, len(every) - 1, nfacets).astype(int))
        facets = [every[i] for i in pick]
    else:
        rng = np.random.default_rng(1008)
        r = npix * cell / 3600 * np.pi / 180 / 2
        facets = geometry.voronoi_facets(npix, cell, rng.uniform(-r, r, nfacets), rng.uniform(-r, r, nfacets),
                                         PADDING).facets
    b, _, _ = _baselines(nant, radius, lograd)
    wmax = float(np.abs(_uvw(np.linspace(-1.06, 1.06, 97), b)[:, 2]).max()) * 1.001
    freqs = np.linspace(0.90e9, 1.67e9, nchan)
    return facets, configs.build_wterms(facets, cell, 7, nw, wmax, [f.npix_padded for f in facets], freqs, OVERS)


def _field_of(c):
    return _field(c["npix"], c["cell"], c["side"], c["nfacets"], c["nw"], c["nchan"], c["nant"], c["radius"], c["lograd"])


def _corr_ids(c):
    return {1: [1], 2: [9, 12], 4: [9, 10, 11, 12]}[c["ncorr"]]


def _inputs(c, seed):
    """Observation, visibilities, flags, weights, Jones terms and model grids, from the seed."""
    dev = _device()
    rng = np.random.default_rng([seed, 1])
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    b, a0, a1 = _baselines(c["nant"], c["radius"], c["lograd"])
    nt, nchan, ncorr = c["ntimes"], c["nchan"], c["ncorr"]
    start = rng.uniform(-4 * 3600.0, 4 * 3600.0 - nt * c["dump"])
    t = start + np.arange(nt) * c["dump"]
    x = dict(uvw=_uvw(OMEGA * t, b), a0=np.tile(a0, nt), a1=np.tile(a1, nt), times=np.repeat(t, a0.size),
             freqs=_freqs(c), chan_map=(np.arange(nchan) * c["nband"] // nchan).astype(np.int32))
    nrow = x["uvw"].shape[0]
    uvw = torch.from_numpy(x["uvw"]).to(dev)
    fr = torch.from_numpy(x["freqs"] / C).to(dev)
    # twenty point sources and noise
    rad = c["npix"] * c["cell"] / 3600 * np.pi / 180 / 2 * 0.9
    l, m, s = synth.point_sky(seed % 100003, 20, rad, flux=("powerlaw", 1e-2, 1.0))
    lmn = torch.from_numpy(np.stack([l, m, np.sqrt(1 - l * l - m * m) - 1])).to(dev)
    vis = torch.view_as_complex(torch.randn((nrow, nchan, ncorr, 2), generator=gen, device=dev) * 1e-3)
    for k in range(20):
        turns = (uvw @ lmn[:, k])[:, None] * fr[None, :]
        v = torch.polar(torch.full_like(turns, float(s[k]), dtype=torch.float32),
                        (2 * math.pi * (turns - torch.round(turns))).to(torch.float32))
        for p in range(ncorr):
            vis[:, :, p] += v * (1.0 if p in (0, ncorr - 1) else 0.1)
    x["vis"] = vis
    x["flags"] = (torch.rand((nrow, nchan, 1), generator=gen, device=dev) < c["flag"]).expand(-1, -1, ncorr).contiguous()
    x["weights"] = 0.5 + torch.rand((nrow, nchan), generator=gen, device=dev)
    x["uvw_dev"] = uvw
    facets, _ = _field_of(c)
    if c["jones"]:
        slots = max(1, int(math.ceil(nt * c["dump"] / 300.0)))
        j = torch.view_as_complex(torch.randn((slots, len(facets), c["nant"], 1, 2, 2, 2), generator=gen, device=dev) * 0.1)
        x["kms"] = (j + torch.eye(2, device=dev)).contiguous()
        x["tmap"] = np.minimum((x["times"] - t[0]) // 300.0, slots - 1).astype(np.int32)
    npol = len(c["stokes"])
    if c["kind"] != "grid":  # model grids: smooth power falling off from the uv centre
        x["models"] = []
        for f in facets:
            n = f.npix_padded
            y = torch.arange(n, device=dev, dtype=torch.float32) - n // 2
            amp = 1.0 / (1.0 + (y[:, None] ** 2 + y[None, :] ** 2) / (0.15 * n) ** 2)
            g = torch.randn((c["nband"], npol, n, n, 2), generator=gen, device=dev)
            x["models"].append(torch.view_as_complex(g) * amp)
    return x


def _block_map(c, x):
    if not c["average"]:
        return _plain_map(c["nant"], c["ntimes"], c["nchan"])
    facets, _ = _field_of(c)
    lmax = max(f.npix_facet for f in facets) * c["cell"] / 3600 * np.pi / 180 * np.sqrt(2) / 2
    dfreq = float(x["freqs"][1] - x["freqs"][0])
    return bda.smear_mapping_gpu(x["a0"], x["a1"], x["uvw_dev"], x["freqs"], dfreq, np.sqrt(6 * c["average"]), lmax,
                                 x["chan_map"])


def prepare(case, seed):
    if case["kind"] == "images":
        return _prepare_images(case, seed)
    if case["kind"] == "worker":
        return _prepare_worker(case, seed)
    c, dev = case, _device()
    x = _inputs(c, seed)
    facets, wts = _field_of(c)
    vs = D.VisData.create(x["vis"], x["uvw_dev"], x["flags"], x["weights"], x["freqs"], x["chan_map"], _block_map(c, x))
    if c["average"]:  # blocks in uv order, long walks to whole warps, as the averaged configuration runs
        tile = 64 / (max(f.npix_padded for f in facets) * c["cell"] / 3600 * np.pi / 180)
        vs = vs.with_block_order(bda.uv_locality_order(vs.bda_map, vs.block_start, vs.uvw, vs.freqs, tile))
        vs = vs.with_large_blocks(2048)
    jones = None
    if c["jones"]:
        jones = D.JonesData(mode=1, kms=x["kms"], kms_tmap=torch.from_numpy(x["tmap"]).to(dev),
                            kms_cmap=torch.zeros(c["nchan"], dtype=torch.int32, device=dev),
                            a0=torch.from_numpy(x["a0"]).to(dev), a1=torch.from_numpy(x["a1"]).to(dev),
                            wavelength_mean=float(np.mean(C / x["freqs"])))
    npol, nf = len(c["stokes"]), len(facets)
    rad = c["cell"] / 3600 * np.pi / 180
    sums = dict(sumwt=torch.zeros((nf, c["nband"], npol), dtype=torch.float64, device=dev),
                sumjones=torch.zeros((nf, 2, c["nband"]), dtype=torch.float64, device=dev),
                sumjones_chan=torch.zeros((nf, 2, c["nchan"]), dtype=torch.float64, device=dev))
    fgs = []
    for i, (f, wt) in enumerate(zip(facets, wts)):
        tabs = D.CFTables.create(wt.Wplanes, wt.WplanesConj, OVERS, wt.RefWave, wt.wmax)
        n = f.npix_padded
        g = x["models"][i] if "models" in x else torch.zeros((c["nband"], npol, n, n), dtype=torch.complex64, device=dev)
        fg = D.FacetGrid(grid=g, cf=tabs, incr=(-rad, rad), cu=wt.Cu, cv=wt.Cv, l0=f.l0, m0=f.m0, idir_kms=i,
                         **{k: v[i] for k, v in sums.items()})
        fgs.append(fg.with_fp64_accumulation() if c["kind"] == "grid" and c["fp64"] else fg)
    pol = D.make_pol(_corr_ids(c), ["IQUV".index(s) + 1 for s in c["stokes"]])
    batch = None if c["pack"] < 0 else D.Batch.create(facets_per_pack=c["pack"], stripes_per_item=c["items"])
    st = dict(kind=c["kind"], vs=vs, facets=fgs, pol=pol, jones=jones, batch=batch, sums=sums)
    if c["kind"] == "degrid":
        st["data"] = vs.vis
        st["vs"] = dataclasses.replace(vs, vis=torch.empty_like(vs.vis))
    elif c["kind"] == "predict":
        st["setup"] = autograd.PredictSetup(vs=vs, facets=fgs, pol=pol, jones=jones)
        st["grids"] = [f.grid.requires_grad_() for f in fgs]
        st["kms"] = x["kms"].requires_grad_()
        st["residual"] = x["vis"]
    return st


def _prepare_worker(c, seed):
    x = _inputs(c, seed)
    facets, wts = _field_of(c)
    f, wt = facets[0], wts[0]
    gd = gridmachine.default_gd()
    gd["Image"]["Cell"] = c["cell"]
    gd["CF"]["Nw"] = c["nw"]
    cf = {"wmax": wt.wmax, "Sphe": np.float32(wt.ifzfCF.real), "CuCv": np.array([wt.Cu, wt.Cv]),
          "W": list(wt.Wplanes) + list(wt.WplanesConj)}
    bmap = _block_map(c, x)
    gm = gridmachine.ClassDDEGridMachine(gd, x["freqs"], f.npix_facet, lmShift=(f.l0, f.m0), cf_dict=cf, bda_grid=bmap,
                                         bda_degrid=bmap, DataCorrelationFormat=_corr_ids(c),
                                         ExpectedOutputStokes=["IQUV".index(s) + 1 for s in c["stokes"]],
                                         NFreqBands=c["nband"], Padding=PADDING)
    dico = {"DicoJones_killMS": {"Dirs": {"l": np.array([f.l0]), "m": np.array([f.m0]), "I": np.ones(1)},
                                 "Jones": {"Jones": x["kms"].cpu().numpy(),
                                           "VisToJonesChanMapping": np.zeros(c["nchan"], np.int32)},
                                 "TimeMapping": x["tmap"]}}
    return dict(kind="worker", gm=gm, x=x, vis=x["vis"].cpu().numpy(), flags=x["flags"].cpu().numpy(),
                weights=x["weights"].cpu().numpy(), model=x["models"][0].cpu().numpy(), dico=dico,
                grid=np.zeros(gm.GridShape, np.complex64))


def _prepare_images(c, seed):
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    fm = facetmachine.FacetMachine(c["npix"], c["cell"], c["side"], _freqs(c), padding=PADDING, nband=c["nband"],
                                   stokes_ids=["IQUV".index(s) + 1 for s in c["stokes"]], nw=c["nw"], wmax=3000.0)
    grids = []
    for f in fm.facets:
        n = f.grid.grid.shape[-1]
        y = torch.arange(n, device=dev, dtype=torch.float32) - n // 2
        amp = 100.0 / (1.0 + (y[:, None] ** 2 + y[None, :] ** 2) / (0.15 * n) ** 2)
        grids.append(torch.view_as_complex(torch.randn((*f.grid.grid.shape, 2), generator=gen, device=dev)) * amp)
        f.grid.sumwt += 1e5 * (1 + torch.rand(f.grid.sumwt.shape, generator=gen, device=dev, dtype=torch.float64))
        f.grid.sumjones += 1e5 * (1 + torch.rand(f.grid.sumjones.shape, generator=gen, device=dev, dtype=torch.float64))
    m = fm.npix_out
    model = torch.zeros((c["nband"], fm.npol, m, m), device=dev)
    at = torch.randint(int(0.05 * m), int(0.95 * m), (2, 500), generator=gen, device=dev)
    model[:, :, at[0], at[1]] = torch.rand((c["nband"], fm.npol, 500), generator=gen, device=dev)
    return dict(kind="images", fm=fm, grids=grids, model=model)


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------
def run(state):
    s = state
    if s["kind"] == "grid":
        for f in s["facets"]:
            f.grid.zero_()
        for v in s["sums"].values():
            v.zero_()
        D.grid(s["vs"], s["facets"], s["pol"], s["jones"], batch=s["batch"])
        return {"grids": [f.grid for f in s["facets"]], **s["sums"]}
    if s["kind"] == "degrid":
        s["vs"].vis.copy_(s["data"])  # the residuals start from the data
        D.degrid(s["vs"], s["facets"], s["pol"], s["jones"], batch=s["batch"])
        return {"residual": s["vs"].vis}
    if s["kind"] == "predict":
        p = autograd.predict(s["setup"], s["grids"], s["kms"])
        grads = torch.autograd.grad(p, [s["kms"], *s["grids"]], grad_outputs=s["residual"])
        return {"vis": p.detach(), "jones": grads[0], "grids": list(grads[1:])}
    if s["kind"] == "worker":
        gm, x = s["gm"], s["x"]
        gm.reinitGrid()
        s["grid"][...] = 0
        vis = s["vis"].copy()
        kw = dict(DicoJonesMatrices=s["dico"], freqs=x["freqs"], ChanMapping=x["chan_map"])
        gm.get(x["times"], x["uvw"], vis, s["flags"], (x["a0"], x["a1"]), s["model"], ImToGrid=False, **kw)
        gm.put(x["times"], x["uvw"], vis, s["flags"], (x["a0"], x["a1"]), W=s["weights"], ResidueGrid=s["grid"], **kw)
        return {"residual": vis, "grid": s["grid"], "sumwt": gm.SumWeigths, "sumjones": gm.SumJones,
                "sumjones_chan": gm.SumJonesChan}
    fm = s["fm"]
    for f, g in zip(fm.facets, s["grids"]):
        f.grid.grid.copy_(g)  # transformed in place
    image = fm.facets_to_image()
    fm.image_to_facets(s["model"])
    return {"image": image, "grids": [f.model.grid for f in fm.facets]}


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
def work(case):
    c = case
    npol = len(c["stokes"])
    if c["kind"] == "images":
        tess = geometry.regular_facets(c["npix"], c["side"], c["cell"], PADDING)
        n, planes = tess.npix_padded, c["nband"] * npol
        px, im = len(tess.facets) * planes * n * n, planes * tess.npix ** 2
        return {"bytes": 16 * px + 12 * tess.npix ** 2 + 8 * im, "flops": px * 2 * 5 * 2 * math.log2(n)}
    facets, wts = _field_of(c)
    nrow = c["ntimes"] * c["nant"] * (c["nant"] - 1) // 2
    nvis, K, F = nrow * c["nchan"], c["ncorr"], len(facets)
    cells = sum(f.npix_padded ** 2 for f in facets) * c["nband"] * npol
    cfs = sum(p.nbytes for wt in wts for p in wt.Wplanes)
    s2 = float(np.mean([s * s for s in wts[0].supports]))
    # S^2 complex multiply-adds a Stokes plane, the 2 x 2 Jones products and the phasor
    flops = F * nvis * (8 * s2 * npol + 132)
    side = 24 * nrow + 8 * cells + cfs
    g, d = nvis * (8 * K + K + 4) + side, nvis * 16 * K + side
    if c["kind"] == "worker":
        return {"bytes": g + d, "flops": 2 * flops}
    if c["kind"] == "predict":  # the prediction, its adjoint, and the gather and two products of the Jones gradient
        return {"bytes": nvis * 8 * K * 2 + side + 8 * cells, "flops": 3 * flops}
    return {"bytes": g if c["kind"] == "grid" else d, "flops": flops}


# ------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------
class _Facet64:
    """One facet's geometry and W tables for the 64-bit restatement below."""

    def __init__(self, f, wt, cell, swap, dev):
        self.n, self.l0, self.m0, self.n0 = f.npix_padded, f.l0, f.m0, math.sqrt(1 - f.l0 ** 2 - f.m0 ** 2) - 1
        self.cu, self.cv, self.ref, self.wmax, self.nw = wt.Cu, wt.Cv, wt.RefWave, wt.wmax, len(wt.Wplanes)
        self.incr = cell / 3600 * np.pi / 180
        planes = list(wt.WplanesConj) + list(wt.Wplanes) if swap else list(wt.Wplanes) + list(wt.WplanesConj)
        self.sup = torch.tensor([p.shape[0] // OVERS for p in planes], device=dev)
        self.off = torch.tensor(np.concatenate([[0], np.cumsum([p.size for p in planes])[:-1]]), device=dev)
        self.cf = torch.from_numpy(np.concatenate([p.ravel() for p in planes])).to(dev, torch.complex128)

    def footprints(self, u, v, w, recip, ok):
        """For every support in use: (which points, their first tap's cell, their taps' table offset, S)."""
        iw = torch.round(((self.nw - 1.0) * w.abs()) * (self.ref * recip) / self.wmax)
        ok = ok & (iw < self.nw)
        plane = torch.where(w > 0, iw, self.nw + iw).long().clamp(0, 2 * self.nw - 1)
        S = self.sup[plane]
        h = (S - 1) // 2
        px = (self.n * -self.incr * u) * recip + self.n // 2
        py = (self.n * self.incr * v) * recip + self.n // 2
        lx, ly = torch.round(px), torch.round(py)
        ok = ok & (lx - h >= 0) & (lx + h < self.n) & (ly - h >= 0) & (ly + h < self.n)
        mid = (S * OVERS - 1) // 2 - h * OVERS
        k = (torch.round((ly - py) * OVERS).long() + mid) * OVERS + torch.round((lx - px) * OVERS).long() + mid
        ok = ok & (k >= 0) & (k < OVERS * OVERS)
        for s in torch.unique(S[ok]).tolist():
            at = torch.nonzero(ok & (S == s)).flatten()
            for p in at.split(max(1, 24_000_000 // (s * s))):
                yield p, ((ly[p].long() - s // 2) * self.n + lx[p].long() - s // 2), self.off[plane[p]] + k[p] * s * s, s

    def taps(self, cell, off, s):
        t = torch.arange(s * s, device=cell.device)
        return cell[:, None] + (t // s) * self.n + t % s, self.cf[off[:, None] + t]

    def phase(self, x, sign):
        turns = x["U"] * self.l0 + x["V"] * self.m0 + x["W"] * self.n0
        turns = sign * x["nu"] * turns / C
        return torch.polar(torch.ones_like(turns), 2 * math.pi * (turns - torch.round(turns)))


def _walk(c, x, bmap, dev):
    """The map's blocks in groups: each visibility's row, channel and block, and the inputs at it."""
    m = torch.as_tensor(bmap).to(dev)
    nb = int(m[0])
    size = m[2:2 + nb].long()
    start = 2 + nb + torch.cumsum(size, 0) - size
    ch0, nch, nr = m[start].long(), (m[start + 1] - m[start]).long(), size - 2
    fr = torch.from_numpy(x["freqs"]).to(dev)
    uvw = torch.from_numpy(x["uvw"]).to(dev)
    tmap = torch.from_numpy(x["tmap"]).to(dev) if c["jones"] else None
    a0, a1 = (torch.from_numpy(x[k]).to(dev).long() for k in ("a0", "a1"))
    band = torch.from_numpy(x["chan_map"]).to(dev).long()
    for blk in torch.arange(nb, device=dev).split(1_000_000):
        n = nr[blk] * nch[blk]
        own = torch.repeat_interleave(torch.arange(blk.numel(), device=dev), n)
        k = torch.arange(own.numel(), device=dev) - (torch.cumsum(n, 0) - n)[own]
        b = blk[own]
        row = m[start[b] + 2 + k // nch[b]].long()
        ch = ch0[b] + k % nch[b]
        d = dict(own=own, n=blk.numel(), row=row, ch=ch, U=uvw[row, 0], V=uvw[row, 1], W=uvw[row, 2], nu=fr[ch],
                 band=band[ch0[blk]], a0=a0[row], a1=a1[row], freqs=fr)
        if c["jones"]:
            d["slot"] = tmap[row].long()
        yield d


def _mean(w, val, own, n, cnt):
    return torch.zeros(n, dtype=torch.float64, device=val.device).index_add_(0, own, w * val) / cnt


def _two_by_two(v):
    """[n, ncorr] correlations as [n, 2, 2] (a single one on the diagonal, a pair on it)."""
    if v.shape[1] == 4:
        return v.reshape(-1, 2, 2)
    out = torch.zeros((v.shape[0], 2, 2), dtype=v.dtype, device=v.device)
    out[:, 0, 0], out[:, 1, 1] = v[:, 0], v[:, -1]
    return out


def _corr_of(stokes, ncorr, s):
    """Stokes planes [npol, n] to [n, 2, 2] correlations of linear feeds."""
    z = torch.zeros_like(s[0])
    q, u, v = (s[1], s[2], s[3]) if stokes == "IQUV" else (z, z, z)
    return torch.stack([s[0] + q, u + 1j * v, u - 1j * v, s[0] - q], -1).reshape(-1, 2, 2)


def _grid64(c, x, bmap, f, i, vis, dev):
    npol, nb = len(c["stokes"]), c["nband"]
    grid = torch.zeros((nb * npol, f.n * f.n), dtype=torch.complex128, device=dev)
    swt = torch.zeros((nb, npol), dtype=torch.float64, device=dev)
    sj = torch.zeros((2, nb), dtype=torch.float64, device=dev)
    sjc = torch.zeros((2, c["nchan"]), dtype=torch.float64, device=dev)
    for d in _walk(c, x, bmap, dev):
        good = (~x["flags"][d["row"], d["ch"], 0]).double()
        own, n = d["own"], d["n"]
        cnt = torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, own, good)
        mean = functools.partial(_mean, good, own=own, n=n, cnt=cnt)
        wgt = x["weights"][d["row"], d["ch"]].double() * good
        V = _two_by_two(vis[d["row"], d["ch"]].to(torch.complex128))
        bb = torch.zeros_like(wgt)
        if c["jones"]:
            J = x["kms"][:, i, :, 0].to(torch.complex128)
            j0, j1 = J[d["slot"], d["a0"]], J[d["slot"], d["a1"]]
            V = j0.mH @ V @ j1
            bb = ((j0[:, 0, 0].abs() * j1[:, 0, 0].abs() + j0[:, 1, 1].abs() * j1[:, 1, 1].abs()) / 2) ** 2
        V = V * (f.phase(d, -1) * wgt)[:, None, None]
        if c["ncorr"] < 4:
            V = V * torch.eye(2, device=dev)
        if c["ncorr"] == 1:
            V[:, 1, 1] = V[:, 0, 0]
        S = [(V[:, 0, 0] + V[:, 1, 1]) / 2]
        if npol == 4:
            S += [(V[:, 0, 0] - V[:, 1, 1]) / 2, (V[:, 0, 1] + V[:, 1, 0]) / 2, -0.5j * (V[:, 0, 1] - V[:, 1, 0])]
        S = torch.zeros((npol, n), dtype=torch.complex128, device=dev).index_add_(1, own, torch.stack(S))
        took = torch.zeros(n, dtype=torch.bool, device=dev)
        for p, cell, off, s in f.footprints(mean(d["U"] + d["W"] * f.cu), mean(d["V"] + d["W"] * f.cv), mean(d["W"]),
                                            mean(d["nu"]) / C, cnt > 0):
            cells, cf = f.taps(cell, off, s)
            took[p] = True
            for q in range(npol):
                at = (d["band"][p] * npol + q)[:, None] * (f.n * f.n) + cells
                v = torch.view_as_real((S[q, p, None] * cf).reshape(-1))
                torch.view_as_real(grid.view(-1)).index_add_(0, at.reshape(-1), v)
        hit, bnd = wgt * took[own], d["band"][own]
        swt += torch.zeros(nb, dtype=torch.float64, device=dev).index_add_(0, bnd, hit)[:, None]
        if c["jones"]:
            for r, val in enumerate((npol * bb * hit, npol * hit)):
                sj[r].index_add_(0, bnd, val)
                sjc[r].index_add_(0, d["ch"], val)
    return grid.view(nb, npol, f.n, f.n), swt, sj, sjc


def _predict64(c, x, bmap, f, i, model, kms, dev):
    """Yields (rows, channels, prediction [n, ncorr]) of one facet's model grid."""
    npol = len(c["stokes"])
    flat = model.reshape(c["nband"], npol, -1)
    for d in _walk(c, x, bmap, dev):
        own, n = d["own"], d["n"]
        one = torch.ones_like(d["U"])
        cnt = torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, own, one)
        mean = functools.partial(_mean, one, own=own, n=n, cnt=cnt)
        S = torch.zeros((npol, n), dtype=torch.complex128, device=dev)
        seen = torch.zeros(n, dtype=torch.bool, device=dev)
        for p, cell, off, s in f.footprints(mean(d["U"] + d["W"] * f.cu), mean(d["V"] + d["W"] * f.cv), mean(d["W"]),
                                            mean(d["nu"]) / C, cnt > 0):
            cells, cf = f.taps(cell, off, s)
            seen[p] = True
            S = S.index_put((torch.arange(npol, device=dev)[:, None], p[None, :]), torch.stack(
                [(flat[d["band"][p][:, None], q, cells] * cf).sum(1) for q in range(npol)]))
        V = _corr_of(c["stokes"], c["ncorr"], S)[own]
        if kms is not None:
            J = kms[:, i, :, 0]
            V = J[d["slot"], d["a0"]] @ V @ J[d["slot"], d["a1"]].mH
        V = V * f.phase(d, 1)[:, None, None] * seen[own][:, None, None]
        V = V.reshape(-1, 4)
        yield d["row"], d["ch"], V if c["ncorr"] == 4 else V[:, [0, 3]] if c["ncorr"] == 2 else V[:, :1]


def exact(case, seed):
    c, dev = case, _device()
    if c["kind"] == "images":
        return _exact_images(c, seed)
    x = _inputs(c, seed)
    bmap = _block_map(c, x)
    facets, wts = _field_of(c)
    every = range(len(facets))
    fs = {i: _Facet64(facets[i], wts[i], c["cell"], c["kind"] != "grid", dev) for i in every}
    kms = x["kms"].to(torch.complex128) if c["jones"] else None
    if c["kind"] == "grid":
        # three facets' grids (64-bit scatters are slow), every facet's layout
        some = {0, len(facets) // 2, len(facets) - 1}
        got = {i: _grid64(c, x, bmap, fs[i], i, x["vis"], dev) for i in some}
        return {"grids": [got[i][0] if i in got else None for i in every], "sumwt": None, "sumjones": None,
                "sumjones_chan": None}
    if c["kind"] == "predict":
        kms.requires_grad_()
        vis = torch.zeros(x["vis"].shape, dtype=torch.complex128, device=dev)
        grads = []
        for i in every:
            g = x["models"][i].to(torch.complex128).requires_grad_()
            for row, ch, p in _predict64(c, x, bmap, fs[i], i, g, kms, dev):
                vis.index_put_((row, ch), p.detach(), accumulate=True)
                p.backward(x["vis"][row, ch].to(torch.complex128))
            grads.append(g.grad)
        return {"vis": vis, "jones": kms.grad, "grids": grads}
    res = x["vis"].to(torch.complex128)
    for i in every:
        for row, ch, p in _predict64(c, x, bmap, fs[i], i, x["models"][i].to(torch.complex128), kms, dev):
            res.index_put_((row, ch), -p, accumulate=True)
    if c["kind"] == "degrid":
        return {"residual": res}
    f = _Facet64(facets[0], wts[0], c["cell"], False, dev)
    grid, swt, sj, sjc = _grid64(c, x, bmap, f, 0, res, dev)
    return {"residual": res, "grid": grid, "sumwt": swt, "sumjones": sj, "sumjones_chan": sjc}


def _box(centre, m, n):
    """First and last + 1 pixel of a facet's padded box inside the image, and in the facet."""
    lo = max(0, centre - n // 2)
    hi = min(m - 1, centre + n // 2)
    return lo, hi + 1, lo - (centre - n // 2), n - (centre + n // 2 - hi)


def _exact_images(c, seed):
    s = _prepare_images(c, seed)
    fm = s["fm"]
    m = fm.npix_out
    image = torch.zeros((c["nband"], fm.npol, m, m), dtype=torch.float64, device=fm.device)
    norm = fm.facet_norm.double()
    dims = (-2, -1)
    grids = []
    for f, g in zip(fm.facets, s["grids"]):
        n = g.shape[-1]
        (x0, x1, fx0, fx1), (y0, y1, fy0, fy1) = (_box(p, m, n) for p in f.geom.pix_central)
        dirty = torch.fft.fftshift(torch.fft.ifft2(torch.fft.ifftshift(g.to(torch.complex128) * OVERS ** 2, dim=dims),
                                                   norm="forward"), dim=dims).real
        sj = f.grid.sumjones
        wgt = f.grid.sumwt * torch.sqrt(sj[0] / sj[1])[:, None]
        taper = f.sphe.double()
        part = torch.where(f.sphe < 1e-3, 0.0, dirty * f.invsphe.double() * f.sw_grid.double() / wgt[:, :, None, None])
        part = part.flip(-2).transpose(-2, -1)
        image[:, :, x0:x1, y0:y1] += part[:, :, fx0:fx1, fy0:fy1]
        crop = torch.zeros((c["nband"], fm.npol, n, n), dtype=torch.float64, device=fm.device)
        crop[:, :, fx0:fx1, fy0:fy1] = s["model"].double()[:, :, x0:x1, y0:y1] / norm[x0:x1, y0:y1]
        crop = torch.where(f.sphe < 1e-3, 0.0, crop * f.sw_img.double() / taper)
        crop = crop.transpose(-2, -1).flip(-2) * (OVERS * n) ** 2
        grids.append(torch.fft.fftshift(torch.fft.fft2(torch.fft.ifftshift(crop, dim=dims)), dim=dims) / n ** 2)
    return {"image": image / norm, "grids": grids}
