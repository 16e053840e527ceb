"""Performance cases of the surface-flow library: what a user's program runs, through the public
entry points, over the range of grids, precisions, forcings and network shapes it is used for.

A case is a dict of plain values; its ``kind`` says which call it times:

* ``run``       ``SurfaceFlow.fused_steps`` on one resident grid and the read-back of its maps, as a
                simulation does between two outputs;
* ``ensemble``  ``Ensemble.steps`` over members of uneven grid sizes and the read-back of their
                peak-depth maps;
* ``stages``    the drop-in sequence of a MATLAB main loop, one call per reference function
                (hydrology, routing, time step, maxima), and the read-back of the depth;
* ``predict``   the screening network's inference on a batch of members;
* ``train``     one training step of the screening network (loss, gradients, Adam);
* ``conv``      one 3x3 convolution layer of the network, forward and backward.

Inputs are seeded and made on the GPU, with the geometry of the benchmark configurations
(``hydropol2d_b200.synthetic``): V-tilted catchments, a fractal valley with a flood wave in it,
urban terrain with buildings.  ``exact`` restates the step and the network in 64-bit torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

from hydropol2d_b200.ensemble import Ensemble
from hydropol2d_b200.surface import SurfaceFlow
from hydropol2d_b200.surrogate import Conv3x3, UNet, forward_flops, layer_level, unet_spec
from hydropol2d_b200.synthetic import green_ampt_soil_tables

DEV = "cuda"
LONG = 1.0e9   # routing_time [min]: no pass reaches the end of its simulation


def _grid(name, ny, nx, precision, terrain, steps, rain="uniform", soil=False, depth=0.0, share=0.0, hazard=False,
          kind="run"):
    return dict(name=name, kind=kind, ny=ny, nx=nx, precision=precision, terrain=terrain, rain=rain, soil=soil,
                depth=depth, share=share, hazard=hazard, steps=steps)


def listed():
    return [
        # the smallest grid a study uses, in the reference's precision, from a dry start: the
        # V-tilted verification catchment, bound by the latency of a step
        _grid("vtilt_200_fp64", 200, 200, "fp64", "vtilt", 64),
        # one rain member of the screening study on its own
        _grid("rain_256_fp32", 256, 256, "fp32", "vtilt", 64, depth=5.0),
        # a catchment of odd sides with the velocity and hazard maxima kept
        _grid("hazard_509x701_fp32", 509, 701, "fp32", "vtilt", 64, depth=20.0, hazard=True),
        # rain on a fully wet grid: every cell takes the whole step
        _grid("wet_2048_fp32", 2048, 2048, "fp32", "vtilt", 64, depth=50.0),
        # urban rain-on-grid: Green-Ampt soils and 64 x 64 rain maps on 2 m cells
        _grid("urban_2048_fp32", 2048, 2048, "fp32", "urban", 64, rain="maps", soil=True, depth=5.0),
        # the dam-break valley at its full size, the flood wave over 29 % of it
        _grid("valley_4096x8192_fp32", 4096, 8192, "fp32", "valley", 128, rain="none", share=0.41),
        # the urban grid in the reference's precision, for runs that must track it
        _grid("urban_1000_fp64", 1000, 1000, "fp64", "urban", 32, rain="maps", soil=True, depth=5.0),
        # a batch of uneven members, as a probabilistic study or a calibration runs them
        dict(name="ensemble_48", kind="ensemble", members=48, lo=256, hi=1024, breach=0.25, steps=64),
        # the reference's main loop calling one function after the other
        _grid("stages_1024_fp64", 1024, 1024, "fp64", "vtilt", 4, depth=20.0, kind="stages"),
        # screening a batch of members
        dict(name="predict_32x256", kind="predict", batch=32, height=256, width=256),
        # training the screening network with its default batch
        dict(name="train_16x256", kind="train", batch=16, height=256, width=256),
        # a decoder layer on members whose sides are multiples of 32 only
        dict(name="conv_dec0a_224x160", kind="conv", layer="dec0a", batch=16, height=224, width=160),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["ensemble", "stages", "predict", "train", "conv", "conv"])
    if kind in ("run", "stages"):
        terrain = rng.choice(["vtilt", "urban", "valley"])
        ny, nx = _log_int(rng, 128, 2500), _log_int(rng, 128, 2500)
        stages = kind == "stages"
        return dict(kind=kind, ny=ny, nx=nx, precision=rng.choice(["fp32", "fp32", "fp64"]), terrain=terrain,
                    rain="none" if terrain == "valley" else rng.choice(["uniform", "maps"] if terrain == "urban" else ["uniform"]),
                    soil=terrain == "urban", depth=0.0 if terrain == "valley" else float(rng.choice([0.0, 5.0, 50.0])),
                    share=round(rng.uniform(0.1, 0.9), 3) if terrain == "valley" else 0.0,
                    hazard=(not stages) and rng.random() < 0.15, steps=rng.randint(2, 5) if stages else rng.randint(32, 96))
    if kind == "ensemble":
        return dict(kind=kind, members=_log_int(rng, 8, 64), lo=256, hi=rng.choice([256, 512, 1024]),
                    breach=rng.choice([0.0, 0.25]), steps=rng.randint(32, 96))
    h, w = 32 * rng.randint(4, 12), 32 * rng.randint(4, 12)
    if kind == "conv":
        layer = rng.choice([n for n, _, _, _ in unet_spec()])
        return dict(kind=kind, layer=layer, batch=rng.choice([4, 8, 16]), height=h, width=w)
    batch = 4 * _log_int(rng, 1, 8 if kind == "predict" else 4)
    return dict(kind=kind, batch=batch, height=h, width=w)


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _field(ny, nx, gen, slope=-3.0):
    """Zero-mean, unit-std random field with an isotropic power spectrum k^slope, on the GPU."""
    noise = torch.randn(ny, nx, generator=gen, device=DEV, dtype=torch.float64)
    ky = torch.fft.fftfreq(ny, device=DEV, dtype=torch.float64)[:, None]
    kx = torch.fft.rfftfreq(nx, device=DEV, dtype=torch.float64)[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    k[0, 0] = math.inf
    f = torch.fft.irfft2(torch.fft.rfft2(noise) * k ** (slope / 2.0), s=(ny, nx))
    f -= f.mean()
    return f / f.std()


def _classes(ny, nx, n, gen):
    """A map of n classes in contiguous patches."""
    f = _field(ny, nx, gen)
    cuts = torch.special.ndtri(torch.arange(1, n, device=DEV, dtype=torch.float64) / n)
    return torch.bucketize(f, cuts)


def _site(case, seed):
    """The arrays of one grid on the GPU in FP64 (m, mm, mm/h) and its parameters."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    ny, nx = case["ny"], case["nx"]
    f64 = dict(device=DEV, dtype=torch.float64)
    terrain, soil = case["terrain"], None
    if terrain == "vtilt":
        dx = 10.0
        left = (nx - 2) // 2
        x, y = torch.arange(nx, **f64) * dx, torch.arange(ny, **f64) * dx
        side = torch.clamp(left * dx - x, min=0.0) + torch.clamp(x - (left + 1) * dx, min=0.0)
        z = 100.0 + 0.002 * y[:, None] + 0.005 * side[None, :] + 0.5 * _field(ny, nx, gen)
        rough = torch.full((ny, nx), 0.02, **f64) * float(0.7 + 0.6 * torch.rand(1, generator=gen, device=DEV).item())
        rows, cols = np.zeros(2), np.arange(left, left + 2)
        params = dict(alfa_min=0.7, alfa_max=0.7, outlet_type=1, slope_outlet=0.002)
        d0 = case["depth"] * (1.0 + 0.2 * torch.rand(ny, nx, generator=gen, **f64))
    elif terrain == "urban":
        dx = 2.0
        f = _field(ny, nx, gen)
        z = (f - f.min()) / (f.max() - f.min()) * 40.0
        b = 12   # buildings of up to 12 x 12 cells, 10 m high, on about 30 % of the grid
        lots = torch.rand((ny + b - 1) // b, (nx + b - 1) // b, generator=gen, device=DEV) < 0.3
        z = z + 10.0 * lots.repeat_interleave(b, 0).repeat_interleave(b, 1)[:ny, :nx]
        rough = torch.tensor([0.013, 0.03, 0.05, 0.1], **f64)[_classes(ny, nx, 4, gen)]
        rows = np.concatenate([np.zeros(nx), np.full(nx, ny - 1), np.arange(1, ny - 1), np.arange(1, ny - 1)])
        cols = np.concatenate([np.arange(nx), np.arange(nx), np.zeros(ny - 2), np.full(ny - 2, nx - 1)])
        params = dict(alfa_min=0.5, alfa_max=0.7, outlet_type=2)
        d0 = case["depth"] * (1.0 + 0.2 * torch.rand(ny, nx, generator=gen, **f64))
    else:   # a valley along x, water 30 m deep over the thalweg in the first `share` of its length
        dx = 5.0
        scale = min(1.0, max(ny / 4096.0, 0.1))
        y = (torch.arange(ny, **f64) + 0.5) / ny * 2.0 - 1.0
        x = torch.arange(nx, **f64) * dx
        bed = 0.001 * (x[-1] - x)[None, :] + 20.0
        z = 60.0 * scale * (y[:, None] ** 2) + bed + 5.0 * scale * _field(ny, nx, gen)
        d0 = torch.clamp(bed + 30.0 * scale - z, min=0.0) * 1000.0
        d0[:, max(2, int(round(case["share"] * nx))):] = 0.0
        rough = torch.full((ny, nx), 0.035, **f64)
        rows, cols = np.arange(ny), np.full(ny, nx - 1)
        params = dict(alfa_min=0.5, alfa_max=0.7, outlet_type=1, slope_outlet=0.001)
    if case["soil"]:
        cls = _classes(ny, nx, 3, gen)
        soil = dict(cls=cls, tables=green_ampt_soil_tables([1.0, 10.0, 30.0], [50.0, 110.0, 200.0], [0.2, 0.3, 0.4]))
        params["flag_infiltration"] = 1
    rate = maps = None
    if case["rain"] == "uniform":
        rate = float(20.0 + 130.0 * torch.rand(1, generator=gen, device=DEV).item())
    elif case["rain"] == "maps":
        maps = 120.0 * torch.rand(25, 64, 64, generator=gen, device=DEV, dtype=torch.float32)
    params |= dict(routing_time=LONG, min_time_step=0.01, max_time_step=10.0)
    return dict(z=z, rough=rough, dx=dx, rows=rows.astype(np.int32), cols=cols.astype(np.int32), params=params, d0=d0,
                soil=soil, rate=rate, maps=maps)


def _host(t):
    return t.cpu().numpy()


def _flow(site, precision):
    """A SurfaceFlow with the site's data uploaded, as a program has it before its main loop."""
    ny, nx = site["z"].shape
    sf = SurfaceFlow(ny, nx, site["dx"], precision, **site["params"])
    sf.upload_static(_host(site["z"]), _host(site["rough"]), site["rows"], site["cols"])
    storage = None
    if site["soil"] is not None:
        sf.set_soil(_host(site["soil"]["cls"]).astype(np.uint8), **site["soil"]["tables"])
        storage = np.full((ny, nx), 5.0)
    sf.set_state(_host(site["d0"]), None, storage)
    if site["rate"] is not None:
        sf.set_rain_uniform(np.array([0.0]), np.array([site["rate"]]))
    if site["maps"] is not None:
        sf.set_rain_maps(_host(site["maps"]), 5.0)
    return sf


def _pinned(n):
    """Page-locked FP64 host memory for read-backs, kept by the program."""
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def _fields(case):
    """The maps a program reads back: all of the state on ordinary grids, the depth and its
    maximum on the largest."""
    if case["kind"] == "stages":
        return ["depth", "dmax"]
    f = ["depth", "dmax"]
    if case["ny"] * case["nx"] <= 8_000_000:
        f += ["qout_right", "qout_up"]
    if case["soil"]:
        f += ["soil_storage"]
    if case["hazard"]:
        f += ["vmax", "hazard_max"]
    return f


def _member_sites(case, seed):
    """Members with grid sides log-uniform in [lo, hi], multiples of 32; a share of them dam-break
    valleys, the others rain on a V-tilted catchment.  The sides and the kinds belong to the case,
    terrain and forcing come from the seed."""
    rng = np.random.default_rng([case["members"], case["lo"], case["hi"], case["steps"]])
    for m in range(case["members"]):
        ny, nx = (int(32 * round(math.exp(v) / 32)) for v in rng.uniform(math.log(case["lo"]), math.log(case["hi"]), 2))
        breach = rng.uniform() < case["breach"]
        spec = dict(ny=ny, nx=nx, terrain="valley" if breach else "vtilt", depth=0.0 if breach else 5.0,
                    share=float(rng.uniform(0.05, 0.5)), soil=False, rain="none" if breach else "uniform")
        yield _site(spec, seed * 1009 + m)


def _network_batch(case, seed):
    """Normalised member inputs [B, H, W, 4] (BF16) and targets / weights [B H W, 2] (FP32)."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    B, H, W = case["batch"], case["height"], case["width"]
    x = torch.zeros(B, H, W, 4, device=DEV)
    t = torch.zeros(B, H, W, 2, device=DEV)
    for b in range(B):
        x[b, ..., 0] = _field(H, W, gen).float()
        n, rain = torch.rand(2, generator=gen, device=DEV)
        x[b, ..., 1] = 0.28 + 0.24 * n
        x[b, ..., 2] = 0.1 + 2.0 * rain
        t[b, ..., 0] = torch.clamp(2.0 - x[b, ..., 0] + rain, min=0.0)
        t[b, ..., 1] = torch.clamp(0.5 + 0.3 * x[b, ..., 0], 0.0, 1.5)
    w = 0.1 + 0.9 * (t[..., 1:] < 1.5).float().expand(-1, -1, -1, 2)
    return x.to(torch.bfloat16), t.reshape(-1, 2).contiguous(), w.reshape(-1, 2).contiguous()


def _layer_spec(case):
    """Channels and spatial size of the case's layer in the network."""
    name, ci, co, relu = next(s for s in unet_spec() if s[0] == case["layer"])
    lvl = layer_level(name)
    return name, ci, co, relu, case["height"] >> lvl, case["width"] >> lvl


def _layer_batch(case, seed):
    name, ci, co, relu, H, W = _layer_spec(case)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(case["batch"], H, W, ci, generator=gen, device=DEV)
    if name != "enc0a":
        x = torch.relu(x)   # the layer before ends in a ReLU
    dy = 0.01 * torch.randn(case["batch"], H, W, co, generator=gen, device=DEV)
    return x.to(torch.bfloat16), dy.to(torch.bfloat16)


def _layer(case, seed):
    name, ci, co, relu, _, _ = _layer_spec(case)
    return Conv3x3(name, ci, co, relu, torch.Generator().manual_seed(seed), DEV)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("run", "stages"):
        sf = _flow(_site(case, seed), case["precision"])
        if case["hazard"]:
            sf.set_hazard_tracking(True)
        ny, nx = case["ny"], case["nx"]
        maps = {f: _pinned(ny * nx).reshape(ny, nx) for f in _fields(case)}
        return dict(kind=kind, sf=sf, steps=case["steps"], maps=maps)
    if kind == "ensemble":
        ens = Ensemble()
        for site in _member_sites(case, seed):
            ens.add(_flow(site, "fp32"))
        flat = _pinned(ens.cells())
        maps, at = [], 0
        for m in ens.members:
            maps.append(flat[at:at + m.ny * m.nx].reshape(m.ny, m.nx))
            at += m.ny * m.nx
        return dict(kind=kind, ens=ens, steps=case["steps"], flat=flat, maps=maps)
    if kind in ("predict", "train"):
        x, t, w = _network_batch(case, seed)
        return dict(kind=kind, net=UNet(seed=seed), x=x, t=t, w=w)
    x, dy = _layer_batch(case, seed)
    return dict(kind=kind, layer=_layer(case, seed), x=x, dy=dy)


def _run_stages(sf, steps):
    """The main loop of the reference: one call per function, the clock kept by the caller."""
    d = sf.diag()
    t, ts, k = d["t"], d["time_step"], d["k"]
    for _ in range(steps):
        sf.hydrology_step(ts)
        sf.li_step(ts)
        new, vmax = sf.cfl_dt()
        sf.track_maxima(t + ts)
        t, ts, k = t + new, new, k + 1
        sf.set_clock(t, ts, k)
    return t, ts, k, vmax


def run(state):
    kind = state["kind"]
    if kind == "run":
        sf = state["sf"]
        sf.fused_steps(state["steps"])
        out = {f: sf.download_into(f, buf) for f, buf in state["maps"].items()}
        d = sf.diag()
        out["clock"] = [d["t"], d["time_step"], d["k"]]
        out["volumes"] = [d["rain_volume"], d["infiltration_volume"], d["outlet_volume"]]
        return out
    if kind == "stages":
        sf = state["sf"]
        t, ts, k, vmax = _run_stages(sf, state["steps"])
        out = {f: sf.download_into(f, buf) for f, buf in state["maps"].items()}
        out["clock"] = [t, ts, k]
        out["max_velocity"] = vmax
        return out
    if kind == "ensemble":
        ens = state["ens"]
        ens.steps(state["steps"])
        for m, buf in zip(ens.members, state["maps"]):
            m.download_into("dmax", buf)
        return {"dmax": state["flat"]}
    if kind == "predict":
        return state["net"].predict(state["x"])
    if kind == "train":
        net = state["net"]
        loss = net.train_step(state["x"], state["t"], state["w"], 1e-4)
        return {"loss": loss, "grads": {n: [c.gW, c.gb] for n, c in net.layers.items()}}
    c = state["layer"]
    c.gW.zero_()
    c.gb.zero_()
    y = c.forward(state["x"])
    dx = c.backward(state["dy"])
    return {"y": y, "dx": dx, "gW": c.gW, "gb": c.gb}


def work(case):
    kind = case["kind"]
    if kind in ("run", "stages"):
        R = 4 if case["precision"] == "fp32" else 8
        cells = case["ny"] * case["nx"]
        wet = cells if case["terrain"] != "valley" else cells * case["share"] * math.sqrt(0.5)
        if kind == "stages":
            # hydrology h in/out; routing h, q_x, q_y, z, n in, h, q_x, q_y, two face depths out;
            # time step four face arrays in; maxima h, dmax in, dmax out
            per = 19 * R + (5 * R if case["soil"] else 0)
        else:
            # h, q_x, q_y, dmax, z, n in and h, q_x, q_y, dmax out; soil storage and timer in and
            # out, the class in; two maxima in and out
            per = 10 * R + (4 * R + 1 if case["soil"] else 0) + (4 * R if case["hazard"] else 0)
        return dict(bytes=float(per * wet * case["steps"] + 8 * cells * len(_fields(case))),
                    flops=float(150 * wet * case["steps"]))
    if kind == "ensemble":
        side2 = ((case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])) ** 2 if case["hi"] > case["lo"] else case["lo"] ** 2
        cells = case["members"] * side2 * (1.0 - 0.8 * case["breach"])
        return dict(bytes=float((40 * case["steps"] + 8) * cells), flops=float(150 * cells * case["steps"]))
    if kind in ("predict", "train"):
        P = case["batch"] * case["height"] * case["width"]
        f = forward_flops(case["height"], case["width"]) * case["batch"]
        # the activations between layers (BF16, channels x resolution) once in and once out
        act = sum(2 * (ci + co) * P / 4 ** layer_level(n) for n, ci, co, _ in unet_spec())
        return dict(bytes=float(act * (3 if kind == "train" else 1)), flops=float(f * (3 if kind == "train" else 1)))
    _, ci, co, _, H, W = _layer_spec(case)
    P = case["batch"] * H * W
    return dict(bytes=float(2 * P * (2 * ci + 2 * co) + 12 * 9 * ci * co), flops=float(3 * 2 * P * 9 * ci * co))


# ---------------------------------------------------------------------------------------------
# 64-bit restatement
# ---------------------------------------------------------------------------------------------
def _pad(a, left, right, dim):
    shape = list(a.shape)
    parts = []
    if left:
        parts.append(a.new_zeros([1 if d == dim else s for d, s in enumerate(shape)]))
    n = a.shape[dim]
    parts.append(a.narrow(dim, 1 if right else 0, n - 1))
    if right:
        parts.append(a.new_zeros([1 if d == dim else s for d, s in enumerate(shape)]))
    return torch.cat(parts, dim)


def _left(a):    # value of the cell to the left (0 on the first column)
    return _pad(a, True, False, 1)


def _right(a):
    return _pad(a, False, True, 1)


def _above(a):
    return _pad(a, True, False, 0)


def _below(a):
    return _pad(a, False, True, 0)


def _map_depth(maps, a, b, ny, nx):
    """Rain depth [m] of the maps (5 min each) over [a, b] min, bilinear at the cell centres."""
    out = 0.0
    for m in range(maps.shape[0]):
        ov = min(b, 5.0 * (m + 1)) - max(a, 5.0 * m)
        if ov > 0:
            f = F.interpolate(maps[m].double()[None, None], size=(ny, nx), mode="bilinear", align_corners=False)[0, 0]
            out = out + f * (ov / 60000.0)
    return out


class _Exact:
    """The surface-flow step in 64 bits: local-inertial fluxes, draining limiter, continuity,
    outlet sink, Green-Ampt infiltration, rain of the lagged clock interval, CFL time step."""

    def __init__(self, site):
        self.s, self.dx, p = site, site["dx"], site["params"]
        z = site["z"]
        self.ny, self.nx = z.shape
        self.n2 = site["rough"] ** 2
        self.amin, self.amax = p["alfa_min"], p["alfa_max"]
        zx = _right(z)
        zx[:, -1] = math.inf
        zy = _above(z)
        zy[0] = math.inf
        self.dzx, self.dzy = zx - z, zy - z
        self.h = site["d0"] / 1000.0
        self.qx, self.qy = torch.zeros_like(z), torch.zeros_like(z)
        self.dmax = torch.full_like(z, -math.inf)
        self.t, self.ts, self.k, self.tsp = 0.01 / 60, 0.01 / 60, 1, 0.0
        self.ra, self.rb, self.tp = 0.0, 0.01 / 60, 0.0
        self.out = (torch.as_tensor(site["rows"].astype(np.int64), device=DEV), torch.as_tensor(site["cols"].astype(np.int64), device=DEV))
        rough_o = site["rough"][self.out]
        self.coef = math.sqrt(p["slope_outlet"]) / (rough_o * self.dx) if p["outlet_type"] == 1 else torch.full_like(rough_o, math.sqrt(9.81) / self.dx)
        self.otype = p["outlet_type"]
        if site["soil"] is not None:
            tab = {k: torch.as_tensor(v, device=DEV, dtype=torch.float64)[site["soil"]["cls"]] for k, v in site["soil"]["tables"].items()}
            self.soil = dict(ks=tab["ksat"] / 3.6e6, psi=tab["psi"] / 1000, dth=tab["dtheta"], lu=tab["Lu"],
                             kout=tab["k_out"] / 3.6e6, tr=tab["Tr"] * 3600, minsm=tab["min_soil_moisture"] / 1000)
            self.I, self.T = torch.full_like(z, 0.005), self.soil["tr"].clone()
        self.rows01 = torch.zeros_like(z)

    def face(self, ha, hb, dz, q, x):
        dt = self.ts * 60
        closed = torch.isinf(dz)
        d = torch.where(closed, torch.zeros_like(dz), dz)
        if x:
            H = torch.maximum(ha - d.clamp(min=0), hb + d.clamp(max=0)).clamp(min=0)
            S = (d + (hb - ha)) / self.dx
        else:
            H = torch.maximum(ha + d.clamp(max=0), hb - d.clamp(min=0)).clamp(min=0)
            S = (d + (ha - hb)) / self.dx
        H = torch.where(closed, torch.zeros_like(H), H)
        h73 = H ** (7.0 / 3.0)
        new = (q - 9.81 * dt * H * S) * h73 / (9.81 * dt * self.n2 * q.abs() + h73)
        new = torch.where(H > 0, new, torch.zeros_like(new))
        return H, torch.clamp(new, -10 * H, 10 * H)

    def hydrology(self):
        s, h, dt = self.s, self.h, self.ts * 60
        if s["rate"] is not None:
            h = h + s["rate"] * max(0.0, self.rb - self.ra) / 60000.0
        elif s["maps"] is not None:
            h = h + _map_depth(s["maps"], self.ra, self.rb, self.ny, self.nx)
        if s["soil"] is not None:
            q = self.soil
            ia = h / dt
            C = torch.where(self.I > q["lu"], q["ks"], q["ks"] * (1 + (h + q["psi"]) * q["dth"] / self.I))
            T = torch.where(ia > C, q["tr"], self.T - dt)
            f = torch.minimum(C, ia)
            I = torch.maximum(self.I + f * dt - torch.where(ia <= C, q["kout"] * dt, torch.zeros_like(f)), q["minsm"])
            self.I, self.T = torch.where(T < 0, q["minsm"], I), T
            h = (h - f * dt).clamp(min=0)
        self.h = torch.where(h < 1e-9, torch.zeros_like(h), h)

    def step(self):
        dt, h = self.ts * 60, None
        self.hydrology()
        h = self.h
        hfx, qx = self.face(h, _right(h), self.dzx, self.qx, True)
        hfy, qy = self.face(_above(h), h, self.dzy, self.qy, False)
        out = qx.clamp(min=0) + (-_left(qx)).clamp(min=0) + qy.clamp(min=0) + (-_below(qy)).clamp(min=0)
        avail = h * (self.dx / dt)
        sc = torch.where(out > avail, avail / out, torch.ones_like(out))
        qx = torch.where(qx > 0, qx * sc, qx * _right(sc))
        qy = torch.where(qy > 0, qy * sc, qy * _above(sc))
        h = (h + dt / self.dx * (_left(qx) - qx - qy + _below(qy))).clamp(min=0)
        ho = h[self.out]
        qo = torch.minimum(self.coef * (ho ** (5.0 / 3.0) if self.otype == 1 else ho * torch.sqrt(ho)), ho / dt)
        h[self.out] = ho - qo * dt
        hf3 = torch.zeros_like(h)
        hf3[self.out] = ho
        self.h, self.qx, self.qy = h, qx, qy
        self.dmax = torch.maximum(self.dmax, h)
        self.advance(self.refresh(hfx, hfy, hf3))

    def refresh(self, hfx, hfy, hf3):
        save = (math.ceil(self.t * 60 / 1e-4) - 1.0) * 1e-4 / 60
        delta, self.tsp = save - self.tsp, save
        if not (delta > 0 or self.k == 1):
            return self.ts * 60
        tol, big = 0.001, 1e9
        vr = self.qx / torch.where(hfx < tol, big, hfx)
        vu = self.qy / torch.where(hfy < tol, big, hfy)
        rc = vr.clone()
        rc[:, 0] *= 0.5
        sp = torch.hypot(rc, 0.5 * (vu + _below(vu)))
        vmax = float(sp.max())
        wc = torch.sqrt(9.81 * torch.maximum(torch.maximum(hfx, hfy), hf3)).clamp(min=1e-10)
        cmax = float(torch.where(sp < 0.01, torch.zeros_like(wc), wc).max())
        adv = min(self.dx / vmax * max(self.amax - 2 * max(vmax - 5.0, 0.0), self.amin), 10.0) if vmax > 0 else 10.0
        new = min(adv, self.amin * self.dx / cmax if cmax > 0 else 10.0)
        return min(max(0.001 * math.floor(new / 0.001), 0.01), 10.0)

    def advance(self, dt):
        self.ra, self.rb, self.tp = self.tp, self.t, (dt / 60 if self.k == 1 else self.t)
        self.ts = dt / 60
        self.t += self.ts
        self.k += 1

    def fields(self, names):
        mmh = 3.6e6 / self.dx
        got = dict(depth=lambda: self.h * 1000, dmax=lambda: self.dmax * 1000, qout_right=lambda: self.qx * mmh,
                   qout_up=lambda: self.qy * mmh, soil_storage=lambda: self.I * 1000)
        return {f: got[f]() if f in got else None for f in names}


def _conv64(x, W, b, ci):
    """3x3 convolution of NCHW x with weights [co, >= 9 ci] (K index (ky*3 + kx)*ci + c)."""
    k = W[:, :9 * ci].reshape(-1, 3, 3, ci).permute(0, 3, 1, 2)
    return F.conv2d(x, k, b, padding=1)


def _net64(net, x, weights):
    """The network's forward pass in 64 bits with `weights` {name: (W, b)}."""
    def conv(name, v):
        c = net.layers[name]
        y = _conv64(v, weights[name][0], weights[name][1], c.ci)
        return torch.relu(y) if c.relu else y
    h, skips = x.double().permute(0, 3, 1, 2), []
    for lvl in range(net.levels):
        h = conv(f"enc{lvl}b", conv(f"enc{lvl}a", h))
        if lvl < net.levels - 1:
            skips.append(h)
            h = F.max_pool2d(h, 2)
    for lvl in range(net.levels - 2, -1, -1):
        u = conv(f"up{lvl}", h.repeat_interleave(2, 2).repeat_interleave(2, 3))
        h = conv(f"dec{lvl}b", conv(f"dec{lvl}a", torch.cat([u, skips[lvl]], 1)))
    return conv("head", h).permute(0, 2, 3, 1).reshape(-1, 2)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("run", "stages"):
        e = _Exact(_site(case, seed))
        for _ in range(case["steps"]):
            e.step()
        out = e.fields(_fields(case))
        out["clock"] = [None, None, None]
        if kind == "run":
            out["volumes"] = [None, None, None]
        else:
            out["max_velocity"] = None
        return out
    if kind == "ensemble":
        got = []
        for site in _member_sites(case, seed):
            e = _Exact(site)
            for _ in range(case["steps"]):
                e.step()
            got.append(e.dmax.reshape(-1) * 1000)
        return {"dmax": torch.cat(got)}
    if kind == "predict":
        x, _, _ = _network_batch(case, seed)
        net = UNet(seed=seed)
        w = {n: (c.W16.double(), c.b.double()) for n, c in net.layers.items()}
        with torch.no_grad():
            return torch.cat([_net64(net, x[b:b + 4], w) for b in range(0, x.shape[0], 4)])
    if kind == "train":
        x, t, wt = _network_batch(case, seed)
        net = UNet(seed=seed)
        w = {n: tuple(v.double().requires_grad_() for v in (c.W16, c.b)) for n, c in net.layers.items()}
        per = case["height"] * case["width"]
        total = 0.0
        for b in range(0, x.shape[0], 2):
            sl = slice(b * per, min(b + 2, x.shape[0]) * per)
            loss = (wt[sl].double() * (_net64(net, x[b:b + 2], w) - t[sl].double()) ** 2).sum() / t.numel()
            loss.backward()
            total = total + loss.detach()
        return {"loss": total.reshape(1), "grads": {n: [v[0].grad, v[1].grad] for n, v in w.items()}}
    x, dy = _layer_batch(case, seed)
    c = _layer(case, seed)
    B, H, W, ci = x.shape
    xx = x.double().permute(0, 3, 1, 2)
    W64 = c.W16.double()
    gW, gb, y, dx = torch.zeros_like(W64), torch.zeros(c.co, device=DEV, dtype=torch.float64), [], []
    for b in range(B):
        xb, wb, bb = xx[b:b + 1].requires_grad_(), W64.clone().requires_grad_(), c.b.double().requires_grad_()
        yb = _conv64(xb, wb, bb, ci)
        yb = torch.relu(yb) if c.relu else yb
        yb.backward(dy[b:b + 1].double().permute(0, 3, 1, 2))
        gW, gb = gW + wb.grad, gb + bb.grad
        y.append(yb.detach())
        dx.append(xb.grad)
    nhwc = lambda v: torch.cat(v).permute(0, 2, 3, 1).contiguous()  # noqa: E731
    return {"y": nhwc(y), "dx": nhwc(dx), "gW": gW, "gb": gb}
