"""Workloads of the lattice engine, as the programs that use it run them.

Every case is one output interval (or one training step) of such a program:
a call of the integrator followed by what the program reads back at that
point.  The engine is driven through its public Python binding only.

``listed()``  the workloads at fixed sizes; ``draw(rng)`` one more of the same
kinds; ``prepare`` the state a program holds before the call; ``run`` one pass;
``work`` the bytes and operations the pass cannot do without; ``exact`` the
same outputs in plain torch FP64.

Kinds
-----
fd        finite-difference lattices (7 and 27 points, GW strains, expansion):
          steps, then the energies and optionally P(k) and the GW spectrum
spectral  pseudospectral lattices: steps, then the energies and P(k)
host      a driver that keeps its fields in host arrays (Fortran layout,
          pinned): upload, steps, energies, download
output    the analysis output of an evolved lattice: energies, power and cross
          spectra, shell counts
ensemble  a batch of independent runs of uneven sizes
closure   a coarse lattice evolved with the learned closure attached
train     one training step of the closure network
"""
from __future__ import annotations

import ctypes
import importlib
import math
import random

import numpy as np
import torch

L = importlib.import_module("lattice-dev_gb300")

F64, KAHAN = L.FP64, L.FP32_KAHAN


# ------------------------------------------------------------------- cases
def listed():
    return [
        # The plain method: phi^4, 64^3, 7 points, leapfrog, FP64, an energy record and a
        # 32-bin P(k) every ten steps; the launch shapes tuned once, as the README's program does.
        dict(name="fd7_phi4_64_fp64", kind="fd", nx=64, ny=64, nz=64, nfld=1, lap=7, conformal=False, gw=False,
             kahan=False, order=2, steps=10, bins=32, tune=True),
        # The smallest lattice in use (the oracle-checked 32^3 expanding runs): a driver that
        # advances one Yoshida-4 step at a time and follows the scale factor.
        dict(name="preheat_32_fp64_step", kind="spectral", nx=32, ny=32, nz=32, nfld=2, conformal=True, kahan=False,
             order=4, steps=1, bins=0, record="a", separable=False, tune=False),
        # The headline run: two-field preheating at 256^3, FP32 with Kahan drifts, on the
        # streamed passes (what the autotuner picks there), an energy record every four steps.
        dict(name="preheat_256_kahan", kind="spectral", nx=256, ny=256, nz=256, nfld=2, conformal=True, kahan=True,
             order=4, steps=4, bins=0, record="energies", separable=True, tune=False),
        # The same run in the reference's own arithmetic (-r8), one step per record.
        dict(name="preheat_256_fp64", kind="spectral", nx=256, ny=256, nz=256, nfld=2, conformal=True, kahan=False,
             order=4, steps=1, bins=0, record="energies", separable=False, tune=True),
        # One field on a box of uneven, not power-of-two sides, FP64, with its P(k).
        dict(name="phi4_ragged_fp64", kind="spectral", nx=150, ny=108, nz=96, nfld=1, conformal=False, kahan=False,
             order=4, steps=2, bins=48, record="energies", separable=False, tune=False),
        # Bubble collision with GW sourcing at its full size: leapfrog steps between outputs.
        dict(name="bubbles_gw_512_kahan", kind="fd", nx=512, ny=512, nz=512, nfld=1, lap=27, conformal=False, gw=True,
             kahan=True, order=2, steps=4, bins=0, tune=True, record="none"),
        # A smaller collision in FP64 on a box of ragged sides, with the full output record
        # (energies and the TT-projected GW spectrum) at the end of the interval.
        dict(name="bubbles_gw_ragged_fp64", kind="fd", nx=144, ny=100, nz=90, nfld=1, lap=27, conformal=False, gw=True,
             kahan=False, order=2, steps=5, bins=48, tune=False),
        # A Fortran driver with host-resident fields: up, ten leapfrog steps, energies, down.
        dict(name="host_phi4_128_kahan", kind="host", nx=128, ny=128, nz=128, nfld=1, conformal=False, kahan=True,
             order=2, steps=10),
        # The analysis output of the two-field run (energy_spec.out and spectrum.out records):
        # energies, P(phi), P(chi), P(pi), the cross spectrum and the shell counts.
        dict(name="output_256_kahan", kind="output", nx=256, ny=256, nz=256, nfld=2, conformal=True, kahan=True,
             bins=128),
        # Seeds of one model on lattices of uneven size advanced together (a quarter of the
        # 96-run ensemble), with every run's energies and P(k) of one run per size.
        dict(name="ensemble_24_kahan", kind="ensemble", n64=8, n96=8, n128=6, n192=2, kahan=True, order=4, steps=4,
             bins=32),
        # The coarse lattice with the learned closure in its kick.
        dict(name="closure_64_kahan", kind="closure", nx=64, ny=64, nz=64, conformal=True, kahan=True, order=4,
             steps=5, every=3),
        # One Adam step of the closure network on a batch of four 64^3 samples.
        dict(name="train_64_batch4", kind="train", nx=64, ny=64, nz=64, batch=4),
    ]


def _side(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng: random.Random):
    kind = rng.choice(["fd", "fd", "spectral", "spectral", "spectral", "host", "output", "ensemble", "closure",
                       "train"])
    kahan = rng.random() < 0.5
    if kind == "fd":
        gw = rng.random() < 0.5
        top = 256 if kahan else 192
        n = [_side(rng, 24, top) for _ in range(3)]
        if rng.random() < 0.5:
            n = [max(32, n[0] // 32 * 32)] * 3
        conf = not gw and rng.random() < 0.5
        return dict(kind="fd", nx=n[0], ny=n[1], nz=n[2], nfld=2 if conf else 1, lap=rng.choice([7, 27]),
                    conformal=conf, gw=gw, kahan=kahan, order=rng.choice([2, 2, 4]), steps=rng.randint(2, 20),
                    bins=rng.choice([0, 32, 48]), tune=rng.random() < 0.3)
    if kind == "spectral":
        nfld = rng.choice([1, 2])
        conf = rng.random() < 0.5
        if rng.random() < 0.6:  # the power-of-two boxes most runs use, sides equal or not
            sides = [32, 64, 128, 256]
            n = [rng.choice(sides)] * 3 if rng.random() < 0.6 else [rng.choice(sides) for _ in range(3)]
        else:
            n = [_side(rng, 24, 200, rng.choice([1, 2, 4, 6])) for _ in range(3)]
        big = n[0] * n[1] * n[2] > 1 << 22
        return dict(kind="spectral", nx=n[0], ny=n[1], nz=n[2], nfld=nfld, conformal=conf, kahan=kahan,
                    order=rng.choice([2, 4, 4, 6]), steps=rng.randint(1, 2 if big else 6),
                    bins=rng.choice([0, 0, 32]), record="energies", separable=False, tune=rng.random() < 0.5)
    if kind == "host":
        n = [_side(rng, 32, 160, rng.choice([1, 2, 8])) for _ in range(3)]
        return dict(kind="host", nx=n[0], ny=n[1], nz=n[2], nfld=rng.choice([1, 2]), conformal=rng.random() < 0.5,
                    kahan=kahan, order=rng.choice([2, 4]), steps=rng.randint(1, 10))
    if kind == "output":
        n = [_side(rng, 48, 224, rng.choice([1, 2, 8])) for _ in range(3)]
        return dict(kind="output", nx=n[0], ny=n[1], nz=n[2], nfld=rng.choice([1, 2]), conformal=rng.random() < 0.5,
                    kahan=kahan, bins=rng.choice([32, 64, 100]))
    if kind == "ensemble":
        return dict(kind="ensemble", n64=2 * rng.randint(1, 10), n96=2 * rng.randint(0, 8), n128=2 * rng.randint(0, 5),
                    n192=2 * rng.randint(0, 2), kahan=rng.random() < 0.8, order=rng.choice([2, 4]),
                    steps=rng.randint(1, 4), bins=32)
    if kind == "closure":
        n = rng.choice([32, 48, 64, 64, 96, 128])
        return dict(kind="closure", nx=n, ny=n, nz=n, conformal=rng.random() < 0.7, kahan=kahan or n > 64, order=4,
                    steps=rng.randint(1, 5), every=rng.randint(1, 3))
    return dict(kind="train", nx=16 * rng.randint(1, 6), ny=8 * rng.randint(3, 10), nz=_side(rng, 16, 80),
                batch=rng.randint(1, 5))


# ----------------------------------------------------------- configurations
AMP, KCUT = 1e-8, 0.5
DEL = 0.01       # tilt of the double well
KAPPA = 2.0      # GW coupling
LR = 5e-4


def _shape(c):
    return c["nx"], c["ny"], c["nz"]


def _two(c):
    return c.get("nfld", 2) == 2


def _length(c):
    if c["kind"] == "fd":
        return c["nx"] / 4.0 if c["gw"] else 20.0
    return 10 * math.pi if _two(c) else 20.0


def _dt(c):
    return _length(c) / c["nx"] / (10 if c["order"] == 2 else 20)


def _config(c):
    fd = c["kind"] == "fd"
    well = fd and c["gw"]
    return L.make_config(
        _shape(c), nfld=2 if _two(c) else 1, length=_length(c),
        laplacian=c["lap"] if fd else L.LAP_SPECTRAL,
        background=L.BG_CONFORMAL if c["conformal"] else L.BG_MINKOWSKI,
        precision=KAHAN if c["kahan"] else F64,
        split_order=L.SPLIT_DEFROST if well else L.SPLIT_PSEUDOSPEC,
        model=L.MODEL_DOUBLE_WELL if well else (L.MODEL_PHI4_G2 if _two(c) else L.MODEL_PHI4),
        model_params=(DEL,) if well else ((1.0, 2.0) if _two(c) else (1.0,)),
        gw=well, gw_coupling=KAPPA if well else 0.0,
        spectral_impl=L.SPEC_IMPL_SEPARABLE if c.get("separable") else L.SPEC_IMPL_AUTO)


def _means(c):
    """Homogeneous fields and momenta (a generic phase of the oscillation) and effective masses of the draw."""
    return ([0.8, 0.0], [-0.5, 0.0], [3.0, 2.0]) if _two(c) else ([0.8], [-0.5], [3.0])


def _bubbles(c, seed):
    """Centres (1-based sites), nucleation radius and age of a pair of expanding bubbles, displaced by the seed."""
    r = np.random.default_rng(seed)
    n = np.array(_shape(c))
    at = np.array([[0.34375, 0.5, 0.5], [0.65625, 0.5, 0.5]]) + r.uniform(-0.03, 0.03, (2, 3))
    return np.floor(at * n).astype(np.int32) + 1, 0.0625 * float(n.min()) / 4.0, 0.0625 * float(n.min()) / 4.0


def _start(c, g, seed):
    if c["kind"] == "fd" and c["gw"]:
        g.init_bubbles_boosted(*_bubbles(c, seed), -1.0, 1.0)
        return
    f0, d0, m2 = _means(c)
    g.init_vacuum(seed, f0, d0, m2, amp=AMP, kcut_frac=KCUT)
    if c["conformal"]:
        g.set_scale_factor(1.0, 0.0)
        g.calc_metric()


class _DeviceView:
    """The engine's device buffer as a CUDA array; keeps the lattice alive."""

    def __init__(self, g, ptr, shape, typestr):
        self.g = g
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(ptr, False), version=3, strides=None)


def _view(s, what):
    """Zero-copy tensor of the current fields (0) or momenta (1); made once per buffer."""
    g = s["g"]
    p = g.device_ptr(what)
    v = s["views"].get(p)
    if v is None:
        kind = "<f4" if s["case"]["kahan"] else "<f8"
        v = torch.as_tensor(_DeviceView(g, p, (g.nfld, g.nz, g.ny, g.nx), kind), device="cuda")
        s["views"][p] = v
    return v


ENS_SIZES = (64, 96, 128, 192)


def _ens_sizes(c):
    return [n for n in ENS_SIZES for _ in range(c["n%d" % n])]


def _ens_seeds(c, seed):
    return [(seed * 1000 + i) & 0x7FFFFFFF for i in range(len(_ens_sizes(c)))]


def _net_params(seed):
    """Random weights of the network at the scale training leaves them, padded channels zero."""
    r = np.random.default_rng(seed)
    w1 = r.standard_normal((27, 8, 32)) / math.sqrt(27 * 4)
    w1[:, 4:] = 0.0
    w2 = r.standard_normal((27, 32, 32)) / math.sqrt(27 * 32)
    w3 = r.standard_normal((27, 32, 8)) / math.sqrt(27 * 32)
    w3[:, :, 2:] = 0.0
    b1, b2, b3 = 0.05 * r.standard_normal(32), 0.05 * r.standard_normal(32), 0.05 * r.standard_normal(8)
    b3[2:] = 0.0
    return np.concatenate([v.ravel() for v in (w1, b1, w2, b2, w3, b3)]).astype(np.float32)


# normalisation of the network's inputs (phi, chi, pi_phi, pi_chi) and outputs on the preheating fields
NORM = (np.zeros(4), np.array([1.4, 3000.0, 1.8, 400.0]), np.array([2.0e4, 4.0e5]))


def _samples(c, seed):
    """A batch of training samples [batch][6][nz][ny][nx]: smooth fields and a force correlated with them."""
    nx, ny, nz = _shape(c)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(c["batch"], 4, nz, ny, nx, device="cuda", generator=gen, dtype=torch.float64)
    for d in (2, 3, 4):
        x = (x + torch.roll(x, 1, d) + torch.roll(x, -1, d)) / math.sqrt(3.0)
    y = torch.stack([x[:, 0] ** 2 * x[:, 1] - x[:, 2], x[:, 0] * x[:, 1] + 0.3 * x[:, 3]], 1)
    scale = torch.as_tensor(np.concatenate([1 / NORM[1], 1 / NORM[2]]), device="cuda").view(1, 6, 1, 1, 1)
    return (torch.cat([x, y], 1) * scale).float()


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    c = case
    s = dict(case=c, views={})
    if c["kind"] == "train":
        nx, ny, nz = _shape(c)
        s["net"] = L.Net(seed=1)
        s["net"].set_params(_net_params(seed))
        s["net"].set_norm(*NORM)
        host = _samples(c, seed).cpu().numpy()
        s["data"] = L.DeviceArray(host.size)
        s["data"].upload(host)
        s["stride"] = 6 * nx * ny * nz
        s["idx"] = list(range(c["batch"]))
        return s
    if c["kind"] == "ensemble":
        base = L.make_config(64, nfld=1, length=20.0, laplacian=L.LAP_SPECTRAL,
                             precision=KAHAN if c["kahan"] else F64, model=L.MODEL_PHI4, model_params=(1.0,))
        sizes = _ens_sizes(c)
        s["ens"] = L.Ensemble(base, sizes)
        s["ens"].init_vacuum(_ens_seeds(c, seed), 0.8, -0.5, 3.0, amp=AMP, kcut_frac=KCUT)
        s["ens"].prepare_symp(c["order"], 1.0 / 20, c["steps"])
        s["ens"].sync()
        s["shown"] = [sizes.index(n) for n in ENS_SIZES if n in sizes]
        return s
    g = s["g"] = L.Lattice(_config(c))
    _start(c, g, seed)
    if c["kind"] == "closure":
        net = s["net"] = L.Net(seed=1)
        net.set_params(_net_params(seed))
        net.set_norm(*NORM)
        g.attach_closure(net, c["every"], L.UNITS_CONFORMAL if c["conformal"] else L.UNITS_PROGRAM)
    if c.get("tune"):
        g.autotune(None)
    if c["kind"] == "output":
        c2 = dict(c, order=2)
        g.symp(2, _dt(c2), 2)
        g.sync()
        return s
    g.prepare_symp(c["order"], _dt(c), c["steps"])
    if c["kind"] == "host":
        n = g.nfld * g.N
        s["mem"] = [_Pinned(8 * n) for _ in range(2)]
        s["arr"] = [m.array((g.nz, g.ny, g.nx, g.nfld)) for m in s["mem"]]
        g.download_fortran(s["arr"][0], 0, 0, s["arr"][1], 0, 0)
    g.sync()
    return s


class _Pinned:
    """Pinned host memory of the engine (the program's own field arrays)."""

    def __init__(self, nbytes):
        self.nbytes = nbytes
        self.ptr = L.host_alloc(nbytes)

    def array(self, shape):
        buf = (ctypes.c_double * (self.nbytes // 8)).from_address(self.ptr)
        buf.owner = self  # the memory lives as long as an array of it does
        return np.ctypeslib.as_array(buf).reshape(shape)

    def __del__(self):
        if getattr(self, "ptr", None):
            L.host_free(self.ptr)
            self.ptr = None


# --------------------------------------------------------------------- run
def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "train":
        loss = s["net"].train_step(s["data"], s["stride"], s["idx"], _shape(c), LR)
        return {"loss": loss, "params": s["net"].params()}
    if kind == "ensemble":
        e = s["ens"]
        e.symp(c["order"], 1.0 / 20, c["steps"])
        out = {"energies": e.energies()}
        for r in s["shown"]:
            out["S%d" % r], out["W%d" % r] = e.spectrum(r, c["bins"])
        return out
    g = s["g"]
    if kind == "output":
        nb = c["bins"]
        out = {"energies": g.energies()}
        for f in range(g.nfld):
            out["fld%d" % f] = list(g.spectrum(L.SPEC_FLD, f, L.SPEC_WEIGHTED, nb))
        out["fldp0"] = g.spectrum_3d(L.SPEC_FLDP, 0, nb)
        out["cross"] = list(g.crossspec_3d(L.SPEC_FLDP, 0, L.SPEC_FLD, 0, nb))
        out["count"] = list(g.spectrum_bin(L.SPEC_FLD, 0, nb))
        return out
    if kind == "host":
        f, p = s["arr"]
        g.upload_fortran(f, 0, 0, p, 0, 0)
        g.symp(c["order"], _dt(c), c["steps"])
        e = g.energies()
        g.download_fortran(f, 0, 0, p, 0, 0)
        return {"energies": e, "fld": f, "fldp": p}
    g.symp(c["order"], _dt(c), c["steps"])
    out = {}
    record = c.get("record", "energies")
    if record == "energies":
        out["energies"] = g.energies()
    elif record == "a":
        out["a"] = list(g.scale_factor())
    if c.get("bins"):
        if kind == "fd" and c["gw"]:
            out["gw"] = list(g.gw_spectrum(c["bins"]))
        else:
            out["pk"] = list(g.spectrum(L.SPEC_FLD, 0, L.SPEC_WEIGHTED, c["bins"]))
    out["fld"], out["fldp"] = _view(s, 0), _view(s, 1)
    return out


# -------------------------------------------------------------------- work
KICKS = {2: 1, 4: 3, 6: 7}


def work(case):
    """Bytes: the state read and written once per kick (the kick couples all sites, so the next one needs it
    complete), the fields once more per output.  Operations: the stencil or the transforms."""
    c = case
    if c["kind"] == "train":
        n = c["nx"] * c["ny"] * c["nz"] * c["batch"]
        return {"bytes": 24.0 * n + 6 * 4 * 41544, "flops": 3.0 * 65664 * n}
    if c["kind"] == "ensemble":
        b = fl = 0.0
        rw = 24 if c["kahan"] else 32
        for n in _ens_sizes(c):
            kicks = KICKS[c["order"]] * c["steps"]
            b += n ** 3 * (rw * kicks + rw / 3)
            fl += kicks * n ** 3 * (2 * 2.5 * 3 * math.log2(n) + 20)
        return {"bytes": b, "flops": fl}
    n = c["nx"] * c["ny"] * c["nz"]
    nf = 2 if _two(c) else 1
    r = 4 if c["kahan"] else 8
    fft = 2.5 * n * math.log2(n)
    if c["kind"] == "output":
        return {"bytes": float(n * nf * 2 * r), "flops": (nf + 1) * (fft + 10 * n)}
    rw = (24 if c["kahan"] else 32) * nf
    kicks = KICKS[c["order"]] * c["steps"]
    gw = c["kind"] == "fd" and c["gw"]
    b = float(n) * kicks * (rw + (24 * r if gw else 0))
    if c["kind"] == "fd":
        per = 11 if c["lap"] == 7 else 31
        fl = float(n) * kicks * ((nf + (6 if gw else 0)) * per + 10 * nf)
    else:
        fl = kicks * nf * (2 * fft + 15.0 * n)
    if c["kind"] == "closure":
        fl += 65664.0 * n * -(-kicks // c["every"])
    if c["kind"] == "host":
        b += 4 * 8.0 * n * nf
    if c.get("record", "energies") == "energies":
        b += n * r * (2 * nf + (12 if gw else 0))
    if c.get("bins"):
        b += n * r * (6 if gw else 1)
        fl += fft * (6 if gw else 1)
    return {"bytes": b, "flops": fl}


# ------------------------------------------------- the same in torch, 64 bits
def _mix(z):
    z = z + _i64(0x9E3779B97F4A7C15)
    z = (z ^ _shr(z, 30)) * _i64(0xBF58476D1CE4E5B9)
    z = (z ^ _shr(z, 27)) * _i64(0x94D049BB133111EB)
    return z ^ _shr(z, 31)


def _i64(v):
    return v - (1 << 64) if v >= 1 << 63 else v


def _shr(z, n):
    return (z >> n) & ((1 << (64 - n)) - 1)


def _gauss(seed, field, mode):
    one = torch.full((1,), seed, dtype=torch.int64, device="cuda")
    key = _mix(_mix(_mix(one) ^ field) ^ mode)
    u1 = (_shr(_mix(key ^ 1), 11).double() + 1.0) * 2.0 ** -53
    u2 = (_shr(_mix(key ^ 2), 11).double() + 1.0) * 2.0 ** -53
    r, th = torch.sqrt(-2.0 * torch.log(u1)), 2 * math.pi * u2
    return r * torch.cos(th), r * torch.sin(th)


def _fold(n, m=None):
    i = torch.arange(n if m is None else m, device="cuda")
    return torch.minimum(i, n - i)


def _grid(shape):
    """Folded integer wave numbers of the half spectrum [nz][ny][nx/2+1]."""
    nx, ny, nz = shape
    return _fold(nx, nx // 2 + 1).view(1, 1, -1), _fold(ny).view(1, -1, 1), _fold(nz).view(-1, 1, 1)


def _vacuum(shape, length, seed, field, f0, d0, m2):
    nx, ny, nz = shape
    hx, n, dx = nx // 2 + 1, nx * ny * nz, length / nx
    kx, ky, kz = _grid(shape)
    dk = [2 * math.pi / (m * dx) for m in shape]
    k2 = (kx.double() * dk[0]) ** 2 + (ky.double() * dk[1]) ** 2 + (kz.double() * dk[2]) ** 2
    live = (k2 > 0) & (torch.sqrt(k2) <= KCUT * math.pi / dx)
    w = torch.sqrt(k2 + m2)
    sig = torch.sqrt(AMP * n * n / (2.0 * n * dx ** 3) / w)
    x = torch.arange(hx, device="cuda").view(1, 1, -1)
    y, z = torch.arange(ny, device="cuda").view(1, -1, 1), torch.arange(nz, device="cuda").view(-1, 1, 1)
    m = (z * ny + y) * hx + x
    mp = (((nz - z) % nz) * ny + (ny - y) % ny) * hx + x
    plane = (x == 0) | (2 * x == nx)
    own, conj = plane & (mp == m), plane & (mp < m)
    gr, gi = _gauss(seed, field, torch.where(conj, mp, m))
    h = math.sqrt(0.5)
    re = torch.where(own, sig * gr, sig * gr * h)
    im = torch.where(own, torch.zeros_like(gi), torch.where(conj, -sig * gi * h, sig * gi * h))
    F = torch.where(live, torch.complex(re, im), 0.0)
    turn = torch.where(own, 0.0, torch.where(conj, w, -w))
    P = torch.complex(-turn * F.imag, turn * F.real)
    s = (nz, ny, nx)
    return f0 + torch.fft.irfftn(F, s=s), d0 + torch.fft.irfftn(P, s=s)


def _nb(g, d):
    return torch.roll(g, 1, d) + torch.roll(g, -1, d)


STENCIL = {7: (-6.0, 1.0, 0.0, 0.0, 1.0), 27: (-128.0, 14.0, 3.0, 1.0, 30.0)}


def _ranks(g):
    """Sums over the 6 face, 12 edge and 8 corner neighbours."""
    sx, sy = _nb(g, 2), _nb(g, 1)
    sxy = _nb(sx, 1)
    return sx + sy + _nb(g, 0), sxy + _nb(sx + sy, 0), _nb(sxy, 0)


class _Exact:
    """A lattice in torch FP64 with the integrator's splitting, operation by operation."""

    def __init__(self, c, seed):
        self.c, self.shape = c, _shape(c)
        nx, ny, nz = self.shape
        self.n, self.length = nx * ny * nz, _length(c)
        self.dx = self.length / nx
        self.fd = c["kind"] == "fd"
        self.gw = self.fd and c["gw"]
        self.conf = c["conformal"]
        self.a, self.ap, self.net, self.u = 1.0, 0.0, None, None
        if self.gw:
            cen, r0, t0 = _bubbles(c, seed)
            x, y, z = (torch.arange(1, m + 1, device="cuda", dtype=torch.float64).view(v)
                       for m, v in ((nx, (1, 1, -1)), (ny, (1, -1, 1)), (nz, (-1, 1, 1))))
            f = torch.full((nz, ny, nx), -1.0, device="cuda", dtype=torch.float64)
            p = torch.zeros_like(f)
            for b in cen.tolist():
                r2 = ((x - b[0]) ** 2 + (y - b[1]) ** 2 + (z - b[2]) ** 2) * self.dx ** 2
                s1 = torch.sqrt(torch.where(r2 > t0 * t0, r2 - t0 * t0, 1.0))
                w = (s1 - r0) / math.sqrt(2.0)
                f += torch.where(r2 > t0 * t0, 1.0 - torch.tanh(w), 2.0)
                p += torch.where(r2 > t0 * t0, t0 / s1 / math.sqrt(2.0) / torch.cosh(w) ** 2, 0.0)
            self.f, self.p = [f], [p]
            self.u = [torch.zeros_like(f) for _ in range(6)]
            self.pu = [torch.zeros_like(f) for _ in range(6)]
        else:
            f0, d0, m2 = _means(c)
            fp = [_vacuum(self.shape, self.length, seed, i, f0[i], d0[i], m2[i]) for i in range(len(f0))]
            self.f, self.p = [v[0] for v in fp], [v[1] for v in fp]
        if self.conf:
            self.ap = -math.sqrt(12.0 * self.energies()[4])

    def k2(self):
        kx, ky, kz = _grid(self.shape)
        nx, ny, nz = self.shape
        d = [(2 * math.pi / (m * self.dx)) ** 2 for m in (nx, ny, nz)]
        return (kx * kx).double() * d[0] + (ky * ky).double() * d[1] + (kz * kz).double() * d[2]

    def lap(self, g):
        if not self.fd:
            return torch.fft.irfftn(-self.k2() * torch.fft.rfftn(g), s=g.shape)
        st = STENCIL[self.c["lap"]]
        r1, r2, r3 = _ranks(g)
        return (st[0] * g + st[1] * r1 + st[2] * r2 + st[3] * r3) / (st[4] * self.dx ** 2)

    def dv(self):
        f = self.f
        if self.gw:
            return [(f[0] ** 2 - 1.0) * f[0] - DEL]
        if len(f) == 2:
            return [f[0] ** 3 + 2.0 * f[0] * f[1] ** 2, 2.0 * f[0] ** 2 * f[1]]
        return [f[0] ** 3]

    def pot(self):
        f = self.f
        if self.gw:
            v = 0.25 * (f[0] ** 2 - 1.0) ** 2 - DEL * (f[0] + 1.0)
        elif len(f) == 2:
            v = 0.25 * f[0] ** 4 + f[0] ** 2 * f[1] ** 2
        else:
            v = 0.25 * f[0] ** 4
        return float(v.mean())

    def drift(self, h):
        ke = sum(float((p * p).sum()) for p in self.p)
        for f, p in zip(self.f, self.p):
            f += (h / self.a ** 2) * p
        if self.gw:
            for u, pu in zip(self.u, self.pu):
                u += h * pu
        if self.conf:
            self.ap += h * ke / self.n / self.a ** 3

    def kick(self, h):
        corr = None
        if self.net is not None:
            if self.net["left"] == 0:
                self.net["force"] = self.force()
                self.net["left"] = self.c["every"]
            self.net["left"] -= 1
            corr = self.net["force"]
        laps, dv = [self.lap(f) for f in self.f], self.dv()
        ge2 = -sum(float((f * q).sum()) for f, q in zip(self.f, laps)) if self.conf else 0.0
        pe = self.pot() if self.conf else 0.0
        if self.gw:
            d = [(torch.roll(self.f[0], -1, k) - torch.roll(self.f[0], 1, k)) / (2 * self.dx) for k in (2, 1, 0)]
            for (i, j), u, pu in zip(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)), self.u, self.pu):
                pu += h * (self.lap(u) + KAPPA * d[i] * d[j])
        a = self.a
        for k, p in enumerate(self.p):
            p += h * (a * a * laps[k] - a ** 4 * dv[k])
            if corr is not None:
                p += h * (a if self.conf else 1.0) * corr[k]
        if self.conf:
            self.ap -= a ** 3 * (ge2 / a ** 2 / self.n + 4.0 * pe) * h

    def grav(self, h):
        self.a -= h * self.ap / 6.0

    def o2step(self, dt, w1, w2):
        if self.gw:  # metric, drift, kick
            self.drift(w1 * dt / 2)
            self.kick(w1 * dt)
            self.drift(w1 * dt / 2)
            return
        if self.conf:
            self.grav(w1 * dt / 2)
        self.kick(w1 * dt)
        if self.conf:
            self.grav(w1 * dt / 2)
        self.drift((w1 + w2) * dt / 2)

    def symp(self, order, dt, steps):
        if self.net is not None:
            self.net["left"] = 0
        if order == 2:
            w = [1.0]
        elif order == 4:
            w1 = 1.0 / (2.0 - 2.0 ** (1.0 / 3.0))
            w = [w1, 1.0 - 2.0 * w1, w1]
        else:
            a, b, d = 0.784513610477560, 0.235573213359357, (-1.17767998417887 if self.gw else -1.177679984177887)
            w = [a, b, d, 1.0 - 2.0 * (a + b + d), d, b, a]
        if not self.gw:
            self.drift(w[0] * dt / 2)
        for j in range(steps):
            for i, v in enumerate(w):
                last = i == len(w) - 1
                self.o2step(dt, v, w[i + 1] if not last else (0.0 if j == steps - 1 else w[0]))

    def energies(self):
        n, a, conf = self.n, self.a, self.conf
        ke = 0.5 * sum(float((p * p).sum()) for p in self.p) / n / (a ** 6 if conf else 1.0)
        ge = 0.5 * -sum(float((f * self.lap(f)).sum()) for f in self.f) / n / (a * a)
        gg = ge
        if self.fd:
            st = STENCIL[self.c["lap"]]
            q = 0.0
            for f in self.f:
                r, s = _ranks(f), _ranks(f * f)
                for k, cnt in ((1, 6.0), (2, 12.0), (3, 8.0)):
                    q += st[k] * float((s[k - 1] - 2.0 * f * r[k - 1] + cnt * f * f).sum())
            gg = 0.25 / (a * self.dx) ** 2 / st[4] * q / n
        pe = self.pot()
        rho = ke + ge + pe
        hub = -self.ap / 6.0 / (a * a) if conf else 0.0
        means = [float(f.mean()) for f in self.f] + [0.0]
        gw = 0.0
        if self.gw:
            wt = (1.0, 1.0, 1.0, 2.0, 2.0, 2.0)
            gw = 0.5 / n * sum(w * float((pu * pu).sum() - (u * self.lap(u)).sum())
                               for w, u, pu in zip(wt, self.u, self.pu))
        return np.array([ke, ge, gg, pe, rho, -3.0 * hub * hub, (rho - 3.0 * hub * hub) / rho, a,
                         self.ap if conf else 0.0, means[0], means[1], gw])

    def bins(self, values, nb, weighted):
        """Shell sums of each half-spectrum array in `values` and of the weights."""
        kx, ky, kz = _grid(self.shape)
        m2 = (kx * kx + ky * ky + kz * kz).reshape(-1)
        p = torch.sqrt(m2.double())
        l = torch.floor(p).long()
        l -= (l * l > m2).long()
        l += ((l + 1) * (l + 1) <= m2).long()
        nx = self.shape[0]
        x = torch.arange(nx // 2 + 1, device="cuda").view(1, 1, -1)
        wx = torch.where((x == 0) | (2 * x == nx), 1.0, 2.0).double().expand(self.shape[2], self.shape[1], -1).reshape(-1)
        out = []
        for v in [None] + list(values):
            t = wx if v is None else wx * v.reshape(-1)
            if weighted:
                c0, c1 = (1.0 - (l - p) ** 2) ** 2, (1.0 - (l + 1 - p) ** 2) ** 2
                s = torch.bincount(l, t * c0, minlength=nb + 2)[:nb]
                s[1:] += torch.bincount(l, t * c1, minlength=nb + 2)[:nb - 1]
            else:
                s = torch.bincount(l, t, minlength=nb + 2)[:nb]
            out.append(s)
        w = out[0]
        safe = torch.where(w != 0, w, 1.0)
        return [(s / safe).cpu().numpy() for s in out[1:]], w.cpu().numpy()

    def power(self, g, nb, weighted=True):
        F = torch.fft.rfftn(g)
        S, W = self.bins([F.real ** 2 + F.imag ** 2], nb, weighted)
        return [S[0], W]

    def cross(self, g, h, nb):
        F = torch.fft.rfftn(g) * torch.fft.rfftn(h).conj()
        return self.bins([F.real, F.imag], nb, True)[0]

    def gw_spectrum(self, nb):
        nx, ny, nz = self.shape
        i = [torch.arange(m, device="cuda", dtype=torch.float64) for m in (nx // 2 + 1, ny, nz)]
        sx, sy, sz = (torch.sin(2 * math.pi * v / m) for v, m in zip(i, self.shape))
        sx, sy, sz = sx.view(1, 1, -1), sy.view(1, -1, 1), sz.view(-1, 1, 1)
        k = [v.expand(nz, ny, nx // 2 + 1) / self.dx for v in (sx, sy, sz)]
        k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
        ok = k2 > 0
        inv = torch.where(ok, 1.0 / torch.where(ok, k2, 1.0), 0.0)
        F = [torch.fft.rfftn(v) for v in self.pu]
        at = ((0, 3, 4), (3, 1, 5), (4, 5, 2))
        P = [[(1.0 if i == j else 0.0) - k[i] * k[j] * inv for j in range(3)] for i in range(3)]
        A = [[sum(P[i][m] * F[at[m][j]] for m in range(3)) for j in range(3)] for i in range(3)]
        tr = A[0][0] + A[1][1] + A[2][2]
        tot = torch.zeros_like(k2)
        for i in range(3):
            for j in range(3):
                t = sum(A[i][m] * P[m][j] for m in range(3)) - 0.5 * P[i][j] * tr
                tot += t.real ** 2 + t.imag ** 2
        S, W = self.bins([torch.where(ok, tot, 0.0)], nb, False)
        return [S[0], W]

    def force(self):
        """The network's force on the two fields, divided by its output normalisation."""
        a = self.a if self.conf else 1.0
        x = torch.stack([self.f[0] * a, self.f[1] * a, self.p[0] / a, self.p[1] / a])[None]
        y = _net_forward(self.net["params"], x)[0]
        o = NORM[2]
        return [y[..., 0] / o[0], y[..., 1] / o[1]]


def _unflatten(q):
    o, out = 0, []
    for shp in ((27, 8, 32), (32,), (27, 32, 32), (32,), (27, 32, 8), (8,)):
        m = math.prod(shp)
        out.append(q[o:o + m].reshape(shp))
        o += m
    return out


def _net_forward(q, x):
    """x [batch][4][nz][ny][nx] raw inputs -> normalised outputs [batch][nz][ny][nx][2]."""
    w1, b1, w2, b2, w3, b3 = _unflatten(q)
    scale = torch.as_tensor(NORM[1], device=x.device).view(1, 4, 1, 1, 1)
    h = (x * scale).permute(0, 2, 3, 4, 1)

    def conv(h, w, b):
        out = b.expand(h.shape[:-1] + b.shape)
        for t in range(27):
            d = (t // 9 - 1, t // 3 % 3 - 1, t % 3 - 1)
            out = out + torch.roll(h, (-d[0], -d[1], -d[2]), (1, 2, 3)) @ w[t]
        return out

    gelu = lambda z: 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))  # noqa: E731
    h = gelu(conv(h, w1[:, :4], b1))
    h = gelu(conv(h, w2, b2))
    return conv(h, w3[:, :, :2], b3[:2])


def _exact_train(c, seed):
    q = torch.as_tensor(_net_params(seed), device="cuda").double().requires_grad_(True)
    d = _samples(c, seed).double()
    y = _net_forward(q, d[:, :4])
    tgt = torch.stack([d[:, 4] * NORM[2][0], d[:, 5] * NORM[2][1]], -1)
    loss = ((y - tgt) ** 2).mean()
    (g,) = torch.autograd.grad(loss, q)
    # the first Adam step: both moments bias-corrected to g and g^2
    new = q.detach() - LR * g / (g.abs() + 1e-8)
    return {"loss": float(loss.detach()), "params": new.cpu().numpy()}


def exact(case, seed):
    c = case
    if c["kind"] == "train":
        if c["nx"] * c["ny"] * c["nz"] * c["batch"] > 1 << 21:  # autograd's FP64 activations
            return None
        return _exact_train(c, seed)
    if c["kind"] == "ensemble":
        return _exact_ensemble(c, seed)
    if c["kind"] == "output":
        e = _Exact(c, seed)
        e.symp(2, _dt(dict(c, order=2)), 2)
        nb = c["bins"]
        out = {"energies": e.energies()}
        for f in range(len(e.f)):
            out["fld%d" % f] = e.power(e.f[f], nb)
        out["fldp0"] = e.power(e.p[0], nb)[0]
        out["cross"] = e.cross(e.p[0], e.f[0], nb)
        out["count"] = e.power(e.f[0], nb, False)
        return out
    e = _Exact(c, seed)
    if c["kind"] == "closure":
        e.net = dict(params=torch.as_tensor(_net_params(seed), device="cuda").double(), left=0)
    e.symp(c["order"], _dt(c), c["steps"])
    f, p = torch.stack(e.f), torch.stack(e.p)
    if c["kind"] == "host":
        return {"energies": e.energies(), "fld": f.permute(1, 2, 3, 0).cpu().numpy(),
                "fldp": p.permute(1, 2, 3, 0).cpu().numpy()}
    out = {"fld": f, "fldp": p}
    record = c.get("record", "energies")
    if record == "energies":
        out["energies"] = e.energies()
    elif record == "a":
        out["a"] = [e.a, e.ap]
    if c.get("bins"):
        if e.gw:
            out["gw"] = e.gw_spectrum(c["bins"])
        else:
            out["pk"] = e.power(e.f[0], c["bins"])
    return out


def _exact_ensemble(c, seed):
    sizes, seeds = _ens_sizes(c), _ens_seeds(c, seed)
    rows, out = [], {}
    shown = [sizes.index(n) for n in ENS_SIZES if n in sizes]
    for r, n in enumerate(sizes):
        one = dict(kind="spectral", nx=n, ny=n, nz=n, nfld=1, conformal=False, order=c["order"])
        e = _Exact(one, seeds[r])
        e.symp(c["order"], 20.0 / n / 20, c["steps"])
        rows.append(e.energies())
        if r in shown:
            out["S%d" % r], out["W%d" % r] = e.power(e.f[0], c["bins"])
    out["energies"] = np.array(rows)
    return out
