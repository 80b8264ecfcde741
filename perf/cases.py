"""Performance cases: the work a user of this framework has it do, per control step.

Kinds of case (each through its public entry point):

``step``   tomography + DM fit of ``batch`` instances, gradients resident on the
           device (``Reconstructor.step_device``): the control step itself.
``block``  the same from a cold start (``Reconstructor.reset`` first), for right-hand
           sides that are unrelated to the ones before, as in the control-matrix build.
``host``   the reference's call pattern with host FP64 buffers, ``gpu_tomo`` then
           ``gpu_fit`` (``Reconstructor.tomo_only`` + ``fit``).
``serve``  one masked batch of a serving pool, pinned host gradients in and
           commands out (``Reconstructor.serve_step``).
``wfs``    geometric Shack-Hartmann gradients of ``batch`` instances through the
           DMs, with noise (``GeomWfs.grad``): the simulation half of the loop.
``mvm``    the precomputed control matrix applied to ``batch`` gradient vectors
           (``mb_mvm_apply_device``), in each storage type.
"""
from __future__ import annotations

import copy
import ctypes as C
import dataclasses
import functools
import math

import numpy as np
import torch

from maos_b200 import config, fit_assemble, fit_setup, geometry, native, turbulence, wfs_setup
from maos_b200.recon import Reconstructor
from maos_b200.wfs import GeomWfs

DTYPES = {"f32": native.MB_MVM_F32, "bf16": native.MB_MVM_BF16, "fp8": native.MB_MVM_FP8}
# An FDPCG solve in FP32 ends a few 1e-6 from its 64-bit value, by rounding in the directions the gradients
# constrain least: a handful of modes, so the distance of one instance scatters by a factor of two with the
# order of any sum.  Over this many instances it averages out and says how precise the solve is.
WIDE = 24


def listed():
    return [
        # one 8 m SCAO loop, warm-started CG: the smallest solve, launch-sized kernels
        {"name": "scao_1", "kind": "step", "system": "scao_8m", "order": 20, "batch": 1, "fit": "assembled",
         "maxit": 20, "tune": True},
        # one 8 m LTAO simulation calling gpu_tomo and gpu_fit with host buffers
        {"name": "ltao_host", "kind": "host", "system": "ltao_8m", "order": 20, "batch": 1, "fit": "assembled",
         "maxit": 30, "tune": False},
        # the LTAO pool of the served mix, two thirds of its slots with a frame to step (pools are not tuned)
        {"name": "ltao_serve_26", "kind": "serve", "system": "ltao_8m", "order": 20, "batch": 26, "fit": "assembled",
         "maxit": 30, "tune": False},
        # one 30 m MCAO telescope in open loop, tuned at start-up: step latency of the flagship system
        {"name": "mcao_1", "kind": "step", "system": "mcao_30m", "order": 60, "batch": 1, "fit": "assembled",
         "maxit": 10, "tune": True},
        # a small pool of 30 m systems in closed loop (4 warm-started FDPCG iterations, the reference's default)
        {"name": "mcao_6", "kind": "step", "system": "mcao_30m", "order": 60, "batch": 6, "fit": "assembled",
         "maxit": 4, "tune": False},
        # the benchmark's batch of 30 m systems, with the open-loop iteration count
        {"name": "mcao_32", "kind": "step", "system": "mcao_30m", "order": 60, "batch": 32, "fit": "assembled",
         "maxit": 10, "tune": True},
        # a block of 256 30 m right-hand sides from a cold start, as the control-matrix build solves them
        {"name": "mcao_256", "kind": "block", "system": "mcao_30m", "order": 60, "batch": 256, "fit": "assembled",
         "maxit": 30, "tune": False},
        # 39 m ELT with 9 layers and 3 DMs in closed loop, grid-form fit (gpu.fit=2)
        {"name": "elt_2", "kind": "step", "system": "elt_39m", "order": 80, "batch": 2, "fit": "grid",
         "maxit": 4, "tune": False},
        # gradients of one 8 m LTAO loop
        {"name": "wfs_ltao_1", "kind": "wfs", "system": "ltao_8m", "order": 20, "batch": 1},
        # gradients of a batch of 30 m closed loops
        {"name": "wfs_mcao_8", "kind": "wfs", "system": "mcao_30m", "order": 60, "batch": 8},
        # control matrix of an 8 m LTAO system, one instance
        {"name": "mvm_f32_ltao_1", "kind": "mvm", "dtype": "f32", "nact": 476, "ngrad": 2656, "batch": 1},
        # one GPU's columns (three of six WFS) of the 30 m control matrix, a served pool
        {"name": "mvm_bf16_mcao_12", "kind": "mvm", "dtype": "bf16", "nact": 7048, "ngrad": 16920, "batch": 12},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["block", "host"] + ["serve"] * 2 + ["wfs"] * 3 + ["mvm"] * 3)
    if kind == "mvm":
        nact = _log(rng, 150, 8000)
        return {"kind": kind, "dtype": rng.choice(list(DTYPES)), "nact": nact,
                "ngrad": _log(rng, 300, min(34000, 130000000 // nact)), "batch": _log(rng, 1, 64)}
    if kind == "block":
        return {"kind": kind, "system": "mcao_30m", "order": 60, "batch": _log(rng, WIDE, 255), "fit": "assembled",
                "maxit": rng.randint(15, 30), "tune": False}
    large = rng.random() < (0.6 if kind == "step" else 0.4)
    system = rng.choice(["mcao_30m", "mcao_30m", "elt_39m"] if kind == "step" else ["mcao_30m"]) if large else \
        rng.choice(["scao_8m", "ltao_8m"])
    order = {"mcao_30m": 60, "elt_39m": 80}.get(system) or rng.randint(16, 30)
    case = {"kind": kind, "system": system, "order": order}
    if kind == "wfs":
        return dict(case, batch=_log(rng, 1, 12 if large else 48))
    if kind == "host":
        batch = 1
    else:
        batch = _log(rng, 1, {"mcao_30m": 160, "elt_39m": 24}.get(system, 64))
    fit = rng.choice(["assembled", "grid"]) if system == "mcao_30m" else "grid" if large else "assembled"
    if large:  # FDPCG: the closed-loop and the open-loop count
        maxit = rng.choice([4, 10]) if system == "mcao_30m" else 4
    else:
        maxit = rng.choice([10, 20] if system == "scao_8m" else [20, 30])
    return dict(case, batch=batch, fit=fit, maxit=maxit, tune=rng.random() < 0.5 and kind == "step")


# ---------------------------------------------------------------------------
# systems (tables a program builds once and keeps)
# ---------------------------------------------------------------------------
def _key(case):
    return case["system"], case["order"]


@functools.lru_cache(maxsize=None)
def _system(name, order):
    cfg = config.PRESETS[name]()
    if order != cfg.powfs[0].order:  # another sampling of the same 8 m telescope
        dsa = cfg.D / order
        cfg = dataclasses.replace(
            cfg, atmr_dx=dsa, powfs=[dataclasses.replace(p, order=order, dsa=dsa) for p in cfg.powfs],
            dms=[dataclasses.replace(d, dx=dsa, order=order + 1) for d in cfg.dms])
    return geometry.build_tomo(cfg)


@functools.lru_cache(maxsize=None)
def _fit(name, order, form):
    build = fit_assemble.build_fit_assembled if form == "assembled" else fit_setup.build_fit
    return build(_system(name, order))


@functools.lru_cache(maxsize=None)
def _geom(name, order):
    return wfs_setup.build_geom_wfs(_system(name, order))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gradients(sysm, batch, seed):
    """[batch, ngrad] FP32 gradients of seeded von Karman atmospheres with the
    system's noise.  Up to 6 frames of one frozen-flow sequence are sampled
    exactly; further instances are unit-variance mixtures of them (a mixture
    of Gaussian fields of one spectrum has that spectrum)."""
    atm = turbulence.FrozenFlowAtmosphere(sysm.cfg, seed % (1 << 31))
    dev = turbulence.DeviceAtmosphere(atm)
    n = min(batch, 6)
    rng = np.random.default_rng(seed)
    fr = torch.as_tensor(np.stack([dev.gradients(sysm, 0.5 * k, rng, noise=False) for k in range(n)]), device="cuda")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    mix = torch.randn(batch, n, generator=gen, device="cuda", dtype=torch.float64)
    mix = mix / mix.norm(dim=1, keepdim=True)
    mix[:n] = torch.eye(n, device="cuda", dtype=torch.float64)
    g = mix @ fr
    nea = torch.as_tensor(np.concatenate([np.sqrt(w.sanea) for w in sysm.wfs]), device="cuda")
    g += nea * torch.randn(g.shape, generator=gen, device="cuda", dtype=torch.float64)
    return g.float()


def _inputs(case, seed):
    return _gradients(_system(*_key(case)), case["batch"], seed)


def _mask(case, seed):
    m = (np.random.default_rng(seed).random(case["batch"]) < 0.67).astype(np.int32)
    m[seed % case["batch"]] = 1
    return m


def _matrix(case, seed):
    """nact x ngrad FP64 control matrix on the device, rows of differing scale."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    na, ng = case["nact"], case["ngrad"]
    M = torch.randn(ng, na, generator=gen, device="cuda") * 1e-2
    M *= torch.exp(torch.randn(na, generator=gen, device="cuda") * 0.5)
    g = torch.randn(case["batch"], ng, generator=gen, device="cuda") * 1e-6
    return M, g  # M transposed: column-major nact x ngrad


def _screens(case, seed):
    """One FrozenFlowAtmosphere per instance: the same periodic screens, each
    instance's shifted by its own offset."""
    sysm = _system(*_key(case))
    a0 = turbulence.FrozenFlowAtmosphere(sysm.cfg, seed % (1 << 31))
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["batch"]):
        a = copy.copy(a0)
        sh = rng.integers(0, a0.n, 2)
        a.screens = [np.roll(s, sh, axis=(0, 1)) for s in a0.screens]
        out.append(a)
    isim = int(rng.integers(0, 4000))
    nact = _fit(*_key(case), "grid").nact
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    dm = torch.randn(case["batch"], nact, generator=gen, device="cuda") * 1e-7
    return out, isim, dm, (seed & 0xFFFFFF) + 1


class _View:
    """A reconstructor's FP32 device array (the view keeps its owner)."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f4", "data": (int(ptr), False),
                                         "version": 3, "strides": None}


class _Mvm:
    def __init__(self, M, dtype, batch):
        self.lib = native.load()
        ng, na = M.shape
        Mc = M.double().cpu().numpy()
        h = C.c_void_p()
        native.check(self.lib.mb_mvm_create(Mc.ctypes.data_as(C.POINTER(C.c_double)), na, ng, DTYPES[dtype], batch,
                                            C.byref(h)), "mb_mvm_create")
        self.h = h

    def __del__(self):
        if getattr(self, "h", None):
            self.lib.mb_mvm_free(self.h)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mvm":
        M, g = _matrix(case, seed)
        return {"kind": kind, "mvm": _Mvm(M, case["dtype"], case["batch"]), "g": g,
                "out": torch.empty(case["batch"], case["nact"], device="cuda")}
    sysm = _system(*_key(case))
    if kind == "wfs":
        atms, isim, dm, noise = _screens(case, seed)
        W = GeomWfs.for_system(sysm, atms, fit=_fit(*_key(case), "grid"), nbatch=case["batch"], geom=_geom(*_key(case)))
        return {"kind": kind, "W": W, "isim": isim, "dm": dm, "noise": noise}
    R = Reconstructor(sysm, nbatch=case["batch"], maxit=case["maxit"], fit=_fit(*_key(case), case["fit"]))
    if case["tune"]:
        R.autotune(reps=5)
    g = _inputs(case, seed)
    st = {"kind": kind, "R": R, "g": g}
    if kind == "host":
        st["g"] = g.double().cpu().numpy()
    elif kind == "serve":
        st["g"] = g.cpu().pin_memory()
        st["out"] = torch.zeros(case["batch"], R.nact).pin_memory()
        st["mask"] = _mask(case, seed)
    else:
        st["a"] = torch.as_tensor(_View(R, R.fit_solution_ptr(), (R.nbatch, R.nact)), device="cuda")
        # the layers are the warm start of the next step; a 30 m FP32 solve leaves rounding noise of
        # 1e-3 in the layer directions that neither the gradients nor the commands see
        if sysm.fdpcg is None:
            st["x"] = torch.as_tensor(_View(R, R.solution_ptr(), (R.nbatch, R.nxtot)), device="cuda")
    torch.cuda.synchronize()
    return st


def run(state):
    kind = state["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "mvm":
        m = state["mvm"]
        native.check(m.lib.mb_mvm_apply_device(m.h, C.c_void_p(state["g"].data_ptr()),
                                               C.c_void_p(state["out"].data_ptr()), C.c_void_p(stream)),
                     "mb_mvm_apply_device")
        return state["out"]
    if kind == "wfs":
        return state["W"].grad(state["isim"], dm=state["dm"], seed=state["noise"])
    R = state["R"]
    if kind == "host":
        R.tomo_only(state["g"])
        return R.fit()[0].astype(np.float32)
    if kind == "serve":
        R.serve_step(state["mask"], state["g"].data_ptr(), state["out"].data_ptr(), stream)
        return state["out"]
    if kind == "block":
        torch.cuda.current_stream().synchronize()
        R.reset()
    R.step_device(state["g"].data_ptr(), stream)
    return {"commands": state["a"], "layers": state["x"]} if "x" in state else {"commands": state["a"]}


# ---------------------------------------------------------------------------
# work: inputs, state and tables read once, outputs written once; the
# operators' multiply-adds
# ---------------------------------------------------------------------------
def work(case):
    kind, nb = case["kind"], case["batch"]
    if kind == "mvm":
        na, ng = case["nact"], case["ngrad"]
        return {"bytes": na * ng * {"f32": 4, "bf16": 2, "fp8": 1}[case["dtype"]] + 4 * nb * (na + ng),
                "flops": 2.0 * nb * na * ng}
    sysm = _system(*_key(case))
    nsa = sum(w.nsa for w in sysm.wfs)
    if kind == "wfs":
        cfg, fit, P = sysm.cfg, _fit(*_key(case), "grid"), _geom(*_key(case)).powfs[0]
        nmap = len(cfg.atm_ht) + len(fit.dms)
        # each map's pixels under the pupil once; per subaperture and map its block of pixels
        pix = len(cfg.atm_ht) * (cfg.D / cfg.atm_dx) ** 2
        side = P.dsa / cfg.atm_dx + 3
        return {"bytes": 4.0 * nb * (pix + fit.nact + 2 * nsa), "flops": 4.0 * nb * nsa * nmap * side * side}
    fit = _fit(*_key(case), case["fit"])
    nx, npup, nw, nl = int(sysm.nx_total), sysm.pmap.n, len(sysm.wfs), len(sysm.xmaps)
    it, fit_it = case["maxit"] + 1, fit.maxit + 1
    pos = int(round(sysm.wfs[0].dsa / sysm.pmap.dx))
    ray = 2 * 6.0 * nw * nl * npup  # separable bilinear, each direction
    gp = 2 * 4.0 * nsa * (pos + 1) ** 2
    flops = it * (ray + gp + 30.0 * nx)
    table = 8.0 * nsa * (pos + 1) ** 2 + 12.0 * nsa
    if sysm.fdpcg is not None:
        nbl, bs = sysm.fdpcg.nb // 2, sysm.fdpcg.bs
        flops += it * (8.0 * nbl * bs * bs + sum(5.0 * g.n * math.log2(g.n) for g in sysm.xmaps))
        table += 8.0 * nbl * bs * bs
    if case["fit"] == "assembled":
        flops += 2.0 * (fit.FRM.nnz + fit_it * fit.FLM.nnz)
        table += 8.0 * (fit.FRM.nnz + fit.FLM.nnz)
    else:
        nf, nd = len(fit.thetax), len(fit.dms)
        flops += fit_it * nf * fit.floc.n * (12.0 * nd + 18.0)
        table += 12.0 * fit.W0.nnz
    act = float(_mask(case, 1).sum()) if kind == "serve" else nb
    return {"bytes": table + 4.0 * act * (2 * nsa + 2 * nx + 2 * fit.nact), "flops": flops * act}


# ---------------------------------------------------------------------------
# 64-bit values
# ---------------------------------------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=_dev())


class _Sparse:
    """y = A x and y = A^T x for x [batch, n], FP64."""

    def __init__(self, A):
        def csr(B):
            B = B.tocsr()
            return torch.sparse_csr_tensor(torch.as_tensor(B.indptr.astype(np.int64)),
                                           torch.as_tensor(B.indices.astype(np.int64)), torch.as_tensor(B.data),
                                           size=B.shape, dtype=torch.float64).to(_dev())
        self.A, self.At = csr(A), csr(A.T)

    def __call__(self, x):
        return (self.A @ x.T.contiguous()).T

    def t(self, x):
        return (self.At @ x.T.contiguous()).T


def _axis(n_out, o_out, d_out, scale, disp, o_in, d_in, n_in):
    """[n_out, n_in] linear interpolation along one axis; points off the source get no weight."""
    u = ((o_out + np.arange(n_out) * d_out) * scale + disp - o_in) / d_in
    k = np.floor(u).astype(np.int64)
    f = u - k
    last = (k == n_in - 1) & (f < 1e-12)
    k, f = np.where(last, n_in - 2, k), np.where(last, 1.0, f)
    A = np.zeros((n_out, n_in))
    ok = (u >= 0) & (k >= 0) & (k <= n_in - 2)
    i = np.nonzero(ok)[0]
    A[i, k[i]] += 1 - f[i]
    A[i, k[i] + 1] += f[i]
    return A


class _Solve:
    """Tomography and fit of one system in FP64, from the same tables the framework is given."""

    def __init__(self, sysm, fit):
        self.s, self.f = sysm, fit
        p = sysm.pmap
        self.np = (p.ny, p.nx)
        self.H = []
        for w in sysm.wfs:
            row = []
            for l, g in enumerate(sysm.xmaps):
                h = float(sysm.ht[l])
                sc = 1.0 - h / w.hs
                row.append((_t(_axis(p.ny, p.oy, p.dy, sc, w.thetay * h, g.oy, g.dy, g.ny)),
                            _t(_axis(p.nx, p.ox, p.dx, sc, w.thetax * h, g.ox, g.dx, g.nx))))
            self.H.append(row)
        gp = {id(w.GP): w.GP for w in sysm.wfs}  # WFS of one type share theirs
        gp = {k: _Sparse(G) for k, G in gp.items()}
        self.GP = [gp[id(w.GP)] for w in sysm.wfs]
        self.W = [_t(w.saneai) for w in sysm.wfs]
        self.TT = [None if w.PTT is None else (_t(w.TT), _t(w.PTT)) for w in sysm.wfs]
        self.xo, self.go = sysm.x_offsets(), sysm.g_offsets()
        fd = sysm.fdpcg
        if fd is not None:
            self.M = torch.as_tensor(np.asarray(fd.Mbinv, dtype=np.complex128), device=_dev())
            self.perm = torch.as_tensor(np.asarray(fd.perm, dtype=np.int64), device=_dev())
        if hasattr(fit, "FLM"):
            self.FR, self.FL = _Sparse(fit.FRM), _Sparse(fit.FLM)
            self.lr = [_t(a) for a in (fit.FRU, fit.FRV, fit.FLU, fit.FLV)]
        else:
            q = fit.floc
            self.HXF = [[(_t(_axis(q.ny, q.oy, q.dy, 1.0, ty * g.ht, g.oy, g.dy, g.ny)),
                          _t(_axis(q.nx, q.ox, q.dx, 1.0, tx * g.ht, g.ox, g.dx, g.nx))) for g in sysm.xmaps]
                        for tx, ty in zip(fit.thetax, fit.thetay)]
            self.HA = [[_Sparse(a) for a in row] for row in fit.HA]
            self.W0, self.W1, self.NW = _Sparse(fit.W0), _t(fit.W1), _t(fit.NW)
            self.slave = _Sparse(fit.actslave) if fit.actslave is not None else None
            self.ao = fit.act_offsets()

    def layers(self, x):
        return [x[:, self.xo[l]:self.xo[l + 1]].reshape(-1, g.ny, g.nx) for l, g in enumerate(self.s.xmaps)]

    def back(self, gw, w):  # NEA, GP^T, then Hx^T of one WFS
        o = self.GP[w].t(gw * self.W[w]).reshape(-1, *self.np)
        return torch.cat([(ay.T @ o @ ax).reshape(len(o), -1) for ay, ax in self.H[w]], dim=1)

    def rhs(self, g):
        out = 0
        for w in range(len(self.s.wfs)):
            gw = g[:, self.go[w]:self.go[w + 1]]
            if self.TT[w] is not None:
                tt, ptt = self.TT[w]
                gw = gw - (gw @ ptt.T) @ tt.T
            out = out + self.back(gw, w)
        return out

    def lhs(self, x):
        xs, out = self.layers(x), 0
        for w in range(len(self.s.wfs)):
            o = sum(ay @ X @ ax.T for (ay, ax), X in zip(self.H[w], xs))
            out = out + self.back(self.GP[w](o.reshape(len(x), -1)), w)

        def lap(v):
            return (v.roll(1, 1) + v.roll(-1, 1) + v.roll(1, 2) + v.roll(-1, 2)) - 4 * v
        reg = [float(c) * lap(lap(X)).reshape(len(x), -1) for c, X in zip(self.s.l2c, xs)]
        return out + torch.cat(reg, dim=1)

    def precond(self, r):
        fd = self.s.fdpcg
        f = []
        for X in self.layers(r):
            s = math.sqrt(X.shape[1] * X.shape[2])
            f.append((torch.fft.fft2(X.to(torch.complex128)) / (s if fd.scale else 1.0)).reshape(len(r), -1))
        f = torch.cat(f, dim=1)
        y = torch.einsum("bij,nbj->nbi", self.M, f[:, self.perm].reshape(len(r), fd.nb, fd.bs))
        z = torch.empty_like(f)
        z[:, self.perm] = y.reshape(len(r), -1)
        out = []
        for l, g in enumerate(self.s.xmaps):
            n = g.nx * g.ny
            v = torch.fft.ifft2(z[:, self.xo[l]:self.xo[l + 1]].reshape(-1, g.ny, g.nx)) * n
            out.append((v.real / (math.sqrt(n) if fd.scale else 1.0)).reshape(len(r), -1))
        return torch.cat(out, dim=1)

    def _weight(self, v, k):
        return float(self.f.wt[k]) * (self.W0(v) - (v @ self.W1)[:, None] * self.W1)

    def _grid(self, v):  # v[k]: weighted OPD of fit direction k
        return torch.cat([sum(self.HA[k][d].t(v[k]) for k in range(len(v))) for d in range(len(self.f.dms))], dim=1)

    def fit_rhs(self, x):
        if hasattr(self, "FR"):
            return self.FR(x) - (x @ self.lr[1]) @ self.lr[0].T
        xs = self.layers(x)
        return self._grid([self._weight(sum(ay @ X @ ax.T for (ay, ax), X in zip(row, xs)).reshape(len(x), -1), k)
                           for k, row in enumerate(self.HXF)])

    def fit_lhs(self, a):
        if hasattr(self, "FL"):
            return self.FL(a) - (a @ self.lr[3]) @ self.lr[2].T
        As = [a[:, self.ao[d]:self.ao[d + 1]] for d in range(len(self.f.dms))]
        out = self._grid([self._weight(sum(h(A) for h, A in zip(row, As)), k) for k, row in enumerate(self.HA)])
        out = out + (a @ self.NW) @ self.NW.T
        return out if self.slave is None else out + self.slave(a)

    @staticmethod
    def cg(A, M, b, n):
        """n iterations from zero, restarted from the residual every 100."""
        x = torch.zeros_like(b)
        for k in range(n):
            if k % 100 == 0:
                r = b - A(x)
                z = M(r) if M else r
                p, rz = z, (r * z).sum(1, keepdim=True)
            Ap = A(p)
            al = rz / (p * Ap).sum(1, keepdim=True)
            al = torch.where(torch.isfinite(al), al, torch.zeros_like(al))
            x, r = x + al * p, r - al * Ap
            if k + 1 == n:
                break
            z = M(r) if M else r
            new = (r * z).sum(1, keepdim=True)
            be = new / rz
            p, rz = z + torch.where(torch.isfinite(be), be, torch.zeros_like(be)) * p, new
        return x

    def step(self, g, it, fit_it):
        x = self.cg(self.lhs, self.precond if self.s.fdpcg is not None else None, self.rhs(g.double()), it)
        return x, self.cg(self.fit_lhs, None, self.fit_rhs(x), fit_it)


def _normals(seed, isim, iwfs, inst, nsa):
    """The noise generator's two normals per subaperture: Philox4x32-10
    (Salmon et al. 2011), counter (subaperture, WFS, step, instance), then Box-Muller."""
    mask = np.uint64(0xFFFFFFFF)
    c = [np.arange(nsa, dtype=np.uint64)] + [np.full(nsa, v, dtype=np.uint64) for v in (iwfs, isim, inst)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & mask, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1),
             p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    r = np.sqrt(-2.0 * np.log((c[0].astype(np.float64) + 1.0) * 2.0 ** -32))
    t = 2.0 * math.pi * c[1].astype(np.float64) * 2.0 ** -32
    return r * np.cos(t), r * np.sin(t)


def _sample(S, gx, gy, scale, dispx, dispy, o, d, wrap):
    """Map S [ny, nx] (origin o, spacing d) at the grid points gx x gy; a
    neighbour beyond the last pixel is the first one, points off an unwrapped map give 0."""
    def axis(c, disp, oc, n):
        u = (c * scale + disp - oc) / d
        k = torch.floor(u)
        f = u - k
        k = k.long()
        ok = torch.ones_like(u) if wrap else ((k >= 0) & (k < n)).double()
        return k % n, (k + 1) % n, f, ok
    ix, ix1, fx, okx = axis(gx, dispx, o[0], S.shape[1])
    iy, iy1, fy, oky = axis(gy, dispy, o[1], S.shape[0])
    rows = S[iy] * (1 - fy)[:, None] + S[iy1] * fy[:, None]
    return (rows[:, ix] * (1 - fx) + rows[:, ix1] * fx) * okx * oky[:, None]


def _exact_wfs(case, seed):
    sysm, geom, fit = _system(*_key(case)), _geom(*_key(case)), _fit(*_key(case), "grid")
    cfg = sysm.cfg
    atms, isim, dm, noise = _screens(case, seed)
    ao = fit.act_offsets()
    out = []
    for b, atm in enumerate(atms):
        scr = [_t(s) for s in atm.screens]
        o = (-atm.n / 2 * atm.dx,) * 2
        for w in range(geom.nwfs):
            P = geom.powfs[geom.wfs_powfs[w]]
            gx = P.grid.ox + torch.arange(P.grid.nx, device=_dev(), dtype=torch.float64) * P.grid.dx
            gy = P.grid.oy + torch.arange(P.grid.ny, device=_dev(), dtype=torch.float64) * P.grid.dx
            tx, ty, hs = float(geom.thetax[w]), float(geom.thetay[w]), float(geom.hs[w])
            opd = 0
            for l, h in enumerate(cfg.atm_ht):
                opd = opd + _sample(scr[l], gx, gy, 1.0 - h / hs, h * tx - atm.vx[l] * cfg.sim_dt * isim,
                                    h * ty - atm.vy[l] * cfg.sim_dt * isim, o, atm.dx, True)
            for m, d in enumerate(fit.dms):
                a = dm[b, ao[m]:ao[m + 1]].double().reshape(d.amap.ny, d.amap.nx).to(_dev())
                opd = opd - _sample(a, gx, gy, 1.0 - d.ht / hs, d.ht * tx, d.ht * ty, (d.amap.ox, d.amap.oy),
                                    d.amap.dx, False)
            st = _t(P.stencils)
            wins = opd.unfold(0, P.W, 1).unfold(1, P.W, 1)
            iy = torch.as_tensor(P.iy0.astype(np.int64), device=_dev()) - 1
            ix = torch.as_tensor(P.ix0.astype(np.int64), device=_dev()) - 1
            win = wins[iy, ix].reshape(len(P.ix0), -1)
            sid = torch.as_tensor(P.stencil_id.astype(np.int64), device=_dev())
            g = [(st[sid, k] * win).sum(1).cpu().numpy() for k in (0, 1)]
            n1, n2 = _normals(noise, isim, w, b, len(P.ix0))
            nea = geom.nea[w]
            out += [g[0] + n1 * nea[0], g[1] + n2 * nea[1] + n1 * nea[2]]
    return np.concatenate(out).reshape(case["batch"], -1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "mvm":
        M, g = _matrix(case, seed)
        return g.double() @ M.double()
    if kind == "wfs":
        return _exact_wfs(case, seed)
    sysm = _system(*_key(case))
    if sysm.fdpcg is not None and case["batch"] < WIDE:
        return None  # see WIDE
    fit = _fit(*_key(case), case["fit"])
    x, a = _Solve(sysm, fit).step(_inputs(case, seed), case["maxit"], fit.maxit)
    if kind == "host":
        return a
    if kind == "serve":
        return a * torch.as_tensor(_mask(case, seed), device=a.device)[:, None]
    return {"commands": a, "layers": x} if sysm.fdpcg is None else {"commands": a}
