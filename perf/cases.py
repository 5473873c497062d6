"""Workloads of the gravity path, each run through the package's public entry
points, with inputs made from a seed.

What a host code does with this library falls into five kinds of call, and
each kind is a family of cases here:

* ``step``: one tree-force evaluation from and to page-locked host buffers
  (tvg_force_step_host), for the two problems the package has initial
  conditions for: a periodic Zel'dovich box at z = 50 and an isolated
  Hernquist halo; in the group form with node quadrupoles or monopoles and in
  the plain form, FP32 and FP64, relative and Barnes-Hut criterion, with and
  without the potential.
* ``rung``: a restarted hierarchical time step of a halo: upload of the whole
  particle state, new time steps, kick, drift, forces of the active rungs,
  kick, download.
* ``build``: the domain and tree part alone, as a host code with its own walk
  uses it: keys, sort, top nodes, the reference's tree (moments summed in
  particle order), with the permutation and the tree copied back.
* ``forcetest``: the FP64 direct sum that checks a force, Ewald-summed in a
  periodic box.
* ``mlp``: the gradient of one training batch of the learned Ewald correction.

Positions arrive in the order an initial-condition file has them (lattice
order, or random), not in Peano-Hilbert order; outputs come in the library's
order, with the ids that name the particles.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from tandav_b200 import gravity as G
from tandav_b200 import ics

DEV = "cuda"
BOX_MPC = 100.0
Z_START = 50.0
OPEN_BH = 0.25
FIND = G.CFG_FIND_DOMAIN
TIME_BINS = 32


def listed():
    return [
        # a test problem or an early convergence run: launches and host round
        # trips count
        {"name": "halo_3k_group", "kind": "step", "model": "halo", "n": 3001, "form": "group",
         "bytes": 4, "flags": FIND | G.CFG_QUADRUPOLE, "rel": 8e-3, "alpha": 1e-2, "bh": False,
         "vsize": 32},
        # the smallest cosmological box that the tests and examples step
        {"name": "box_32_group", "kind": "step", "model": "box", "n": 32, "form": "group",
         "bytes": 4, "flags": G.CFG_QUADRUPOLE, "rel": 8e-3, "alpha": 1e-2, "bh": False,
         "vsize": 32},
        # monopoles (the reference's moments, the library's default flags)
        {"name": "box_64_mono", "kind": "step", "model": "box", "n": 64, "form": "group",
         "bytes": 4, "flags": 0, "rel": 1e-3, "alpha": 4e-4, "bh": False, "vsize": 64},
        # a halo run in the reference's double precision, its default opening
        # and bundle size, in the group form
        {"name": "halo_400k_f64", "kind": "step", "model": "halo", "n": 400009, "form": "group",
         "bytes": 8, "flags": FIND, "rel": 5e-3, "alpha": 2.5e-4, "bh": False, "vsize": 64},
        # a production box of ordinary size, not a power of two
        {"name": "box_100_group", "kind": "step", "model": "box", "n": 100, "form": "group",
         "bytes": 4, "flags": G.CFG_QUADRUPOLE, "rel": 8e-3, "alpha": 1e-2, "bh": False,
         "vsize": 32},
        # the headline workload of bench.py
        {"name": "box_256_group", "kind": "step", "model": "box", "n": 256, "form": "group",
         "bytes": 4, "flags": G.CFG_QUADRUPOLE, "rel": 8e-3, "alpha": 1e-2, "bh": False,
         "vsize": 32},
        # the reference algorithm bit for bit, single precision, periodic
        {"name": "box_50_plain", "kind": "step", "model": "box", "n": 50, "form": "plain",
         "bytes": 4, "flags": G.CFG_FIX_SMALL_TOPNODES, "rel": 5e-3, "alpha": 2.5e-4, "bh": False,
         "vsize": 64},
        # the same in double precision with the potential (only this form has it)
        {"name": "halo_30k_plain_pot", "kind": "step", "model": "halo", "n": 30011, "form": "plain",
         "bytes": 8, "flags": G.CFG_FIX_SMALL_TOPNODES | G.CFG_POTENTIAL | FIND, "rel": 5e-3,
         "alpha": 2.5e-4, "bh": False, "vsize": 64},
        # one step of a halo's innermost rungs after a restart
        {"name": "halo_200k_rungs", "kind": "rung", "n": 200003, "depth": 2},
        # domain and tree for a host code that walks by itself
        {"name": "build_1500k", "kind": "build", "n": 1500007, "bytes": 4, "vsize": 64},
        # the force check beside a run
        {"name": "forcetest_64", "kind": "forcetest", "n": 64, "targets": 1000},
        # one batch of the learned correction's training
        {"name": "mlp_grad_16k", "kind": "mlp", "n": 16384},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges. The kinds come about as often as the
    listed cases have them."""
    kind = rng.choice(["box", "box", "box", "halo", "halo", "mono", "plain_box", "plain_halo",
                       "rung", "build", "forcetest", "mlp"])
    step = {"kind": "step", "form": "group", "bytes": 4, "alpha": 1e-2, "bh": False, "vsize": 32}
    if kind == "box":
        return dict(step, model="box", n=_log(rng, 16, 200), flags=G.CFG_QUADRUPOLE,
                    rel=rng.choice([5e-3, 8e-3, 1.2e-2]))
    if kind == "mono":
        return dict(step, model="box", n=_log(rng, 16, 40) if rng.random() < 0.5 else _log(rng, 60, 100),
                    flags=0, alpha=4e-4, rel=rng.choice([1e-3, 5e-3]), vsize=rng.choice([32, 64]))
    if kind == "halo":
        quad = rng.random() < 0.5
        return dict(step, model="halo", n=_log(rng, 2000, 1500000), bytes=rng.choice([4, 8]),
                    flags=FIND | (G.CFG_QUADRUPOLE if quad else 0), rel=8e-3 if quad else 5e-3,
                    bh=rng.random() < 0.25, vsize=rng.choice([32, 64]))
    if kind in ("plain_box", "plain_halo"):
        pot = G.CFG_POTENTIAL if rng.random() < 0.5 else 0
        c = dict(step, form="plain", bytes=rng.choice([4, 8]), flags=G.CFG_FIX_SMALL_TOPNODES | pot,
                 rel=5e-3, alpha=2.5e-4, bh=rng.random() < 0.25, vsize=rng.choice([32, 64]))
        if kind == "plain_box":
            return dict(c, model="box", n=_log(rng, 16, 56))
        return dict(c, model="halo", n=_log(rng, 3000, 60000), flags=c["flags"] | FIND)
    if kind == "rung":
        return {"kind": "rung", "n": _log(rng, 20000, 1000000), "depth": rng.randrange(5)}
    if kind == "build":
        return {"kind": "build", "n": _log(rng, 20000, 3000000), "bytes": rng.choice([4, 8]),
                "vsize": rng.choice([16, 32, 64])}
    if kind == "forcetest":
        return {"kind": "forcetest", "n": _log(rng, 16, 80), "targets": _log(rng, 10, 2000)}
    return {"kind": "mlp", "n": _log(rng, 1000, 200000)}


# ------------------------------------------------------------------ inputs

_SPECTRUM = {}


def _spectrum():
    """Cosmology and the tabulated square root of P(k) at z = 50."""
    if not _SPECTRUM:
        c = ics.Cosmology()
        a = 1.0 / (1.0 + Z_START)
        k = np.logspace(-3, 2.5, 4096)
        amp = np.sqrt(c.power_norm() * k ** c.n_s * c.transfer_eh_nowiggle(k) ** 2) * c.growth(a)
        _SPECTRUM.update(a=a, cosmo=c, logk=np.log(k), logamp=np.log(amp),
                         rho=3.0 * 0.1 ** 2 / (8.0 * math.pi * ics.GRAVITY) * c.omega_m)
    return _SPECTRUM


def _rng(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _interp(x, xp, fp):
    i = torch.clamp(torch.searchsorted(xp, x), 1, len(xp) - 1)
    t = (x - xp[i - 1]) / (xp[i] - xp[i - 1])
    return fp[i - 1] + t * (fp[i] - fp[i - 1])


def _box(n, seed):
    """Zel'dovich box of n^3 particles: positions and displacements (3, n^3),
    particle mass, box side, softening."""
    s = _spectrum()
    L = BOX_MPC * 1000.0
    dt = torch.float64 if n <= 160 else torch.float32
    wk = torch.fft.rfftn(torch.randn((n, n, n), generator=_rng(seed), device=DEV, dtype=dt))
    kf = 2.0 * math.pi / BOX_MPC
    k1 = torch.fft.fftfreq(n, d=1.0 / n, device=DEV, dtype=dt) * kf
    kz = torch.fft.rfftfreq(n, d=1.0 / n, device=DEV, dtype=dt) * kf
    k = (k1[:, None, None], k1[None, :, None], kz[None, None, :])
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    k2[0, 0, 0] = 1.0
    amp = torch.exp(_interp(0.5 * torch.log(k2), torch.tensor(s["logk"], device=DEV, dtype=dt),
                            torch.tensor(s["logamp"], device=DEV, dtype=dt)))
    amp[k2 > (kf * n / 2) ** 2] = 0.0
    amp[0, 0, 0] = 0.0
    wk = wk * (amp / k2) * math.sqrt(n ** 3 / BOX_MPC ** 3)
    disp = torch.stack([torch.fft.irfftn(1j * kc * wk, s=(n, n, n)).reshape(-1) * 1000.0
                        for kc in k])
    q = ((torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) * (L / n)).to(torch.float64)
    pos = torch.stack([a.reshape(-1) for a in torch.meshgrid(q, q, q, indexing="ij")])
    pos = torch.remainder(pos + disp, L)
    below = float(np.nextafter(np.float32(L), np.float32(0)))
    pos = torch.where(pos.float() >= L, torch.full_like(pos, below), pos)
    return pos, disp, s["rho"] * L ** 3 / n ** 3, L, L / n / 30.0


def _halo(n, seed):
    """Hernquist halo (a = 1, M = 1, cut at 100 a): positions and isotropic
    velocities of the local dispersion's size (3, n), particle mass, radii."""
    g = _rng(seed)
    u = torch.rand((5, n), generator=g, device=DEV, dtype=torch.float64)
    sq = torch.sqrt(u[0] * (100.0 / 101.0) ** 2)
    r = sq / (1.0 - sq)

    def direction(a, b):
        c = 2.0 * a - 1.0
        st, ph = torch.sqrt(1.0 - c * c), 2.0 * math.pi * b
        return torch.stack([st * torch.cos(ph), st * torch.sin(ph), c])

    pos = r * direction(u[1], u[2])
    vel = direction(u[3], u[4]) * torch.sqrt(0.3 * ics.GRAVITY * r / (1.0 + r) ** 2)
    return pos, vel, 1.0 / n, r


def _clumpy(n, seed):
    """Periodic box of side 1000: a uniform background and a quarter of the
    particles in 12 Gaussian clumps."""
    g = _rng(seed)
    pos = torch.rand((3, n), generator=g, device=DEV, dtype=torch.float64) * 1000.0
    m = n // 4
    centre = torch.rand((3, 12), generator=g, device=DEV, dtype=torch.float64) * 1000.0
    which = torch.randint(0, 12, (m,), generator=g, device=DEV)
    pos[:, :m] = torch.remainder(centre[:, which] + 20.0 * torch.randn(
        (3, m), generator=g, device=DEV, dtype=torch.float64), 1000.0)
    below = float(np.nextafter(np.float32(1000.0), np.float32(0)))
    return torch.where(pos.float() >= 1000.0, torch.full_like(pos, below), pos)


def _pinned(x, dtype=None):
    """A page-locked host copy of a tensor, as numpy."""
    x = x if dtype is None else x.to(dtype)
    out = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
    out.copy_(x)
    return out.numpy()


def _room(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _zeros(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True).numpy()


def _particles(case, seed):
    """Inputs of a step case as device tensors in the case's width:
    (pos, mass, last_acc, box, softening)."""
    ft = torch.float32 if case["bytes"] == 4 else torch.float64
    if case["model"] == "box":
        pos, disp, m, L, eps = _box(case["n"], seed)
        # linear theory: the acceleration is 4 pi G rho times the displacement
        last = 4.0 * math.pi * ics.GRAVITY * _spectrum()["rho"] * disp.norm(dim=0)
    else:
        pos, _, m, r = _halo(case["n"], seed)
        L, eps = 0.0, 0.01
        last = ics.GRAVITY / (1.0 + r) ** 2
    n = pos.shape[1]
    return pos.to(ft), torch.full((n,), m, device=DEV, dtype=ft), last.to(ft), L, eps


# ------------------------------------------------------------------- cases

def prepare(case, seed):
    return {"step": _prepare_step, "rung": _prepare_rung, "build": _prepare_build,
            "forcetest": _prepare_forcetest, "mlp": _prepare_mlp}[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_step(case, seed):
    pos, mass, last, L, eps = _particles(case, seed)
    n, ft = pos.shape[1], pos.dtype
    periodic = L > 0
    ctx = G.GravityContext(n, float_bytes=case["bytes"], periodic=periodic, boxsize=L, softening=eps,
                           open_bh=OPEN_BH, open_rel=case["rel"], vector_size=case["vsize"],
                           flags=case["flags"])
    if periodic:
        ctx.set_domain((0.0, 0.0, 0.0), L)
        ctx.ewald_init()
    ctx.set_ewald_opening(case["alpha"])
    return {"run": _run_step, "ctx": ctx, "n": n, "bh": case["bh"],
            "form": G.FORM_GROUP if case["form"] == "group" else G.FORM_PLAIN,
            "parts": G.WALK_GRAVITY | (G.WALK_EWALD if periodic else 0),
            "pot": bool(case["flags"] & G.CFG_POTENTIAL),
            "pos": _pinned(pos), "mass": _pinned(mass), "last": _pinned(last),
            "ids": np.arange(n, dtype=np.uint32),
            "grav_acc": _room((3, n), ft), "ids_out": _room((n,), torch.int32).view(np.uint32)}


def _run_step(s):
    ctx = s["ctx"]
    ctx.force_step_host(s["n"], s["pos"], s["mass"], last_acc=s["last"], ids=s["ids"],
                        grav_acc=s["grav_acc"], ids_out=s["ids_out"], form=s["form"],
                        use_bh=s["bh"], parts=s["parts"])
    out = {"grav_acc": s["grav_acc"], "ids": s["ids_out"]}
    if s["pot"]:
        out["grav_pot"] = ctx.download(G.F_GRAV_POT)["grav_pot"]
    return out


RUNG_FIELDS = (G.F_TYPE | G.F_TIME_BIN | G.F_IT_DRIFT | G.F_IT_KICK | G.F_ID | G.F_POS | G.F_VEL
               | G.F_ACC | G.F_MASS | G.F_GRAV_ACC | G.F_LAST_ACC)
RUNG_OUT = (G.F_TIME_BIN | G.F_IT_DRIFT | G.F_IT_KICK | G.F_ID | G.F_POS | G.F_VEL | G.F_ACC
            | G.F_GRAV_ACC | G.F_LAST_ACC)


def _struct(a):
    """tvg_particles of the named host arrays."""
    p = G.Particles()
    for name in ("type", "time_bin", "it_drift_pos", "it_kick_pos", "id", "mass", "last_acc_mag",
                 "tree_parent"):
        if name in a:
            setattr(p, name, a[name].ctypes.data)
    for name in ("pos", "vel", "acc", "grav_acc"):
        if name in a:
            for k in range(3):
                getattr(p, name)[k] = a[name][k].ctypes.data
    return p


def _prepare_rung(case, seed):
    """A halo in the middle of a hierarchical step: time bins from the
    accelerations, and a clock at which the rungs up to `depth` above the
    smallest one end their step."""
    n = case["n"]
    pos, vel, m, r = _halo(n, seed)
    acc = (-ics.GRAVITY / ((1.0 + r) ** 2 * r)) * pos
    ctx = G.GravityContext(n, float_bytes=4, softening=0.01, open_bh=OPEN_BH, open_rel=8e-3,
                           vector_size=32, flags=FIND | G.CFG_QUADRUPOLE)
    a = {"type": np.ones(n, np.int32), "id": np.arange(n, dtype=np.uint32),
         "pos": _pinned(pos, torch.float32), "vel": _pinned(vel, torch.float32),
         "acc": _pinned(acc, torch.float32), "grav_acc": _pinned(acc, torch.float32),
         "mass": np.full(n, m, np.float32), "last_acc_mag": _pinned(acc.norm(dim=0), torch.float32),
         "time_bin": np.full(n, TIME_BINS - 1, np.int32),
         "it_drift_pos": np.zeros(n, np.uint32), "it_kick_pos": np.zeros(n, np.uint32)}
    ctx.timeline_init(comoving=0, time_begin=0.0, time_end=10.0, hubble_constant=0.1,
                      omega_matter=0.3, omega_lambda=0.7, omega_rad=0.0, omega_0=1.0,
                      omega_baryon=0.0, rho_crit0=1.0, time_int_accuracy=0.025, max_timestep=0.05,
                      displ_constraint=0.25)
    src = _struct(a)
    ctx._check(ctx.lib.tvg_upload(ctx.ctx, C.c_int64(n), C.byref(src), C.c_uint32(RUNG_FIELDS)),
               "upload")
    ctx.n = n
    ctx.set_new_timesteps()
    st = ctx.timeline()
    bins = ctx.download(G.F_TIME_BIN)["time_bin"].astype(np.uint32)
    now = ((1 << case["depth"]) - 1 if case["depth"] else 2) << st.time_bin_min
    st.current = now
    st.time_current = now * st.step_min
    st.next = now + (1 << st.time_bin_min)
    st.max_active_bin = (st.next & -st.next).bit_length() - 1
    st.first_step = 0
    st.next_sync_point = 1 << st.time_bin_max
    began = (np.uint32(now) >> bins) << bins
    a.update(time_bin=bins.astype(np.int32), it_drift_pos=began.copy(), it_kick_pos=began.copy())
    a = {k: _pinned(torch.from_numpy(v.view(np.int32) if v.dtype == np.uint32 else v)).view(v.dtype)
         for k, v in a.items()}
    dt = {"pos": 3, "vel": 3, "acc": 3, "grav_acc": 3, "last_acc_mag": 1, "time_bin": 0, "id": 0,
          "it_drift_pos": 0, "it_kick_pos": 0}
    out = {}
    for k, w in dt.items():
        t = _room((3, n) if w == 3 else (n,), torch.float32 if w else torch.int32)
        out[k] = t.view(a[k].dtype)
    return {"run": _run_rung, "ctx": ctx, "n": n, "clock": st, "in": a, "out": out,
            "src": _struct(a), "dst": _struct(out)}


def _run_rung(s):
    ctx = s["ctx"]
    ctx._check(ctx.lib.tvg_upload(ctx.ctx, C.c_int64(s["n"]), C.byref(s["src"]),
                                  C.c_uint32(RUNG_FIELDS)), "upload")
    ctx.n = s["n"]
    ctx.set_timeline(s["clock"])
    ctx.set_new_timesteps()
    ctx.kick_first_halfstep()
    ctx.drift_to_sync_point()
    ctx.compute_acceleration(form=G.FORM_GROUP, parts=G.WALK_GRAVITY)
    ctx.kick_second_halfstep()
    ctx._check(ctx.lib.tvg_download(ctx.ctx, C.byref(s["dst"]), C.c_uint32(RUNG_OUT)), "download")
    return dict(s["out"])


def _prepare_build(case, seed):
    n, ft = case["n"], torch.float32 if case["bytes"] == 4 else torch.float64
    ctx = G.GravityContext(n, float_bytes=case["bytes"], periodic=True, boxsize=1000.0, softening=0.1,
                           vector_size=case["vsize"])
    ctx.set_domain((0.0, 0.0, 0.0), 1000.0)
    dt = G.TREE_DTYPE[case["bytes"]]
    cap = n // 2 + 100000
    return {"run": _run_build, "ctx": ctx, "n": n, "pos": _pinned(_clumpy(n, seed), ft),
            "mass": _pinned(torch.full((n,), 1.0 / n, device=DEV), ft),
            "perm": _room((n,), torch.int32).view(np.uint32),
            "parent": _room((n,), torch.int32),
            "tree": _zeros((cap * dt.itemsize,), torch.uint8).view(dt),
            "top": np.zeros(64, G.TOPNODE_DTYPE)}


def _run_build(s):
    ctx, tree = s["ctx"], s["tree"]
    ctx.upload_fields(s["n"], pos=s["pos"], mass=s["mass"])
    ctx.peano_keys()
    ctx._check(ctx.lib.tvg_sort_particles(ctx.ctx, C.c_void_p(s["perm"].ctypes.data)), "sort")
    ctx.top_nodes()
    ctx.tree_build(exact_moments=True)
    nn, nt = C.c_int64(), C.c_int32()
    ctx._check(ctx.lib.tvg_download_tree(ctx.ctx, C.c_void_p(tree.ctypes.data), C.c_int64(len(tree)),
                                         C.byref(nn), C.c_void_p(s["top"].ctypes.data),
                                         C.c_int32(len(s["top"])), C.byref(nt)), "download_tree")
    ctx._check(ctx.lib.tvg_download(ctx.ctx, C.byref(_struct({"tree_parent": s["parent"]})),
                                    C.c_uint32(G.F_TREE_PARENT)), "download")
    out = {"tree_" + k: tree[k] for k in tree.dtype.names}
    out.update({"top_" + k: s["top"][k] for k in ("First_Part", "Npart", "Mass", "CoM")})
    out.update(top_Key=s["top"]["Key"].view(np.int64), perm=s["perm"], parent=s["parent"],
               nodes=nn.value, tops=nt.value)
    return out


def _prepare_forcetest(case, seed):
    pos, disp, m, L, eps = _box(case["n"], seed)
    n = pos.shape[1]
    # the force being checked: linear theory, rounded as a snapshot holds it
    acc = 4.0 * math.pi * ics.GRAVITY * _spectrum()["rho"] * disp
    ctx = G.GravityContext(n, float_bytes=4, periodic=True, boxsize=L, softening=eps)
    ctx.set_domain((0.0, 0.0, 0.0), L)
    ctx.upload(pos.float().cpu().numpy(), np.full(n, m, np.float32),
               grav_acc=acc.float().cpu().numpy())
    return {"run": _run_forcetest, "ctx": ctx, "targets": _targets(n, case, seed)}


def _targets(n, case, seed):
    return np.sort(np.random.default_rng(seed).choice(n, min(case["targets"], n), replace=False))


def _run_forcetest(s):
    direct, tree, err = s["ctx"].forcetest(s["targets"])
    return {"direct": direct, "tree": tree, "rms": err["rms"], "p99": err["p99"],
            "mean": err["mean"], "max": err["max"]}


def _mlp_inputs(case, seed):
    rng = np.random.default_rng(seed)
    p = (rng.standard_normal(G.MLP_NPARAM) * 0.3).astype(np.float32)
    x = (rng.random((case["n"], 3)) * 0.5).astype(np.float32)
    y = (rng.standard_normal((case["n"], 3)) * 0.5).astype(np.float32)
    return p, x, y


def _prepare_mlp(case, seed):
    p, x, y = _mlp_inputs(case, seed)
    ctx = G.GravityContext(1024, periodic=True, boxsize=1.0)
    ctx.mlp_weights(p)
    return {"run": _run_mlp, "ctx": ctx, "x": x, "y": y}


def _run_mlp(s):
    g, loss = s["ctx"].mlp_grad(s["x"], s["y"])
    return {"grad": g, "loss": loss}


# -------------------------------------------------------------------- work

def work(case):
    """Bytes of a pass's inputs and outputs, and its arithmetic: the terms of
    the sums at the case's opening, by the interaction counts per particle
    that a tree of this kind needs, and by the formulas of the direct sums."""
    kind = case["kind"]
    if kind == "step":
        n = case["n"] ** 3 if case["model"] == "box" else case["n"]
        f = case["bytes"]
        out = 4 * f + 4 if case["flags"] & G.CFG_POTENTIAL else 3 * f + 4
        nbytes = n * (5 * f + 4 + out)
        # measured interactions per particle at these openings
        if case["flags"] & G.CFG_QUADRUPOLE:
            per, flop = (8500.0 if case["model"] == "box" else 1700.0), 45.0
        elif case["model"] == "box":
            per, flop = 30000.0 * (5e-3 / case["rel"]) ** 0.6, 20.0
        else:
            per, flop = (6000.0 if case["bh"] else 2300.0), 20.0
        if case["form"] == "plain":
            per, flop = (1e5, 80.0) if case["model"] == "box" else (8400.0, 20.0)
        return {"bytes": nbytes, "flops": n * min(per, float(n)) * flop}
    if kind == "rung":
        n = case["n"]
        return {"bytes": n * (4 * 5 + 4 * 14 + 4 * 4 + 4 * 13), "flops": 1000.0 * 40.0 * n}
    if kind == "build":
        n, f = case["n"], case["bytes"]
        return {"bytes": n * (4 * f + 8) + (n / 5.0) * (16 + 10 * f), "flops": 0}
    if kind == "forcetest":
        n, t = case["n"] ** 3, min(case["targets"], case["n"] ** 3)
        # real space: ~100 flop a pair; k space: 28,000 waves of the half
        # space, 8 flop for each source's and each target's term
        return {"bytes": 16 * n + 56 * t, "flops": 100.0 * n * t + 28000.0 * 8 * (n + t)}
    n = case["n"]
    return {"bytes": 24 * n + 8 * G.MLP_NPARAM, "flops": 6.0 * 4608 * n}


# ------------------------------------------------------------ 64-bit values

EXACT_MAX = {"halo": 420000, "box": 280000}


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        pos, mass, _, L, eps = _particles(case, seed)
        if pos.shape[1] > EXACT_MAX[case["model"]] or case["bh"]:
            return None
        pos, mass = pos.double(), mass.double()
        origin, size = (torch.zeros(3, device=DEV, dtype=torch.float64), L) if L else _domain(pos)
        order = _hilbert_order(pos, origin, size)
        pos, mass = pos[:, order].contiguous(), mass[order]
        acc, pot = _direct(pos, pos, mass, L, eps, bool(case["flags"] & G.CFG_POTENTIAL))
        out = {"grav_acc": acc.cpu().numpy(), "ids": None}
        if case["flags"] & G.CFG_POTENTIAL:
            out["grav_pot"] = None if pot is None else pot.cpu().numpy()
        return out
    if kind == "forcetest":
        if case["n"] ** 3 * case["targets"] > 2e9:
            return None
        pos, disp, m, L, eps = _box(case["n"], seed)
        pos = pos.float().double()
        mass = torch.full((pos.shape[1],), float(np.float32(m)), device=DEV, dtype=torch.float64)
        t = torch.from_numpy(_targets(pos.shape[1], case, seed)).to(DEV)
        acc, _ = _direct(pos[:, t], pos, mass, L, eps, False)
        tree = (4.0 * math.pi * ics.GRAVITY * _spectrum()["rho"] * disp).float().double()[:, t]
        e = ((tree - acc).norm(dim=0) / acc.norm(dim=0)).sort()[0]
        return {"direct": acc.cpu().numpy(), "tree": tree.cpu().numpy(),
                "rms": float(e.square().mean().sqrt()),
                "p99": float(e[max(math.ceil(0.99 * len(e)) - 1, 0)]),
                "mean": float(e.mean()), "max": float(e[-1])}
    if kind == "mlp":
        return _mlp_exact(case, seed)
    return None


def _domain(pos):
    """Isolated domain: centred on the medians, 2.001 times the largest offset."""
    n = pos.shape[1]
    c = torch.stack([p[1:].sort()[0][(n >> 1) - 1] for p in pos])
    size = 2.001 * float((pos - c[:, None]).abs().max())
    return c - 0.5 * size, size


def _hilbert_order(pos, origin, size):
    """Order of the particles along the Peano-Hilbert curve (Skilling 2004) of
    63 levels, the first 42 compared."""
    x = [((pos[k] - origin[k]) * (2.0 ** 63 / size)).to(torch.int64) for k in range(3)]
    for b in range(63, 0, -1):
        mask = (1 << b) - 1
        for i in range(3):
            hit = ((x[i] >> b) & 1) != 0
            t = (x[0] ^ x[i]) & mask
            x0 = torch.where(hit, x[0] ^ mask, x[0] ^ t)
            if i:
                x[i] = torch.where(hit, x[i], x[i] ^ t)
            else:
                x0 = torch.where(hit, x[0] ^ mask, x[0])
            x[0] = x0
    x[1] = x[1] ^ x[0]
    x[2] = x[2] ^ x[1]
    p = x[2].clone()
    for s in (1, 2, 4, 8, 16, 32):
        p = p ^ (p >> s)
    above = p ^ x[2]
    x = [v ^ above for v in x]
    words = []
    for top in (62, 41):
        w = torch.zeros_like(x[0])
        for lvl in range(21):
            for v in x:
                w = (w << 1) | ((v >> (top - lvl)) & 1)
        words.append(w)
    order = torch.argsort(words[1], stable=True)
    return order[torch.argsort(words[0][order], stable=True)]


def _direct(tgt, pos, mass, L, eps, want_pot):
    """Direct sum over all sources with the softened kernel on the nearest
    image, Ewald-summed when L > 0: accelerations (3, nt), and the potential
    of an isolated system."""
    h = -41.0 / 32.0 * eps
    n, nt = pos.shape[1], tgt.shape[1]
    acc = torch.zeros((3, nt), device=DEV, dtype=torch.float64)
    pot = torch.zeros(nt, device=DEV, dtype=torch.float64) if want_pot and not L else None
    alpha = 10.0 / L if L else 0.0
    rows = max(1, (1 << 26) // n)
    for i in range(0, nt, rows):
        t = tgt[:, i:i + rows]
        d = pos[:, None, :] - t[:, :, None]
        if L:
            d -= L * torch.round(d / L)
        r2 = (d * d).sum(0)
        own = r2 == 0
        r2 = torch.where(own, torch.ones_like(r2), r2)
        ri = torch.rsqrt(r2)
        inner = (r2 < h * h) & ~own
        u2 = r2 / (h * h)
        fac = torch.where(inner, (175.0 - u2 * (294.0 - 135.0 * u2)) / (16.0 * h ** 3), ri ** 3)
        if L:
            r = r2 * ri
            g = 2.0 * alpha / math.sqrt(math.pi) * r * torch.exp(-(alpha * r) ** 2)
            fac -= (torch.erf(alpha * r) - g) * ri ** 3
        fac *= mass * ~own
        acc[:, i:i + rows] = (fac * d).sum(2)
        if pot is not None:
            f = torch.where(inner, (u2 * (175.0 - u2 * (147.0 - 45.0 * u2)) - 105.0) / (32.0 * h), ri)
            pot[i:i + rows] = (f * mass * ~own).sum(1)
        del d, r2, ri, u2, fac
    if L:
        m = 17
        hh = torch.arange(-m, m + 1, device=DEV, dtype=torch.float64)
        k = torch.stack([v.reshape(-1) for v in torch.meshgrid(hh, hh, hh, indexing="ij")])
        k2 = (k * k).sum(0)
        half = (k[0] > 0) | ((k[0] == 0) & ((k[1] > 0) | ((k[1] == 0) & (k[2] > 0))))
        k = k[:, half & (k2 <= m * m)]
        k2 = (k * k).sum(0)
        w = 4.0 / L ** 2 * torch.exp(-(math.pi / (alpha * L)) ** 2 * k2) / k2
        kk = k * (2.0 * math.pi / L)
        sc = torch.zeros_like(w)
        ss = torch.zeros_like(w)
        step = 4096
        for j in range(0, n, step):
            ph = kk.T @ pos[:, j:j + step]
            sc += torch.cos(ph) @ mass[j:j + step]
            ss += torch.sin(ph) @ mass[j:j + step]
        for i in range(0, nt, step):
            ph = tgt[:, i:i + step].T @ kk
            acc[:, i:i + step] += k @ ((torch.cos(ph) * ss - torch.sin(ph) * sc) * w).T
    return acc * ics.GRAVITY, None if pot is None else pot * ics.GRAVITY


def _mlp_exact(case, seed):
    """Gradient of the mean square loss of a 3-64-64-3 tanh network in 64 bits."""
    p, x, y = (torch.from_numpy(a).to(DEV).double() for a in _mlp_inputs(case, seed))
    h, w = 64, p[:4611].clone().requires_grad_(True)
    w1, b1, w2, b2, w3, b3 = torch.split(w, [3 * h, h, h * h, h, 3 * h, 3])
    a = torch.tanh((4.0 * x - 1.0) @ w1.view(h, 3).T + b1)
    a = torch.tanh(a @ w2.view(h, h).T + b2)
    r = a @ w3.view(3, h).T + b3 - y
    r.square().mean().backward()
    g = torch.cat([w.grad, torch.zeros(len(p) - 4611, device=DEV, dtype=torch.float64)])
    return {"grad": g.cpu().numpy(), "loss": float(r.detach().square().sum())}
