"""The work that users of this library have it do, as cases that can be timed.

Every case goes through the C entry points that an lsmpqs program calls, on host
arrays as they hold them (the arrays travel inside the call), over the range of
volumes this repository's configurations, tests and benchmark use:

* ``constcurv``  one curvature step, ``constCurvModel3d`` (variable coefficients,
  contact angle > 0): inner TVD-RK steps, trapping, three reinitialisations,
  volumes.  The quantum of every drainage / imbibition run with a wetting solid;
* ``novar``      the same step for a zero contact angle, ``constCurvModel3dNoVar``;
* ``ladder``     a drainage or imbibition ladder of one or several uneven volumes,
  ``qssgpu_ladder_batch`` (what ``drain_model3d`` does, without step files);
* ``rhs``        one WENO5 right-hand side through ``getrhs3d5th_``, as a program
  that links the kernels one by one calls it;
* ``maskprep``   a segmented 8-bit image to a signed distance, ``qssgpu_create_mask_ubc``
  (reinitialisation sweeps only);
* ``trap``       ``trapComponents_mask``: two 26-connected labellings and the masks;
* ``adjoint``    loss and gradient with respect to a contact-angle field,
  ``qssgpu_adjoint_theta`` (forward and backward).

Grain packs are overlapping spheres (lognormal radii) on a jittered lattice,
which gives the porosities 0.3..0.4 and the signed distances of the seeded packs
of ``synthetic.py`` and is quick to make on the GPU.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lsmpqs-1.0_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)
import qssgpu as Q  # noqa: E402

DX, NG = 0.04, 3
RAD = 3.14159 / 180  # the reference's degree
_lib = None


def lib():
    global _lib
    if _lib is None:
        _lib = Q.load(Q.GPU_LIB)
    return _lib


# ---------------------------------------------------------------------------
# cases

def listed():
    return [
        # a test-sized volume: launches, copies and host control flow are the time
        {"name": "constcurv_24", "kind": "constcurv", "nx": 24, "ny": 24, "nz": 24, "theta": 10.0, "order": 5,
         "time": 3, "radius": 4.0, "tplot": 0.02},
        # a cropped sample with ragged sides (no side a multiple of a tile)
        {"name": "constcurv_97x61x83", "kind": "constcurv", "nx": 97, "ny": 61, "nz": 83, "theta": 30.0, "order": 5,
         "time": 3, "radius": 6.0, "tplot": 0.02},
        # the usual size of a segmented subvolume
        {"name": "constcurv_192", "kind": "constcurv", "nx": 192, "ny": 192, "nz": 192, "theta": 40.0, "order": 5,
         "time": 3, "radius": 8.0, "tplot": 0.02},
        # a large volume: nothing but device arithmetic counts
        {"name": "constcurv_320", "kind": "constcurv", "nx": 320, "ny": 320, "nz": 320, "theta": 40.0, "order": 5,
         "time": 3, "radius": 8.0, "tplot": 0.02},
        # zero contact angle at the order of the 64^3 configuration, on a larger sample
        {"name": "novar_eno2_128", "kind": "novar", "nx": 128, "ny": 128, "nz": 128, "theta": 0.0, "order": 2,
         "time": 2, "radius": 6.0, "tplot": 0.02},
        # the 64^3 ENO2 / TVD-RK2 drainage ladder of the reference's own CPU size
        {"name": "drain_eno2_64", "kind": "ladder", "drain": True, "volumes": 1, "nx": 64, "ny": 64, "nz": 64,
         "theta": 0.0, "order": 2, "time": 2, "radius": 5.0, "tplot": 0.05, "steps": 4},
        # drainage of several uneven volumes at once (a batch of samples)
        {"name": "drain_batch6_48to96", "kind": "ladder", "drain": True, "volumes": 6, "nx": 48, "ny": 96, "nz": 96,
         "theta": 35.0, "order": 5, "time": 3, "radius": 6.0, "tplot": 0.02, "steps": 2},
        # imbibition (decreasing curvature, wetting blobs conserved), nearly neutral angle
        {"name": "imbibe_110", "kind": "ladder", "drain": False, "volumes": 1, "nx": 110, "ny": 110, "nz": 110,
         "theta": 10.0, "order": 5, "time": 3, "radius": 6.0, "tplot": 0.02, "steps": 2},
        # one kernel of the Fortran interface on host arrays
        {"name": "rhs_weno5_130x96x75", "kind": "rhs", "nx": 130, "ny": 96, "nz": 75, "theta": 30.0, "radius": 6.0},
        # image to signed distance, the preprocessing of every sample
        {"name": "maskprep_200", "kind": "maskprep", "nx": 200, "ny": 200, "nz": 200, "radius": 7.0},
        # trapped phases of a well-drained large volume
        {"name": "trap_256", "kind": "trap", "nx": 256, "ny": 256, "nz": 256, "radius": 6.0},
        # gradient of a 20-step run with respect to the contact angle, one checkpoint halfway
        {"name": "adjoint_72", "kind": "adjoint", "nx": 72, "ny": 72, "nz": 72, "theta": 40.0, "radius": 6.0,
         "steps": 20, "ckpt": 10},
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["constcurv"] * 5 + ["novar"] * 2 + ["ladder"] * 2 + ["rhs", "maskprep", "trap", "adjoint"])
    lo, hi = {"constcurv": (20, 300), "novar": (24, 200), "ladder": (24, 110), "rhs": (20, 150),
              "maskprep": (32, 240), "trap": (32, 256), "adjoint": (24, 72)}[kind]
    s = _side(rng, lo, hi)
    dims = [max(lo, min(hi, int(round(s * math.exp(rng.uniform(-0.35, 0.35)))))) for _ in range(3)]
    if kind == "adjoint":  # cubes, as the loss is set up on
        dims = [s] * 3
    c = {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2], "radius": round(rng.uniform(4.0, 8.0), 2)}
    if kind in ("constcurv", "ladder"):
        c.update(theta=round(rng.uniform(5.0, 60.0), 1), order=rng.choice([5, 5, 5, 2]), time=3,
                 tplot=rng.choice([0.02, 0.03]))
        if c["order"] == 2:
            c["time"] = 2
    if kind == "novar":
        c.update(theta=0.0, order=rng.choice([2, 3]), time=rng.choice([2, 3]), tplot=rng.choice([0.02, 0.03]))
        if c["order"] == 3:  # the reference's ENO3 x-stencil reads phi(i+3,j,j)
            c["ny"], c["nz"] = min(dims[1], dims[2]), max(dims[1], dims[2])
    if kind == "ladder":
        c.update(drain=rng.random() < 0.6, volumes=rng.choice([1, 1, 2, 4]), steps=2)
    if kind == "rhs":
        c.update(theta=round(rng.uniform(5.0, 60.0), 1))
    if kind == "adjoint":
        c.update(theta=round(rng.uniform(20.0, 50.0), 1), steps=rng.choice([8, 16, 20]), ckpt=rng.choice([0, 4, 10]))
    return c


# ---------------------------------------------------------------------------
# inputs

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _pack(dims, radius, seed, porosity=0.35, cutoff=6.0):
    """Signed distance (ghost box, positive in grains, clamped at -cutoff voxels)
    to overlapping spheres with lognormal radii on a jittered lattice."""
    nx, ny, nz = (d + 2 * NG for d in dims)
    r = np.random.default_rng(seed)
    cell = radius * (4.18879 * math.exp(4.5 * 0.2 ** 2) / math.log(1 / porosity)) ** (1 / 3)
    m = [int(math.ceil(d / cell)) + 4 for d in (nx, ny, nz)]
    jit = r.uniform(0.0, 1.0, (m[2], m[1], m[0], 3))
    rad = np.minimum(radius * r.lognormal(-0.02, 0.2, (m[2], m[1], m[0])), 1.8 * radius)
    dev = _dev()
    at = torch.as_tensor(np.concatenate([jit, rad[..., None]], axis=-1), device=dev)  # cell, (x, y, z, radius)
    ax = [torch.arange(d, dtype=torch.float64, device=dev) for d in (nx, ny, nz)]
    ci = [torch.floor(a / cell).long() + 2 for a in ax]
    best = torch.full((nz, ny, nx), -cutoff, dtype=torch.float64, device=dev)
    for ok in range(-2, 3):
        for oj in range(-2, 3):
            for oi in range(-2, 3):
                g = at[(ci[2] + ok)[:, None, None], (ci[1] + oj)[None, :, None], (ci[0] + oi)[None, None, :]]
                d2 = ((ci[0] + oi - 2)[None, None, :] + g[..., 0]) * cell - ax[0][None, None, :]
                d2 = d2 * d2
                t = ((ci[1] + oj - 2)[None, :, None] + g[..., 1]) * cell - ax[1][None, :, None]
                d2 += t * t
                t = ((ci[2] + ok - 2)[:, None, None] + g[..., 2]) * cell - ax[2][:, None, None]
                d2 += t * t
                torch.maximum(best, g[..., 3] - torch.sqrt(d2), out=best)
                del g, d2, t
    return best * DX


def _inlet(dims, mask):
    """createInitFromMask: a non-wetting sphere at the inlet face, then max(mask, phi)."""
    ax = [torch.arange(d + 2 * NG, dtype=torch.float64, device=mask.device) * DX for d in dims]
    length = dims[0] * DX
    radius = 0.7 * length
    cx, cy, cz = NG * DX - 0.7 * radius, NG * DX + 0.5 * dims[1] * DX, NG * DX + 0.5 * dims[2] * DX
    d = torch.sqrt((ax[2] - cz)[:, None, None] ** 2 + (ax[1] - cy)[None, :, None] ** 2
                   + (ax[0] - cx)[None, None, :] ** 2) - radius
    return torch.maximum(mask, d)


class Sample:
    """One volume as a program holds it: struct, grid, options, arrays."""

    def __init__(self, dims, case, seed):
        self.dims = tuple(dims)
        self.g = Q.make_grid(lib(), self.dims)
        self.v = Q.Volume(self.g)
        self.o = Q.default_options(lib())
        self.mask = _pack(self.dims, case["radius"], seed)
        self.v["mask"][...] = self.mask.cpu().numpy()
        self.phi0 = _inlet(self.dims, self.mask).cpu().numpy()
        self.v["phi"][...] = self.phi0
        o = self.o
        o.theta = case.get("theta", 0.0) * RAD
        o.order_space_accur, o.order_time_accur = case.get("order", 5), case.get("time", 3)
        o.a, o.b, o.dc, o.check_connectivity = 1.25, 0.04, 0.9722, 1
        o.tplot = o.tmax = case.get("tplot", 0.02)

    def __del__(self):
        if getattr(self, "v", None) is not None:
            lib().qssgpu_release(C.byref(self.v.p))

    def model_setup(self):
        """What drain_model3d does before its first curvature step, through the C API."""
        L, v, o, g = lib(), self.v, self.o, self.g
        gp = C.byref(g)
        for n in ("mask_w", "mask_nw"):
            L.initializeDisconnectedMasks(Q.dptr(v[n]), gp)
        dxs = [Q.dref(g.dx[d]) for d in range(3)]
        L.getcentralgrad3dorder2_(Q.dptr(v["mask_x"]), Q.dptr(v["mask_y"]), Q.dptr(v["mask_z"]), *Q.gb_args(g),
                                  Q.dptr(v["mask"]), *Q.gb_args(g), *Q.fb_args(g), *dxs)
        L.setSpaceDerivFunc(gp, C.byref(o))
        L.setThetaOverlap(C.byref(v.p), gp, C.byref(o))
        L.getMainInd_new(C.byref(o), C.byref(v.p), gp)
        inv = 1.0 / g.dx[0]
        if o.theta > 0:
            bm, um = C.c_double(0), C.c_double(0)
            L.setvarcurvadv3d_(*[Q.dptr(v[n]) for n in ("mask", "mask_x", "mask_y", "mask_z", "curvature_coeff",
                                                        "external_velocity_x", "external_velocity_y",
                                                        "external_velocity_z")], C.byref(bm), C.byref(um),
                               Q.dref(o.b), *Q.gb_args(g), *Q.fb_args(g), Q.dref(g.dx[0]))
            o.b_max_over_dx, o.max_U_over_dx = bm.value, um.value
            L.setvarnorm3d_(*[Q.dptr(v[n]) for n in ("mask", "mask_x", "mask_y", "mask_z", "normal_velocity")],
                            Q.dref(o.a), Q.dref(o.theta), *Q.gb_args(g), *Q.fb_args(g), Q.dref(g.dx[0]))
        else:
            o.b_max_over_dx, o.max_U_over_dx = 2 * o.b * 3 * inv * inv, 0.0
        Q.check(L)


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _batch_dims(case):
    """Sides of a ladder's volumes: nx .. max side, spread evenly, the last one whole."""
    n = case["volumes"]
    if n == 1:
        return [_dims(case)]
    lo, hi = min(_dims(case)), max(_dims(case))
    return [(lo + (hi - lo) * k // (n - 1),) * 3 for k in range(n)]


def _smooth_angle(dims, mean_deg, seed):
    """A contact-angle field (radians, ghost box): a few smooth waves around the mean."""
    r = np.random.default_rng(seed)
    ax = [torch.arange(d + 2 * NG, dtype=torch.float64, device=_dev()) / d for d in dims]
    out = torch.full([d + 2 * NG for d in dims[::-1]], mean_deg, dtype=torch.float64, device=_dev())
    for _ in range(4):
        f, p = r.uniform(1.0, 9.0, 3), r.uniform(0, 6.28, 3)
        out = out + 3.0 * (torch.sin(f[2] * ax[2] + p[2])[:, None, None] * torch.sin(f[1] * ax[1] + p[1])[None, :, None]
                           * torch.sin(f[0] * ax[0] + p[0])[None, None, :])
    return (out * (math.pi / 180)).cpu().numpy()


def _heaviside(phi, eps):
    h = 0.5 + phi / (2 * eps) + np.sin(math.pi * phi / eps) / (2 * math.pi)
    return np.where(phi < -eps, 0.0, np.where(phi > eps, 1.0, h))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ladder":
        vols = []
        for k, d in enumerate(_batch_dims(case)):
            s = Sample(d, case, 1000 * seed + k)
            o = s.o
            if case["drain"]:
                o.a = 1.25
                o.amax = o.a + (case["steps"] - 0.5) * o.b * o.dc
            else:
                o.a = 3.0
                o.amin = o.a - (case["steps"] - 0.5) * o.b * o.dc
            vols.append(s)
        n = len(vols)
        return {"kind": kind, "vols": vols, "drain": 1 if case["drain"] else 0,
                "po": (C.POINTER(Q.Options) * n)(*[C.pointer(s.o) for s in vols]),
                "pp": (C.POINTER(Q.QSSDataArrays) * n)(*[C.pointer(s.v.p) for s in vols]),
                "pg": (C.POINTER(Q.Grid) * n)(*[C.pointer(s.g) for s in vols])}
    s = Sample(_dims(case), case, seed)
    st = {"kind": kind, "s": s, "case": case}
    if kind in ("constcurv", "novar", "rhs"):
        s.model_setup()
    if kind == "maskprep":
        fb = s.v.fb("mask")
        st["ubc"] = np.ascontiguousarray(np.where(fb >= 0, 255, 0).astype(np.uint8))
        s.v["mask"][...] = 0
    if kind == "trap":
        # a drained state: the pore space less a second, sparser pack of wetting patches
        w = _pack(s.dims, 0.8 * case["radius"], seed + 7777, porosity=0.8)
        st["phi0"] = torch.maximum(s.mask, w).cpu().numpy()
        lib().initializeDisconnectedMasks(Q.dptr(s.v["mask_nw"]), C.byref(s.g))
        st["mask_nw0"] = s.v["mask_nw"].copy()
        s.phi0 = None
        lib().getMainInd_new(C.byref(s.o), C.byref(s.v.p), C.byref(s.g))
    if kind == "adjoint":
        o = s.o
        o.a, o.overlap = 0.2 / DX, 0.0
        st["dt"] = 0.5 / (2 * o.b * 3 / DX ** 2 + 2.0 / DX + abs(o.a) * math.sqrt(3) / DX)
        st["theta"] = _smooth_angle(s.dims, case["theta"], seed)
        phi_t = np.zeros(s.v.shape)
        loss = C.c_double(0)
        lib().qssgpu_forward_theta(C.byref(o), C.byref(s.v.p), C.byref(s.g),
                                   Q.dptr(_smooth_angle(s.dims, case["theta"] + 10, seed + 1)),
                                   Q.dptr(np.zeros(s.v.shape)),
                                   case["steps"], st["dt"], C.byref(loss), Q.dptr(phi_t))
        st["target"] = _heaviside(phi_t, 1.5 * DX)
        st["grad"] = np.zeros(s.v.shape)
    s.mask = None
    Q.check(lib())
    return st


# ---------------------------------------------------------------------------
# one pass

MODEL_OUT = ("phi", "phi_prev", "phi_next", "mask_w", "mask_nw", "connectivity", "phi_bin")


def run(st):
    L, kind = lib(), st["kind"]
    if kind == "ladder":
        for s in st["vols"]:  # the ladder starts from the inlet again
            s.v["phi"][...] = s.phi0
        n = len(st["vols"])
        if L.qssgpu_ladder_batch(st["drain"], n, st["po"], st["pp"], st["pg"], None, None, 0):
            Q.check(L)
        return [{k: s.v[k] for k in ("phi", "phi_next", "mask_w", "mask_nw", "connectivity")} for s in st["vols"]]
    s = st["s"]
    v, o, g = s.v, s.o, s.g
    if kind in ("constcurv", "novar"):
        v["phi"][...] = s.phi0  # every pass is a curvature step from the same level set
        if kind == "constcurv":
            t = L.constCurvModel3d(C.byref(o), C.byref(v.p), C.byref(g), None)
        else:
            t = L.constCurvModel3dNoVar(C.byref(o), C.byref(v.p), C.byref(g), None, o.a)
        Q.check(L)
        return {"t": t, **{k: v[k] for k in MODEL_OUT}}
    if kind == "rhs":
        h = C.c_double(0)
        L.getrhs3d5th_(*[Q.dptr(v[n]) for n in ("phi", "normal_velocity", "curvature_coeff", "external_velocity_x",
                                                "external_velocity_y", "external_velocity_z")], C.byref(h),
                       Q.dptr(v["lse_rhs"]), *Q.gb_args(g), *Q.fb_args(g), *[Q.dref(g.dx[d]) for d in range(3)])
        Q.check(L)
        return {"rhs": v["lse_rhs"], "h": h.value}
    if kind == "maskprep":
        L.qssgpu_create_mask_ubc(st["ubc"].ctypes.data_as(C.POINTER(C.c_ubyte)), C.byref(v.p), C.byref(g), C.byref(o))
        Q.check(L)
        return {"mask": v["mask"]}
    if kind == "trap":
        v["phi"][...] = st["phi0"]
        v["mask_nw"][...] = st["mask_nw0"]
        L.trapComponents_mask(C.byref(v.p), C.byref(g), C.byref(o))
        Q.check(L)
        return {k: v[k] for k in ("phi", "mask_w", "mask_nw", "connectivity", "phi_bin")}
    loss = C.c_double(0)
    L.qssgpu_adjoint_theta(C.byref(o), C.byref(v.p), C.byref(g), Q.dptr(st["theta"]), Q.dptr(st["target"]),
                           st["case"]["steps"], st["dt"], st["case"]["ckpt"], C.byref(loss), Q.dptr(st["grad"]))
    Q.check(L)
    return {"loss": loss.value, "grad": st["grad"]}


# ---------------------------------------------------------------------------
# what one pass cannot do without

# FP64 operations per voxel: a WENO5 stage with every face and centre computed
# once (3 x 98 + 94), an ENO2 / ENO3 stage (derivatives, Godunov, curvature, RK),
# a reinitialisation sweep, the reverse of a WENO5 stage
STAGE = {5: 388, 2: 140, 3: 190}
SWEEP, REVERSE = 25, 650


def work(case):
    kind = case["kind"]
    if kind == "ladder":
        sides = _batch_dims(case)
    else:
        sides = [_dims(case)]
    fb = float(sum(a * b * c for a, b, c in sides))
    gb = float(sum((a + 6) * (b + 6) * (c + 6) for a, b, c in sides))
    if kind == "rhs":
        return {"bytes": 8 * (gb * 1 + 5 * fb + fb), "flops": 383 * fb}
    if kind == "maskprep":
        return {"bytes": fb + 8 * gb, "flops": 20 * SWEEP * fb}
    if kind == "trap":
        return {"bytes": gb * (3 * 8 + 3 * 8 + 5), "flops": 8 * gb}
    if kind == "adjoint":
        return {"bytes": 8 * 5 * gb, "flops": case["steps"] * 3 * fb * (STAGE[5] + REVERSE)}
    inner = math.ceil(case["tplot"] / (0.5 / 210))  # the CFL step is near 0.5 / (150 + 40 + 20)
    sweeps = 3 * 20
    per_step = fb * (inner * case["time"] * STAGE[case["order"]] + sweeps * SWEEP)
    n = case.get("steps", 1) if kind == "ladder" else 1
    arrays_in = 2 if kind == "ladder" else (9 if kind == "constcurv" else 4)
    return {"bytes": gb * 8 * (arrays_in + 5) + gb * 5, "flops": n * per_step + (20 * SWEEP * fb if kind == "ladder" else 0)}


# ---------------------------------------------------------------------------
# the same results as plain torch in 64 bits

def _t(a):
    return torch.as_tensor(np.array(a), device=_dev())


def _in(a, di=0, dj=0, dk=0):
    """The fill box of `a`, shifted."""
    nz, ny, nx = a.shape
    return a[NG + dk:nz - NG + dk, NG + dj:ny - NG + dj, NG + di:nx - NG + di]


def _weno_side(v1, v2, v3, v4, v5):
    eps = 1e-6 * torch.stack([v * v for v in (v1, v2, v3, v4, v5)]).amax(0) + 1e-35
    s1 = 13 / 12 * (v1 - 2 * v2 + v3) ** 2 + 0.25 * (v1 - 4 * v2 + 3 * v3) ** 2
    s2 = 13 / 12 * (v2 - 2 * v3 + v4) ** 2 + 0.25 * (v2 - v4) ** 2
    s3 = 13 / 12 * (v3 - 2 * v4 + v5) ** 2 + 0.25 * (3 * v3 - 4 * v4 + v5) ** 2
    a1, a2, a3 = 0.1 / (s1 + eps) ** 2, 0.6 / (s2 + eps) ** 2, 0.3 / (s3 + eps) ** 2
    p = a1 * (v1 / 3 - 7 / 6 * v2 + 11 / 6 * v3) + a2 * (-v2 / 6 + 5 / 6 * v3 + v4 / 3) + a3 * (v3 / 3 + 5 / 6 * v4 - v5 / 6)
    return p / (a1 + a2 + a3)


def _eno2(s):
    d2 = [s[k + 1] + s[k - 1] - 2 * s[k] for k in (1, 2, 3)]
    pick = lambda a, b: torch.where(a.abs() < b.abs(), a, b)  # noqa: E731
    return (s[3] - s[2] - 0.5 * pick(d2[1], d2[2])) / DX, (s[2] - s[1] + 0.5 * pick(d2[0], d2[1])) / DX


def _one_sided(phi, order):
    """(plus, minus) differences of the fill box along x, y, z."""
    out = []
    for ax in ("di", "dj", "dk"):
        r = 3 if order == 5 else 2
        s = [_in(phi, **{ax: m}) for m in range(-r, r + 1)]
        if order == 5:
            d = [(s[m + 1] - s[m]) / DX for m in range(6)]  # d[m]: face m - 2
            out.append((_weno_side(d[5], d[4], d[3], d[2], d[1]), _weno_side(d[0], d[1], d[2], d[3], d[4])))
        else:
            out.append(_eno2(s))
    return out


def _curvature(phi):
    f = 0.5 / DX
    sh = lambda i=0, j=0, k=0: _in(phi, i, j, k)  # noqa: E731
    x, y, z = (sh(1) - sh(-1)) * f, (sh(0, 1) - sh(0, -1)) * f, (sh(0, 0, 1) - sh(0, 0, -1)) * f
    c2 = 2 * sh()
    xx, yy = (sh(2) + sh(-2) - c2) * f * f, (sh(0, 2) + sh(0, -2) - c2) * f * f
    zz = (sh(0, 0, 2) + sh(0, 0, -2) - c2) * f * f
    xy = (sh(1, 1) + sh(-1, -1) - sh(-1, 1) - sh(1, -1)) * f * f
    xz = (sh(1, 0, 1) + sh(-1, 0, -1) - sh(-1, 0, 1) - sh(1, 0, -1)) * f * f
    yz = (sh(0, 1, 1) + sh(0, -1, -1) - sh(0, -1, 1) - sh(0, 1, -1)) * f * f
    g2 = x * x + y * y + z * z
    k = (xx * (y * y + z * z) + yy * (x * x + z * z) + zz * (x * x + y * y)
         - 2 * (xy * x * y + xz * x * z + yz * y * z))
    return torch.where(g2 < 1e-5, torch.zeros_like(k), k / torch.clamp(g2, min=1e-30))


def _rhs(phi, order, vel, b, adv):
    """(rhs, CFL estimate of the last voxel); vel / b tensors over the fill box or numbers."""
    pm = _one_sided(phi, order)
    zero = torch.zeros((), dtype=torch.float64, device=phi.device)
    vel_t = vel if torch.is_tensor(vel) else torch.full_like(pm[0][0], vel)
    pos = vel_t > 0
    n2 = 0
    for p, m in pm:
        up = torch.maximum(torch.maximum(m, zero) ** 2, torch.minimum(p, zero) ** 2)
        dn = torch.maximum(torch.minimum(m, zero) ** 2, torch.maximum(p, zero) ** 2)
        n2 = n2 + torch.where(pos, up, dn)
    norm = vel_t * torch.sqrt(n2)
    if order != 5:
        norm = -norm
    if torch.is_tensor(vel):  # a voxel at rest keeps the term of the last moving one before it
        ok = (vel_t.abs() >= 1e-5).reshape(-1)
        src = torch.where(ok, torch.arange(ok.numel(), device=phi.device), -1).cummax(0).values
        flat = norm.reshape(-1)
        norm = torch.where(src >= 0, flat[src.clamp(min=0)], torch.zeros_like(flat)).reshape(norm.shape)
    rhs = norm + b * _curvature(phi)
    if adv is not None:
        rhs = rhs - sum(u * torch.where(u >= 0, m, p) for u, (p, m) in zip(adv, pm))
    c = [max(float(p[-1, -1, -1].abs()), float(m[-1, -1, -1].abs())) for p, m in pm]
    h = abs(float(vel_t[-1, -1, -1])) / math.sqrt(sum(x * x for x in c) + DX * DX) * sum(c) / DX
    return rhs, h


def _ghost(a):
    """Signed linear extrapolation of the faces, x then y then z."""
    for d in (2, 1, 0):
        n = a.shape[d]
        for f, g, lay in ((NG, NG + 1, range(0, NG)), (n - NG - 1, n - NG - 2, range(n - NG, n))):
            vf, vg = a.select(d, f), a.select(d, g)
            sign = torch.copysign(torch.ones_like(vf), vf)
            for q in lay:
                a.select(d, q).copy_(vf + sign * (vf - vg).abs() * abs(f - q))
    return a


def _with_fill(a, fb):
    r = a.clone()
    _in(r).copy_(fb)
    return _ghost(r)


def _reinit(phi0, sweeps=20):
    nb = [_in(phi0, *o) for o in ((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1))]
    c0 = _in(phi0)
    near = torch.zeros_like(c0, dtype=torch.bool)
    for n in nb:
        near |= ((n > 0) & (c0 <= 0)) | ((n <= 0) & (c0 > 0))
    delta = torch.full_like(c0, 1e-5)
    for p, m in zip(nb[0::2], nb[1::2]):
        delta = torch.maximum(delta, torch.maximum((p - m).abs() / 2, torch.maximum((p - c0).abs(), (c0 - m).abs())))
    dist = c0 / delta
    sgn = torch.where(c0.abs() > 1e-5, torch.copysign(torch.ones_like(c0), c0), torch.zeros_like(c0))
    phi = phi0
    for _ in range(sweeps):
        c = _in(phi)
        pos = c > 0
        n2 = 0
        for o in ((1, 0, 0), (0, 1, 0), (0, 0, 1)):
            gp, gm = (_in(phi, *o) - c) / DX, (c - _in(phi, *[-q for q in o])) / DX
            n2 = n2 + torch.where(pos, torch.maximum(-gp, gm), torch.maximum(gp, -gm)).clamp(min=0) ** 2
        far = torch.where(c.abs() > 1e-5, sgn - sgn * torch.sqrt(n2), torch.zeros_like(c))
        phi = _with_fill(phi, c + 0.5 * DX * torch.where(near, dist - sgn * c.abs() / DX, far))
    return phi


def _reached(b, at):
    """Voxels of the binary image in the 26-connected component of flat index `at`."""
    b = b.to(torch.float32)[None, None]
    seen = torch.zeros_like(b)
    seen.view(-1)[at] = b.view(-1)[at]
    while True:
        before = seen
        for _ in range(16):
            seen = torch.nn.functional.max_pool3d(seen, 3, 1, 1) * b
        if torch.equal(before, seen):
            return seen[0, 0] > 0


def _trap(phi, mask, mask_nw, o):
    phi = torch.where(mask_nw > 0, -mask_nw, phi)
    b = phi < 0
    b[NG:-NG, NG:-NG, NG - 1] = True
    off = b & ~_reached(b, o.phi_nw_ind)
    fill = torch.full_like(phi, -20 * DX)
    nw = torch.where(off & (phi < 0), -phi, fill)
    s = torch.maximum(nw, torch.maximum(mask, -phi))
    b = s < 0
    b[NG:-NG, NG:-NG, -NG] = True
    off = b & ~_reached(b, o.phi_w_ind)
    return phi, nw, torch.where(off & (s < 0), -s, fill)


def _model(s, var):
    """One curvature step (a single outer iteration, as tmax = tplot)."""
    v, o = s.v, s.o
    phi, mask, mw, mnw = (_t(a) for a in (s.phi0, v["mask"], v["mask_w"], v["mask_nw"]))
    order = o.order_space_accur
    if var:
        vel, b = _t(v.fb("normal_velocity")), _t(v.fb("curvature_coeff"))
        adv = [_t(v.fb("external_velocity_" + d)) for d in "xyz"]
    else:
        vel, b, adv = o.a, o.b, None
    impose = lambda a: torch.maximum(torch.maximum(torch.maximum(a, mask - o.overlap), mw), mnw)  # noqa: E731
    prev, t, nxt = phi, 0.0, phi
    while t < o.tplot:
        r, h = _rhs(phi, order, vel, b, adv)
        dt = 0.5 / (max(h, -1.0) + o.b_max_over_dx + o.max_U_over_dx)
        t += dt
        s1 = _with_fill(phi, _in(phi) + dt * r)
        r, _ = _rhs(s1, order, vel, b, adv)
        nxt = _with_fill(phi, 0.75 * _in(phi) + 0.25 * (_in(s1) + dt * r))
        if o.order_time_accur == 3:
            r, _ = _rhs(nxt, order, vel, b, adv)
            nxt = _with_fill(phi, _in(phi) / 3 + 2 / 3 * (_in(nxt) + dt * r))
        phi = impose(nxt)
    if var:
        phi = torch.maximum(mask, phi)
    phi, mnw, mw = _trap(phi, mask, mnw, o)
    mw, mnw = _reinit(mw), _reinit(mnw)
    phi = _reinit(torch.where(mnw > 0, -mnw, phi))
    return {"t": t, "phi": phi, "phi_prev": prev, "phi_next": nxt, "mask_w": mw, "mask_nw": mnw,
            "connectivity": None, "phi_bin": None}


def _np(d):
    return {k: a.cpu().numpy() if torch.is_tensor(a) else a for k, a in d.items()}


def exact(case, seed):
    kind = case["kind"]
    # a ladder is a chain of the curvature steps above; the adjoint's gradient
    # through 64-bit autograd of every stage takes far longer than the call; the
    # ENO3 stencil of the reference mixes its axes, which the others do not show
    if kind in ("ladder", "adjoint") or case.get("order") == 3:
        return None
    st = prepare(case, seed)
    s = st["s"]
    if kind in ("constcurv", "novar"):
        return _np(_model(s, kind == "constcurv"))
    v = s.v
    if kind == "rhs":
        r, h = _rhs(_t(v["phi"]), 5, _t(v.fb("normal_velocity")), _t(v.fb("curvature_coeff")),
                    [_t(v.fb("external_velocity_" + d)) for d in "xyz"])
        full = torch.zeros_like(_t(v["phi"]))
        _in(full).copy_(r)
        return _np({"rhs": full, "h": h})
    if kind == "maskprep":
        m = torch.zeros(v.shape, dtype=torch.float64, device=_dev())
        _in(m).copy_(torch.where(_t(st["ubc"]) == 255, DX, -DX))
        return _np({"mask": _reinit(m)})
    phi, nw, w = _trap(_t(st["phi0"]), _t(v["mask"]), _t(st["mask_nw0"]), s.o)
    return _np({"phi": phi, "mask_w": w, "mask_nw": nw, "connectivity": None, "phi_bin": None})
