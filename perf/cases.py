"""Performance cases of the boundary-integral path: what a user of this package has it compute.

Each case is one call (or the few calls that belong together) through the package's public entry
points, on seeded problems of the kinds the package is used for: cube-spheres and two-layer
cube-spheres of bilinear quads, and triangulated cones, on square, rectangular and hexagonal
lattices, periods 0.8 - 1.5 um, wavelengths 0.4 - 0.8 um.  Everything is FP64.

  listed()            the fixed cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) the problem on the device, as a program holds it before the call
  run(state)          one pass; returns every output of the call
  work(case)          bytes and operations that the results cannot do without
  exact(case, seed)   the same results from plain torch in 64 bits (Green's function, fields at
                      points, and the open region's matrices of small quad meshes)
"""
import math
import random

import numpy as np
import torch

import bem3_emf_qd2_b200 as B
from bem3_emf_qd2_b200 import batch, meshgen
from bem3_emf_qd2_b200.dqd2 import PlaneWave, Problem

SQUARE = dict(d1x=1.0, d1y=0.0, d2x=0.0, d2y=1.0)
HEX = dict(d1x=0.9, d1y=0.0, d2x=0.45, d2y=0.7794)


def listed():
    return [
        # A user evaluating the quasi-periodic Green's function itself (checks, other quadratures).
        dict(name="qpgf_4k", kind="qpgf", n=4096, mode=0, lam=0.6328, ni=1.33, **SQUARE),
        # The open region's coefficient matrices, the dominant part of every solve: a coarse mesh (a
        # parameter sweep's or a test's), the usual single sphere, and the outer surface of a two-layer
        # sphere with 6 x 12 x 12 quads (the largest here; larger meshes are the same kernels for longer).
        dict(name="open_quads_96", kind="open", shape="sphere", n=4, r=0.3, lam=0.6328, ni=1.33, **SQUARE),
        dict(name="open_quads_384", kind="open", shape="sphere", n=8, r=0.3, lam=0.6328, ni=1.33, **SQUARE),
        dict(name="open_quads_864", kind="open", shape="sphere", n=12, r=0.35, lam=0.532, ni=1.33, **SQUARE),
        # The same for a triangulated cone on a hexagonal lattice: three times the points per pair, many
        # real-space terms, and a flat base whose pairs lie in one plane.
        dict(name="open_triangles_352", kind="open", shape="cone", n=4, r=0.3, lam=0.7, ni=1.0, **HEX),
        # An interior domain with a complex wave number and the tangential derivatives: the shell of the
        # two-layer sphere sees both surfaces.
        dict(name="shell_quads_1728", kind="shell", shape="twolayer", n=12, r=0.35, lam=0.532, ni=1.33, **SQUARE),
        # Every domain through host pointers, the matrices copied back to the caller's page-locked arrays:
        # the reference program's call.
        dict(name="domains_host_216", kind="domains", shape="sphere", n=6, r=0.3, lam=0.6328, ni=1.33, **SQUARE),
        # An admission wave of the service: several small problems assembled as one batch.
        dict(name="batch_4x", kind="batch", shape="twolayer", n=4, count=4, r=0.3, lam=0.55, ni=1.33,
             d1x=1.0, d1y=0.0, d2x=0.0, d2y=1.2),
        # Field of a solved problem at one point (the interactive use; all latency) and on a probe grid.
        dict(name="field_1pt", kind="field", shape="sphere", n=8, npts=1, type=0, r=0.3, lam=0.6328, ni=1.33, **SQUARE),
        dict(name="field_441pts", kind="field", shape="sphere", n=8, npts=441, type=1, r=0.3, lam=0.6328, ni=1.33,
             **SQUARE),
        # Fields from the derivatives of the potentials (needs the Green's function's second derivatives).
        dict(name="memp_121pts", kind="memp", shape="sphere", n=8, npts=121, type=0, r=0.3, lam=0.6328, ni=1.33,
             **SQUARE),
        # A whole small solve, from the resident problem to the boundary values on the host.
        dict(name="solve_96", kind="solve", shape="sphere", n=4, r=0.3, lam=0.6328, ni=1.33, **SQUARE),
    ]


# ---------------------------------------------------------------------------------------------
# sizes
def _cone_counts(n):
    """rings, rows and sectors of a cone of refinement n (n = 12 is 12, 24 and 48)."""
    return n, 2 * n, 4 * n


def _elements(shape, n):
    if shape == "sphere":
        return 6 * n * n
    if shape == "twolayer":
        return 12 * n * n
    rings, rows, sect = _cone_counts(n)
    return sect * (1 + 2 * (rings - 1)) + sect * (1 + 2 * (rows - 1))


def _points_per_pair(shape):
    return 432 if shape == "cone" else 144


def _cell_load(c):
    """k^2 x cell area: how many lattice terms a point needs, up to a constant."""
    k = 2.0 * math.pi * c["ni"] / c["lam"]
    return k * k * abs(c["d1x"] * c["d2y"] - c["d1y"] * c["d2x"])


def _open_load(c):
    ne = _elements(c["shape"], c["n"])
    if c["shape"] == "twolayer":
        ne //= 2
    return 4.0 * ne * ne * _points_per_pair(c["shape"]) * (60.0 + 0.6 * _cell_load(c)) * c.get("count", 1)


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    top = _open_load(listed()[3])
    while True:
        kind = rng.choice(["qpgf", "open", "open", "open", "shell", "domains", "batch", "field", "memp", "solve"])
        c = dict(kind=kind, lam=round(rng.uniform(0.4, 0.8), 4))
        shape = rng.choice(["sphere", "sphere", "twolayer", "cone"])
        c["ni"] = 1.0 if shape == "cone" else 1.33
        p1, p2 = round(rng.uniform(0.8, 1.5), 4), round(rng.uniform(0.8, 1.5), 4)
        if shape == "cone" and rng.random() < 0.7:  # hexagonal
            c.update(d1x=p1, d1y=0.0, d2x=0.5 * p1, d2y=round(0.866 * p1, 4))
        else:
            c.update(d1x=p1, d1y=0.0, d2x=0.0, d2y=p2)
        if kind == "qpgf":
            c.update(n=_logint(rng, 1, 16384), mode=rng.randrange(2))
            return c
        c["r"] = round(0.3 * min(p1, p2), 4)
        if kind == "shell":
            shape, n = "twolayer", _logint(rng, 2, 12)
        elif kind == "batch":
            shape, n = rng.choice(["sphere", "twolayer"]), rng.randrange(2, 6)
            c["count"] = rng.randrange(2, 6)
        elif kind == "solve":
            shape, n = "sphere", rng.randrange(2, 6)
        elif kind in ("field", "memp"):
            shape, n = "sphere", rng.randrange(3, 11)
            c.update(npts=_logint(rng, 1, 600 if kind == "field" else 160), type=rng.randrange(2))
        elif shape == "cone":
            n = rng.randrange(2, 6)
        elif kind == "domains":
            n = rng.randrange(2, 8) if shape == "sphere" else rng.randrange(2, 6)
        else:
            shape, n = "sphere", rng.randrange(2, 13)
        c.update(shape=shape, n=n)
        if kind in ("field", "memp", "shell") or _open_load(c) <= top:
            return c


# ---------------------------------------------------------------------------------------------
# problems
def _problem(c, seed):
    """A seeded problem of the case's kind: the incidence, the wavelength (within 1 %), the size
    (within 1 %), the media and the polarisation come from the seed."""
    rng = random.Random("%s/%d" % (c["kind"], seed))
    nodes = meshgen._Nodes()
    r = c["r"] * rng.uniform(0.99, 1.01)
    n = c["n"]
    inner = complex(rng.uniform(1.4, 2.2), rng.uniform(0.0, 0.1) if c["shape"] == "cone" else 0.0)
    if c["shape"] == "sphere":
        surf, media = [(meshgen.cube_sphere(nodes, r, n), 1, 0)], [inner]
    elif c["shape"] == "twolayer":
        surf = [(meshgen.cube_sphere(nodes, r, n), 1, 0), (meshgen.cube_sphere(nodes, 0.7 * r, n), 2, 1)]
        media = [complex(1.45, 0.01), inner]
    else:
        rings, rows, sect = _cone_counts(n)
        surf = [(meshgen.cone(nodes, r, 2.0 * r, -r, rings, rows, sect, 0.01, rng.randrange(1 << 30)), 1, 0)]
        media = [inner]
    rn = np.zeros((len(nodes.pts) + 1, 3))
    rn[1:] = np.array(nodes.pts)
    ed, md, sd = [[0, 0, 0, 0]], [0], [0]
    for els, a, b in surf:  # elements given with normals leaving domain a, towards domain b
        for e in els:
            if b == 0:  # the open region is the main domain: reversed order
                e = [e[0], e[3], e[2], e[1]] if len(e) == 4 else [e[0], e[2], e[1]]
                md.append(0)
                sd.append(a)
            else:
                md.append(a)
                sd.append(b)
            ed.append(list(e) + [0] * (4 - len(e)))
    ed = np.array(ed, np.int32)
    lam = c["lam"] * rng.uniform(0.99, 1.01)
    pol = rng.uniform(0.0, math.pi)
    w = PlaneWave(lam, c["ni"], c["ni"] / 2.0, complex(math.cos(pol)), complex(math.sin(pol)), (0.0, 0.0, 0.0),
                  rng.uniform(0.05, math.radians(60.0)), rng.uniform(0.0, 2.0 * math.pi))
    z = np.zeros(len(md), np.int32)
    return Problem([w], 1, (c["d1x"], c["d1y"]), (c["d2x"], c["d2y"]), media, rn, ed, np.array(md, np.int32),
                   np.array(sd, np.int32), z)


def _points(c, p, seed):
    """Field points: a plane through the cell at a seeded height and azimuth, kept 12 % of the radius
    away from the sphere's surface."""
    rng = np.random.default_rng(seed)
    m = c["npts"]
    side = int(math.ceil(math.sqrt(m)))
    g = (np.arange(side) + rng.uniform(0.2, 0.8)) / side - 0.5
    u, v = np.meshgrid(g, g, indexing="ij")
    u, v = u.ravel()[:m], v.ravel()[:m]
    if m == 1:  # a probe in the open region
        u, v = rng.uniform(0.35, 0.5, (2, 1))
    a = rng.uniform(0.0, math.pi)
    s = 1.5 * c["r"] * 2.0
    r = np.stack([s * u * math.cos(a), s * u * math.sin(a), s * v], -1) + rng.uniform(-0.02, 0.02, 3)
    d = np.linalg.norm(r, axis=1)
    rad = c["r"]
    near = np.abs(d - rad) < 0.12 * rad
    r[near] *= (np.where(d < rad, 0.85, 1.15) * rad / np.maximum(d, 1e-3))[near, None]
    return np.ascontiguousarray(r)


def _boundary_values(p, seed):
    """Boundary values of the size and smoothness a solve gives: on each domain, plane waves of its
    wave number with seeded amplitudes and directions, and their normal derivatives."""
    rng = np.random.default_rng(seed + 77)
    out = []
    for d in range(p.MN + 1):
        s = np.abs(p.sid[d])
        k = complex(p.kn[d])
        x = p.ren[s]
        nrm = p.wen[s] / np.linalg.norm(p.wen[s], axis=-1, keepdims=True)
        bv = {}
        for key, dkey, m in (("U", "dU", 4), ("E", "dE", 3), ("H", "dH", 3)):
            f = np.zeros((len(s) + 1, 4, m), np.complex128)
            df = np.zeros_like(f)
            for i in range(m):
                q = rng.normal(size=3)
                q /= np.linalg.norm(q)
                amp = rng.normal() + 1j * rng.normal()
                ph = amp * np.exp(1j * k * (x @ q))
                f[1:, :, i] = ph
                df[1:, :, i] = 1j * k * (nrm @ q) * ph
            bv[key], bv[dkey] = f, df
        out.append(bv)
    return out


def _qpgf_inputs(c, seed):
    rng = np.random.default_rng(seed)
    k = 2.0 * math.pi * c["ni"] / c["lam"]
    th, ph = rng.uniform(0.05, math.radians(60.0)), rng.uniform(0.0, 2.0 * math.pi)
    qd = dict(k=k, vk=[k * math.sin(th) * math.cos(ph), k * math.sin(th) * math.sin(ph), k * math.cos(th)],
              vd1=[c["d1x"], c["d1y"]], vd2=[c["d2x"], c["d2y"]])
    uv = rng.uniform(-1.5, 1.5, (c["n"], 2))
    r = np.empty((c["n"], 3))
    r[:, 0] = uv[:, 0] * c["d1x"] + uv[:, 1] * c["d2x"]
    r[:, 1] = uv[:, 0] * c["d1y"] + uv[:, 1] * c["d2y"]
    r[:, 2] = rng.uniform(-0.8, 0.8, c["n"])
    return qd, r


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "qpgf":
        qd, r = _qpgf_inputs(c, seed)
        return dict(c=c, qd=qd, r=r)
    if kind == "batch":
        insts = [batch.InstanceDevice(_problem(c, 1000 * seed + j)) for j in range(c["count"])]
        return dict(c=c, insts=insts)
    p = _problem(c, seed)
    if kind in ("open", "shell"):
        return dict(c=c, p=p, dev=B.DeviceProblem(p))
    if kind == "domains":
        return dict(c=c, p=p, out={d: B.domain_outputs(p, d, pinned=True) for d in range(p.MN + 1)})
    ctx = B.Context(p)
    if kind in ("field", "memp"):
        ctx.set_boundary_values(_boundary_values(p, seed))
        return dict(c=c, p=p, ctx=ctx, r=_points(c, p, seed))
    return dict(c=c, p=p, ctx=ctx)


def run(state):
    c = state["c"]
    kind = c["kind"]
    if kind == "qpgf":
        out, ret = B.qpgf(state["qd"], state["r"], c["mode"])
        return dict(out=out, ret=ret)
    if kind in ("open", "shell"):
        dev, did = state["dev"], 0 if kind == "open" else 1
        dev.assemble(did)
        n = 4 * len(state["p"].sid[did])

        def m(t, rows, cols):
            return t.reshape(-1)[: rows * cols].view(rows, cols)

        return dict(G=m(dev.G, n, n), H=m(dev.H, n, n), dG=m(dev.dG, 2 * n, n), dH=m(dev.dH, 2 * n, n),
                    dF=m(dev.dF, n, 3))
    if kind == "domains":
        res = B.assemble_domains(state["p"], out=state["out"])
        return {"d%d" % d: v for d, v in res.items()}
    if kind == "batch":
        batch.assemble_entries([e for i in state["insts"] for e in i.domain_entries()])
        # every matrix of every domain; instance by instance, flattened together by kind
        return [{k: torch.cat([o[k].reshape(-1) for o in i.out]) for k in ("G", "H", "dG", "dH", "dF")}
                for i in state["insts"]]
    ctx = state["ctx"]
    if kind == "field":
        E, H, did = ctx.field(state["r"], c["type"], True)
        return dict(E=E, H=H, did=did)
    if kind == "memp":
        E, H, did = ctx.field_memp(state["r"], c["type"], True)
        return dict(E=E, H=H, did=did)
    ctx.solve()
    return [d for d in ctx.boundary_values()]


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
def _domain_sizes(c):
    ne = _elements(c["shape"], c["n"])
    if c["shape"] == "twolayer":
        return [ne // 2, ne, ne // 2]
    return [ne, ne]


def _matrix_bytes(ne):
    n = 4 * ne
    return 96.0 * n * n + 24.0 * n + 384.0 * ne


# operations of one quadrature point: the point's geometry, one closed-form evaluation of the Green's
# function and its gradient, and the sums
POINT_FLOPS = 150.0


def _matrix_flops(c, ne):
    return 4.0 * ne * ne * _points_per_pair(c["shape"]) * POINT_FLOPS


def work(case):
    c, kind = case, case["kind"]
    if kind == "qpgf":
        return dict(bytes=92.0 * c["n"], flops=POINT_FLOPS * c["n"])
    sizes = _domain_sizes(c)
    if kind == "open":
        return dict(bytes=_matrix_bytes(sizes[0]), flops=_matrix_flops(c, sizes[0]))
    if kind == "shell":
        return dict(bytes=_matrix_bytes(sizes[1]), flops=_matrix_flops(c, sizes[1]))
    if kind in ("domains", "batch"):
        m = c.get("count", 1)
        return dict(bytes=m * sum(_matrix_bytes(s) for s in sizes), flops=m * sum(_matrix_flops(c, s) for s in sizes))
    if kind in ("field", "memp"):
        ne = sizes[0]
        per = 4 if c["type"] == 0 else 9
        return dict(bytes=ne * (384.0 + 4 * 12 * 16) + 220.0 * c["npts"], flops=c["npts"] * ne * per * POINT_FLOPS)
    nn = 4 * sizes[0]
    lu = 8.0 / 3.0 * ((4.0 * nn) ** 3 + 2.0 * nn ** 3) + 8.0 * nn ** 3
    return dict(bytes=sum(_matrix_bytes(s) for s in sizes) + 16.0 * (4.0 * nn) ** 2,
                flops=lu + sum(_matrix_flops(c, s) for s in sizes))


# ---------------------------------------------------------------------------------------------
# plain 64-bit results: the Green's function by Ewald's method with one split parameter and fixed sets
# of terms (every term above 1e-19), and the quadrature rules point by point
H_STEP = 0.42


def _w(z):
    """Faddeeva function for Im z >= 0: trapezoidal rule with the pole's correction."""
    u = z.real.abs() / H_STEP
    fr = u - torch.floor(u)
    full = torch.minimum(fr, 1.0 - fr) >= (fr - 0.5).abs()
    one = full.to(torch.float64)
    s = torch.zeros_like(z)
    z2 = z * z
    for n in range(18, -1, -1):
        tf, th = n * H_STEP, (n + 0.5) * H_STEP
        t = one * tf + (1.0 - one) * th
        cf, ch = math.exp(-tf * tf) * (0.5 if n == 0 else 1.0), math.exp(-th * th)
        s = s + (one * cf + (1.0 - one) * ch) / (z2 - t * t)
    w = (1j * H_STEP / math.pi) * 2.0 * z * s
    y = z.imag
    zz = torch.complex(z.real, torch.clamp(y, max=math.pi / H_STEP))
    e = torch.exp(-2j * math.pi * zz / H_STEP)
    pole = 2.0 * torch.exp(-zz * zz) / torch.where(full, 1.0 - e, 1.0 + e)
    return w + torch.where(y < math.pi / H_STEP, pole, torch.zeros_like(pole))


def _qpgf64(qd, r):
    """G and grad G [n, 4] (complex) at r [n, 3]."""
    k, (kx, ky) = qd["k"], qd["vk"][:2]
    d1, d2 = np.array(qd["vd1"], float), np.array(qd["vd2"], float)
    det = d1[0] * d2[1] - d2[0] * d1[1]
    x, y, z = r[:, 0], r[:, 1], r[:, 2]
    l1 = torch.floor((x * d2[1] - y * d2[0]) / det + 0.5)
    l2 = torch.floor(-(x * d1[1] - y * d1[0]) / det + 0.5)
    x, y = x - l1 * d1[0] - l2 * d2[0], y - l1 * d1[1] - l2 * d2[1]
    phase = torch.exp(-1j * (kx * (l1 * d1[0] + l2 * d2[0]) + ky * (l1 * d1[1] + l2 * d2[1])))
    ve = min(math.sqrt(abs(det) / (4.0 * math.pi) * np.linalg.norm(d1 + d2) / np.linalg.norm(d1 - d2)), math.sqrt(3.0) / k)
    ke = k * ve
    out = torch.zeros((len(x), 4), dtype=torch.complex128, device=r.device)
    # real space
    reach = 2.0 * ve * math.sqrt(45.0 + ke * ke) + 0.5 * (np.linalg.norm(d1) + np.linalg.norm(d2))
    m1 = int(reach * np.linalg.norm(d2) / abs(det)) + 2
    m2 = int(reach * np.linalg.norm(d1) / abs(det)) + 2
    for a in range(-m1, m1 + 1):
        for b in range(-m2, m2 + 1):
            R0 = a * d1 + b * d2
            if np.linalg.norm(R0) > reach:
                continue
            px, py = x + R0[0], y + R0[1]
            R = torch.sqrt(px * px + py * py + z * z)
            q = R / (2.0 * ve)
            ef = torch.exp(ke * ke - q * q)
            w = _w(torch.complex(torch.full_like(q, ke), q))
            cb = complex(math.cos(kx * R0[0] + ky * R0[1]), math.sin(kx * R0[0] + ky * R0[1])) / (4.0 * math.pi)
            out[:, 0] += cb * (ef * w.real / R)
            cf = -cb * (ef * (w.real / R - k * w.imag + 1.0 / (ve * math.sqrt(math.pi))) / (R * R))
            out[:, 1] += cf * px
            out[:, 2] += cf * py
            out[:, 3] += cf * z
    # spectral
    g1 = 2.0 * math.pi / det * np.array([d2[1], -d2[0]])
    g2 = 2.0 * math.pi / det * np.array([-d1[1], d1[0]])
    amax = math.sqrt(45.0 / (ve * ve) + k * k) + math.hypot(kx, ky)
    m1, m2 = int(amax * np.linalg.norm(d1) / (2 * math.pi)) + 2, int(amax * np.linalg.norm(d2) / (2 * math.pi)) + 2
    az = z.abs()
    sz = torch.where(z < 0, -1.0, 1.0).to(torch.float64)
    q = az / (2.0 * ve)
    area = abs(det)
    for a in range(-m1, m1 + 1):
        for b in range(-m2, m2 + 1):
            ax, ay = -kx + a * g1[0] + b * g2[0], -ky + a * g1[1] + b * g2[1]
            b2 = k * k - ax * ax - ay * ay
            if -b2 * ve * ve > 45.0:
                continue
            ce = torch.exp(1j * (ax * x + ay * y))
            bn = math.sqrt(abs(b2))
            ef = torch.exp(b2 * ve * ve - q * q)
            if b2 > 0:
                w = _w(torch.complex(torch.full_like(q, bn * ve), q))
                ff = torch.exp(1j * bn * az)
                F = ce * (2.0 / bn) * torch.complex(ff.real, ef * w.imag + ff.imag)
                dz = 2.0 * ce * torch.complex(ef * w.real - ff.real, -ff.imag) * sz
            else:
                u = bn * ve
                f1 = ef * torch.special.erfcx(u + q)
                f2 = torch.where(q <= u, ef * torch.special.erfcx((u - q).clamp(min=0.0)),
                                 2.0 * torch.exp(-bn * az) - ef * torch.special.erfcx((q - u).clamp(min=0.0)))
                F = -1j * ce * (f1 + f2) / bn
                dz = ce * (f1 - f2) * sz
            out[:, 0] += 0.25j / area * F
            out[:, 1] -= 0.25 / area * ax * F
            out[:, 2] -= 0.25 / area * ay * F
            out[:, 3] += 0.25 / area * dz
    return out * phase[:, None]


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _exact_qpgf(c, seed):
    qd, r = _qpgf_inputs(c, seed)
    return dict(out=_qpgf64(qd, _t(r)).cpu().numpy(), ret=None)


def _bilinear(cr, cw, zeta, eta):
    """positions and normals [..., 3] of elements cr [..., 3, 4], cw [..., 3, 3] at zeta, eta."""
    zeta, eta = zeta[..., None], eta[..., None]
    r = cr[..., 0] + cr[..., 1] * zeta + cr[..., 2] * eta + cr[..., 3] * zeta * eta
    return r, cw[..., 0] + cw[..., 1] * zeta + cw[..., 2] * eta


def _shape(zeta, eta):
    a = math.sqrt(3.0)
    return torch.stack([0.25 * (1 - zeta * a) * (1 - eta * a), 0.25 * (1 + zeta * a) * (1 - eta * a),
                        0.25 * (1 + zeta * a) * (1 + eta * a), 0.25 * (1 - zeta * a) * (1 + eta * a)], -1)


def _exact_field(c, seed):
    p = _problem(c, seed)
    bv, pts = _boundary_values(p, seed), _points(c, p, seed)
    E, H = np.zeros((len(pts), 3), complex), np.zeros((len(pts), 3), complex)
    inside = np.linalg.norm(pts, axis=1) < c["r"]
    for d in range(2):
        at = np.nonzero(inside == (d == 1))[0]
        if not len(at):
            continue
        s, sg = np.abs(p.sid[d]), np.sign(p.sid[d])
        cr, cw = _t(p.cr[s]), _t(p.cw[s])
        if c["type"] == 0:
            nodes = [(z / math.sqrt(3.0), e / math.sqrt(3.0), 1.0) for z, e in ((-1, -1), (1, -1), (1, 1), (-1, 1))]
        else:
            g = math.sqrt(0.6)
            nodes = [(g * i, g * j, (5 + 3 * (i == 0)) * (5 + 3 * (j == 0)) / 81.0) for i in (-1, 0, 1) for j in (-1, 0, 1)]
        ne = len(s)
        rt = _t(pts[at])
        acc = torch.zeros((len(at), 6), dtype=torch.complex128, device="cuda")
        F = torch.zeros(len(at), dtype=torch.float64, device="cuda")
        vals = [_t(bv[d][k][1:]) for k in ("E", "dE", "H", "dH")]
        sgn = _t(sg.astype(float))
        if d == 0:  # the cell of each point
            D = np.array([[c["d1x"], c["d2x"]], [c["d1y"], c["d2y"]]])
            cell = np.floor(np.linalg.solve(D, pts[at][:, :2].T) + 0.5)
            off = (D @ cell).T
            rt[:, :2] -= _t(off)
        for z, e, wq in nodes:
            zz = torch.full((ne,), z, dtype=torch.float64, device="cuda")
            ee = torch.full((ne,), e, dtype=torch.float64, device="cuda")
            rq, W = _bilinear(cr, cw, zz, ee)
            N = _shape(zz, ee)
            aW = W.norm(dim=-1)
            v = rq[None] - rt[:, None]
            R = v.norm(dim=-1)
            RW = (v * W[None]).sum(-1)
            if d == 0:
                g = _qpgf64(p.qpd, v.reshape(-1, 3)).reshape(len(at), ne, 4)
                G, Hn = g[..., 0], (g[..., 1:] * W[None]).sum(-1)
            else:
                ik = 1j * complex(p.kn[d])
                G = torch.exp(ik * R) / (4 * math.pi * R)
                Hn = (ik * R - 1.0) * G * RW / (R * R)
            F += (wq * sgn * RW / (4 * math.pi * R ** 3)).sum(-1)
            cg, ch = wq * aW * G, wq * sgn * Hn
            f = [(N[..., None].to(torch.complex128) * x).sum(1) for x in vals]
            acc[:, :3] += cg @ f[1] - ch @ f[0]
            acc[:, 3:] += cg @ f[3] - ch @ f[2]
        a = (acc / ((1.0 + F) if d == 0 else F)[:, None]).cpu().numpy()
        if d == 0:
            kv = np.array(p.qpd["vk"][:2])
            a = a * np.exp(1j * (off @ kv))[:, None]
            w = p.waves[0]
            k3 = w.ki * np.array([w.sin_t * w.cos_p, w.sin_t * w.sin_p, w.cos_t])
            inc = np.exp(1j * (pts[at] @ k3))[:, None] * w.E0
            a[:, :3] += inc * np.array([w.ex, w.ey, w.ez])
            a[:, 3:] += inc * np.array([w.hx, w.hy, w.hz])
        E[at], H[at] = a[:, :3], a[:, 3:]
    return dict(E=E, H=H, did=None)


def _legendre(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return x, w


def _exact_open(c, seed):
    p = _problem(c, seed)
    ne = p.Ne
    dev = "cuda"
    cr, cw = _t(p.cr[1:]), _t(p.cw[1:])
    g3 = 1.0 / math.sqrt(3.0)
    zt = torch.tensor([-g3, g3, g3, -g3], dtype=torch.float64, device=dev)
    et = torch.tensor([-g3, -g3, g3, g3], dtype=torch.float64, device=dev)
    rt = _t(p.ren[1:])  # [ne, 4, 3]
    Tz = cr[:, None, :, 1] + cr[:, None, :, 3] * et[None, :, None]
    Te = cr[:, None, :, 2] + cr[:, None, :, 3] * zt[None, :, None]
    tz, te = Tz / Tz.norm(dim=-1, keepdim=True), Te / Te.norm(dim=-1, keepdim=True)
    N = 4 * ne
    G = torch.zeros((N, ne, 4), dtype=torch.complex128, device=dev)
    H = torch.zeros_like(G)
    F = torch.zeros((N, ne, 3), dtype=torch.float64, device=dev)

    def rule(rows, cols, n):
        """G, H [m, 4] and F, dF [m, 3] of the pairs (rows, cols) by the n x n rule"""
        x, w = _legendre(n)
        xx, ww = torch.tensor(x, device=dev), torch.tensor(w, device=dev)
        zeta, eta = xx.repeat_interleave(n), xx.repeat(n)
        wq = ww.repeat_interleave(n) * ww.repeat(n)
        rq, W = _bilinear(cr[cols][:, None], cw[cols][:, None], zeta[None], eta[None])  # [m, q, 3]
        Nq = _shape(zeta, eta) * wq[:, None]
        t, tn = rows // 4, rows % 4
        v = rq - rt[t, tn][:, None]
        R = v.norm(dim=-1)
        q = _qpgf64(p.qpd, v.reshape(-1, 3)).reshape(*R.shape, 4)
        Hn = (q[..., 1:] * W).sum(-1)
        u = v / R[..., None]
        RW = (u * W).sum(-1)
        f = [(wq * RW / R ** 2).sum(-1)]
        for tv in (tz, te):
            d = tv[t, tn][:, None]
            f.append((wq / R ** 3 * (3.0 * (u * d).sum(-1) * RW - (W * d).sum(-1))).sum(-1))
        Nc = Nq.to(torch.complex128)
        return (q[..., 0] * W.norm(dim=-1)) @ Nc, Hn @ Nc, torch.stack(f, -1) / (4 * math.pi)

    rows = torch.arange(N, device=dev).repeat_interleave(ne)
    cols = torch.arange(ne, device=dev).repeat(N)
    keep = rows // 4 != cols
    rows, cols = rows[keep], cols[keep]
    for i in range(0, len(rows), 1 << 14):
        a, b = rows[i:i + (1 << 14)], cols[i:i + (1 << 14)]
        G[a, b], H[a, b], F[a, b] = rule(a, b, 12)
    near = (F[rows, cols, 1].abs() > 0.5) | (F[rows, cols, 2].abs() > 0.5)
    rows, cols = rows[near], cols[near]
    for i in range(0, len(rows), 512):
        a, b = rows[i:i + 512], cols[i:i + 512]
        G[a, b], H[a, b], F[a, b] = rule(a, b, 64)
    # the elements' own integrals: polar coordinates around the node
    xl, wl = (torch.tensor(v, device=dev) for v in _legendre(12))
    xh, wh = (torch.tensor(v, device=dev) for v in _legendre(64))
    bdc = (cr[..., 1] * cw[..., 2]).sum(-1)  # [ne]
    corners = ((-1, -1), (1, -1), (1, 1), (-1, 1))

    def polar(z0, e0):
        """theta, theta weights and the distance to the far edge, [512] each, around (z0, e0)"""
        th, wt, rm = [], [], []
        dz, de = [a - z0 for a, _ in corners], [b - e0 for _, b in corners]
        ang = [math.atan2(e, z) for z, e in zip(dz, de)]
        for j in range(4):
            t0, t1 = ang[j], ang[(j + 1) % 4] + (2 * math.pi if j == 3 else 0.0)
            r0, r1 = math.hypot(dz[j], de[j]), math.hypot(dz[(j + 1) % 4], de[(j + 1) % 4])
            for half in (0, 1):
                t = 0.25 * (t1 - t0) * xh + 0.25 * ((t1 + 3 * t0) if half == 0 else (3 * t1 + t0))
                th.append(t)
                wt.append(0.25 * (t1 - t0) * wh)
                rm.append(r0 * r1 * math.sin(t1 - t0) / (r0 * torch.sin(t - t0) - r1 * torch.sin(t - t1)))
        return torch.cat(th), torch.cat(wt), torch.cat(rm)

    def K_of(z0, e0, r, ct, st):
        return (cr[:, None, :, 1] * ct[None, :, None] + cr[:, None, :, 2] * st[None, :, None]
                + cr[:, None, :, 3] * (r * ct * st + z0 * st + e0 * ct)[None, :, None])

    def solid(z0, e0):
        th, wt, rm = polar(z0, e0)
        r = (0.5 * rm[:, None] * (xl[None] + 1)).reshape(-1)
        w = (wt[:, None] * 0.5 * rm[:, None] * wl[None]).reshape(-1)
        ct, st = torch.cos(th).repeat_interleave(12), torch.sin(th).repeat_interleave(12)
        K = K_of(z0, e0, r, ct, st)
        return (w * ct * st / K.norm(dim=-1) ** 3).sum(-1) * bdc / (4 * math.pi)

    eye = torch.arange(ne, device=dev)
    plane = (bdc / (cr[..., 1].norm(dim=-1) * cw[..., 2].norm(dim=-1))).abs() < 1e-15
    for tn in range(4):
        z0, e0 = float(zt[tn]), float(et[tn])
        th, wt, rm = polar(z0, e0)
        r = (0.5 * rm[:, None] * (xl[None] + 1)).reshape(-1)
        w = (wt[:, None] * 0.5 * rm[:, None] * wl[None]).reshape(-1)
        ct, st = torch.cos(th).repeat_interleave(12), torch.sin(th).repeat_interleave(12)
        K = K_of(z0, e0, r, ct, st)
        zeta, eta = r * ct + z0, r * st + e0
        _, W = _bilinear(cr[:, None], cw[:, None], zeta[None], eta[None])
        q = _qpgf64(p.qpd, (K * r[None, :, None]).reshape(-1, 3)).reshape(ne, len(r), 4)
        Nc = (_shape(zeta, eta) * (w * r)[:, None]).to(torch.complex128)
        G[4 * eye + tn, eye] = (q[..., 0] * W.norm(dim=-1)) @ Nc
        H[4 * eye + tn, eye] = (q[..., 1:] * W).sum(-1) @ Nc
        h = 1.0e-3
        f = [solid(z0, e0)]
        f.append((solid(z0 + h, e0) - solid(z0 - h, e0)) / (2 * h) / Tz[:, tn].norm(dim=-1))
        f.append((solid(z0, e0 + h) - solid(z0, e0 - h)) / (2 * h) / Te[:, tn].norm(dim=-1))
        F[4 * eye + tn, eye] = torch.where(plane[:, None], 0.0, torch.stack(f, -1))
    dF = F.sum(1)
    dF[:, 0] += 1.0
    G, H = G.reshape(N, N), H.reshape(N, N)
    i = torch.arange(N, device=dev)
    H[i, i] += dF[:, 0]
    zero = torch.zeros((2 * N, N), dtype=torch.complex128, device=dev)
    return dict(G=G, H=H, dG=zero, dH=zero, dF=dF)


def exact(case, seed):
    c = case
    if c["kind"] == "qpgf":
        return _exact_qpgf(c, seed)
    if c["kind"] == "field":
        return _exact_field(c, seed)
    if c["kind"] == "open" and c["shape"] == "sphere" and c["n"] <= 4:
        return _exact_open(c, seed)
    return None
