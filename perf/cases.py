"""The work that programs built on this engine have it do, as cases to time.

A case names a mesh, the look angles, the frequencies that share one ray grid, and the
public call that runs them:

  run     sbr.run: host arrays in, host arrays out (the CLI's sweep, run_sweep, freq_scan)
  plan    a resident sbr.Plan that is executed and read back again and again
  batch   a sbr.Plan over several meshes of uneven size, one ray grid and sweep each
  step    one step of a shape optimisation: new vertices, sweep, gradients
  bound   a sweep with its stated error against FP64
  open    a model that has just been read: scene set-up and its first look

Sizes: 10 rays per wavelength over the bounding aperture, meshes of 1k to 2M triangles,
1 to 64 frequencies, 1 to about 1000 angles, 2 to 6 bounces.  Seeds move the vertices,
turn the meshes and shift the sweep.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import sagittasbr_b200 as sbr
from sagittasbr_b200 import meshes

C0 = 299792458.0
PRECISION = {"mixed": sbr.PREC_MIXED, "fp32": sbr.PREC_FP32, "fp64": sbr.PREC_FP64}
# share of the bounding aperture that a mesh of each kind covers, about (for work())
FILL = {"icosphere": 0.78, "trihedral": 0.3, "aircraft": 0.07, "ellipsoid": 0.15, "plates": 0.2}
AIRCRAFT = 2_148_800  # triangles of the full-size aircraft


def _case(path, mesh, tris, angles, ghz, n_freqs=1, ghz_lo=None, bounces=3, precision="mixed", pol=False,
          per_angle=False, theta=90.0, phi=0.0, step=1.0, n_theta=1, meshes=1, name=None):
    c = dict(path=path, mesh=mesh, tris=tris, angles=angles, n_theta=n_theta, theta=theta, phi=phi, step=step,
             ghz=ghz, ghz_lo=ghz if ghz_lo is None else ghz_lo, n_freqs=n_freqs, bounces=bounces,
             precision=precision, pol=pol, per_angle=per_angle, meshes=meshes)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one look at a small model: what an interactive program or a short script asks for
        _case("run", "icosphere", 20_480, 1, 1.0, name="look-sphere"),
        # the reference sphere over 360 azimuths, repeated on a resident plan
        _case("plan", "icosphere", 20_480, 360, 1.0, name="sweep-sphere"),
        # corner reflector over a two-dimensional angle grid, three bounces on flat plates
        _case("run", "trihedral", 60_000, 961, 10.0, n_theta=31, theta=0.0, step=3.0, name="sweep-trihedral"),
        # the large production sweep: full-size aircraft, a wide band on one trace
        _case("plan", "aircraft", AIRCRAFT, 61, 18.0, 64, 1.0, bounces=5, step=0.5, name="wideband-aircraft"),
        # polarimetric sweep of a medium mesh
        _case("run", "aircraft", 537_000, 37, 6.0, 16, 1.0, bounces=5, pol=True, step=5.0, name="hhvv-aircraft"),
        # single-frequency azimuth sweep, fewer rays per triangle
        _case("run", "aircraft", 133_000, 181, 3.0, bounces=5, step=1.0, name="narrow-aircraft"),
        # validation sweep in double precision
        _case("run", "ellipsoid", 9_000, 31, 5.0, bounces=4, precision="fp64", phi=-30.0, step=2.0,
              name="fp64-ellipsoid"),
        # shape optimisation: forward and backward over 121 azimuths of a 200k-triangle mesh
        _case("step", "ellipsoid", 199_808, 121, 5.0, bounces=4, phi=-30.0, step=0.5, name="step-ellipsoid"),
        # sweep that also states its error
        _case("bound", "ellipsoid", 50_000, 61, 5.0, bounces=4, phi=-30.0, step=1.0, name="bound-ellipsoid"),
        # many meshes of uneven cost drained by one plan
        _case("batch", "mixed", 100_000, 1440, 8.0, bounces=4, meshes=16, name="batch-uneven"),
        # the reference's loop structure and arithmetic: one launch per (angle, frequency)
        _case("run", "plates", 6_912, 73, 6.0, 2, 4.0, bounces=6, precision="fp32", per_angle=True, theta=60.0,
              step=5.0, name="loop-plates"),
        # a model that was just read: tree build, set-up and a first look
        _case("open", "aircraft", 133_000, 1, 3.0, bounces=5, phi=35.0, name="open-aircraft"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(("run", "run", "run", "plan", "plan", "batch", "step", "bound", "open"))
    if path == "batch":
        return _case("batch", "mixed", log(20_000, 100_000), log(100, 1440), rng.uniform(2.0, 8.0),
                     bounces=rng.randint(2, 6), meshes=rng.randint(2, 16))
    mesh = rng.choice(("icosphere", "trihedral", "aircraft", "ellipsoid", "plates"))
    if path in ("step", "bound"):
        mesh = rng.choice(("ellipsoid", "icosphere"))
    # frequencies at which a mesh of this kind has between about 50 and 1000 rays across
    # (the aircraft 300 to 8000) on its aperture
    size = {"icosphere": 2.0, "trihedral": 1.75, "aircraft": 20.4, "ellipsoid": 4.0, "plates": 1.9}[mesh]
    across = log(300, 8000) if mesh == "aircraft" else log(50, 1000)
    ghz = across / (10.0 * size) * C0 / 1e9
    precision = rng.choice(("mixed", "mixed", "mixed", "fp32", "fp64")) if path in ("run", "plan") else "mixed"
    pol = path in ("run", "plan") and precision != "fp32" and rng.random() < 0.25
    n_freqs = rng.choice((1, 1, 2, 3, 4, 5, 8, 16, 31, 32, 33, 64)) if path in ("run", "plan") else 1
    if precision == "fp64":
        n_freqs = min(n_freqs, 8)
    tris = log(1_000, 1_000_000 if mesh == "aircraft" else 200_000)
    # angles up to a budget of rays (the listed sweeps have 2e7 to 2e9 of them in the mesh's shade)
    most = 2.0e8 / (across * across * FILL[mesh]) / (1.0 + n_freqs / 16.0)
    if precision == "fp64" or path == "bound":
        most /= 30.0
    angles = 1 if path == "open" else min(log(1, 1000), max(1, int(most)))
    per_angle = path == "run" and precision == "fp32" and angles * n_freqs <= 500
    return _case(path, mesh, tris, angles, ghz, n_freqs, ghz * rng.uniform(0.1, 0.9), rng.randint(2, 6), precision,
                 pol, per_angle, theta=rng.uniform(20.0, 160.0), phi=rng.uniform(0.0, 360.0),
                 step=rng.choice((0.5, 1.0, 2.0, 3.0)))


def _mesh(kind, tris, rng):
    """A mesh of about `tris` triangles, turned about z and with its vertices moved a little."""
    if kind == "icosphere":
        v, t = meshes.icosphere(min(7, max(2, round(math.log(tris / 20.0) / math.log(4.0)))), 1.0)
    elif kind == "trihedral":
        return meshes.trihedral(1.0, max(1, round(math.sqrt(tris / 6.0))))
    elif kind == "aircraft":
        s = math.sqrt(tris / AIRCRAFT)

        def n(x):
            return max(4, round(x * s))

        return meshes.aircraft(int(rng.integers(1 << 30)), 1e-3, (n(1000), n(600)), (n(100), n(1000)),
                               (n(50), n(250)))
    elif kind == "ellipsoid":
        n_theta = max(6, round(math.sqrt(tris / 4.0)))
        return meshes.ellipsoid_sh(n_theta=n_theta, n_phi=2 * n_theta, seed=int(rng.integers(1 << 30)))
    else:
        k = 24 if tris >= 2_000 else 6
        return meshes.plate_cluster(k, max(1, round(math.sqrt(tris / (2.0 * k)))), seed=int(rng.integers(1 << 30)))
    a = rng.uniform(0.0, 2.0 * math.pi)
    turn = np.array([[math.cos(a), -math.sin(a), 0.0], [math.sin(a), math.cos(a), 0.0], [0.0, 0.0, 1.0]])
    return (v @ turn.T * rng.uniform(0.98, 1.02)).astype(np.float32), t


def _angles(case, shift):
    m = case["n_theta"]
    th = case["theta"] + case["step"] * np.arange(m)
    ph = case["phi"] + case["step"] * np.arange(case["angles"] // m) + shift
    th, ph = np.meshgrid(th, ph, indexing="ij")
    return th.ravel(), ph.ravel()


def _freqs(case):
    if case["n_freqs"] == 1:
        return np.array([case["ghz"] * 1e9])
    return np.geomspace(case["ghz_lo"], case["ghz"], case["n_freqs"]) * 1e9


def _inputs(case, seed):
    """Mesh and job of a single-mesh case."""
    rng = np.random.default_rng(seed)
    v, t = _mesh(case["mesh"], case["tris"], rng)
    th, ph = _angles(case, rng.uniform(0.0, 1.0) * min(1.0, case["step"]))
    g = 2.0 * meshes.bounding_radius(v)
    n = meshes.rays_for(case["ghz"] * 1e9, g)
    return v, t, sbr.JobSpec(th, ph, _freqs(case), n, n, g, case["bounces"]), rng


def _options(case):
    return dict(precision=PRECISION[case["precision"]], polarization=sbr.POL_HHVV if case["pol"] else sbr.POL_SCALAR,
                mode=sbr.MODE_PER_ANGLE if case["per_angle"] else sbr.MODE_BATCHED)


def prepare(case, seed):
    path = case["path"]
    if path == "batch":
        # one mesh after another: triangles, frequency, sweep and bounces of their own
        rng = np.random.default_rng(seed)
        scenes, jobs = [], []
        for k in range(case["meshes"]):
            share = 1000.0 * (case["tris"] / 1000.0) ** (k / max(1, case["meshes"] - 1))
            v, t = _mesh(("icosphere", "trihedral", "ellipsoid", "plates")[k % 4], int(share), rng)
            g = 2.0 * meshes.bounding_radius(v)
            f = case["ghz"] * 1e9 * rng.uniform(0.25, 1.0)
            na = max(1, int(case["angles"] * (0.06 + 0.94 * (0.618 * (k + 1) % 1.0)) / 4))
            scenes.append(sbr.Scene(v, t))
            jobs.append(sbr.JobSpec(np.full(na, rng.uniform(30.0, 150.0)), np.linspace(0.0, 360.0, na, endpoint=False),
                                    [f], meshes.rays_for(f, g), meshes.rays_for(f, g), g,
                                    2 + (case["bounces"] + k) % 5))
        return dict(path=path, scenes=scenes, plan=sbr.Plan(scenes, jobs, job_scene=range(len(jobs))))
    v, t, job, rng = _inputs(case, seed)
    state = dict(path=path, job=job, options=_options(case))
    if path == "open":
        return dict(state, verts=v, tris=t)
    state["scene"] = scene = sbr.Scene(v, t, want_fp64=case["precision"] == "fp64")
    if path == "plan":
        state["plan"] = sbr.Plan(scene, [job], **state["options"])
    if path == "step":
        state["verts"] = (v * (1.0 + 1e-3 * rng.standard_normal((v.shape[0], 1)))).astype(np.float32)
    return state


def _out(r):
    return dict(field=r.field, sigma=r.sigma_m2, dbsm=r.rcs_dbsm, counts=r.stats)


def run(state):
    path = state["path"]
    if path in ("plan", "batch"):
        state["plan"].execute()
        return _out(state["plan"].results())
    if path == "open":
        with sbr.Scene(state["verts"], state["tris"], gpu_build=True) as scene:
            return _out(sbr.run(scene, state["job"], **state["options"]))
    if path == "step":
        # gradient of the mean RCS with respect to every vertex and the frequency
        state["scene"].update_vertices(state["verts"])
        r = sbr.run(state["scene"], state["job"], **state["options"])
        g_verts, g_freq = sbr.adjoint(state["scene"], state["job"], 8.0 * math.pi / r.field.size * r.field)
        return dict(_out(r), g_verts=g_verts, g_freq=g_freq)
    r = sbr.run(state["scene"], state["job"], **state["options"])
    if path == "bound":
        err_field, err_db = sbr.error_bound(state["scene"], state["job"], r)
        return dict(_out(r), err_field=err_field, err_db=err_db)
    return _out(r)


def work(case):
    """Every triangle and result moved once; per ray that meets the mesh one triangle test and
    reflection a bounce (about 100 operations, one bounce), and per channel one sine and cosine
    and their sum (about 20)."""
    channels = case["n_freqs"] * (2 if case["pol"] else 1)
    if case["path"] == "batch":
        angles, tris, fill, size = case["angles"] / 8.0 * case["meshes"], 0.3 * case["tris"] * case["meshes"], 0.3, 2.0
    else:
        angles, tris, fill = case["angles"], case["tris"], FILL[case["mesh"]]
        size = {"icosphere": 2.0, "trihedral": 1.75, "aircraft": 20.4, "ellipsoid": 4.0, "plates": 1.9}[case["mesh"]]
    across = 10.0 * size * case["ghz"] * 1e9 / C0 * (0.6 if case["path"] == "batch" else 1.0)
    rays = angles * across * across * fill
    passes = {"step": 3.0, "bound": 2.0}.get(case["path"], 1.0)
    return {"bytes": 48.0 * tris + 64.0 * angles * channels, "flops": passes * rays * (100.0 + 20.0 * channels)}


# ------------------------------------------------------------------ 64 bits
def _frame(theta, phi, g):
    th, ph = math.radians(theta), math.radians(phi)
    d = np.array([math.sin(th) * math.cos(ph), math.sin(th) * math.sin(ph), math.cos(th)])
    up = np.array([1.0, 0.0, 0.0]) if abs(d[1]) > 0.99 else np.array([0.0, 1.0, 0.0])
    u = np.cross(up, d)
    u *= g / np.linalg.norm(u)
    w = np.cross(d, u)
    w *= g / np.linalg.norm(w)
    return d, u, w, 10.0 * g * d - 0.5 * u - 0.5 * w


def _closest(o, d, a, b, c, n, chunk):
    """Nearest triangle of each ray by the signs of its three edge products, all pairs."""
    dev = o.device
    ray = torch.cat([d, torch.linalg.cross(o, d)], 1)
    best_t = torch.full((o.shape[0],), 1e20, dtype=torch.float64, device=dev)
    best = torch.full((o.shape[0],), -1, dtype=torch.int64, device=dev)
    for k in range(0, a.shape[0], chunk):
        p, q, r, m = a[k:k + chunk], b[k:k + chunk], c[k:k + chunk], n[k:k + chunk]
        s = [ray @ torch.cat([torch.linalg.cross(x, y), y - x], 1).T for x, y in ((p, q), (q, r), (r, p))]
        inside = ((s[0] >= 0) & (s[1] >= 0) & (s[2] >= 0)) | ((s[0] <= 0) & (s[1] <= 0) & (s[2] <= 0))
        dn = d @ m.T
        t = ((p * m).sum(1) - o @ m.T) / dn
        t = torch.where(inside & (dn.abs() >= 1e-6) & (t >= 1e-3), t, torch.inf)
        t, at = t.min(1)
        near = t < best_t
        best_t = torch.where(near, t, best_t)
        best = torch.where(near, at + k, best)
    return best_t, best


def exact(case, seed):
    """The scalar sweep in 64 bits, every ray against every triangle; None where that is too much."""
    if case["path"] not in ("run", "plan") or case["pol"] or not torch.cuda.is_available():
        return None
    v, t, job, _ = _inputs(case, seed)
    if 1.5 * FILL[case["mesh"]] * job.nx * job.ny * len(job.theta_deg) * t.shape[0] > 1.2e11:
        return None
    dev = torch.device("cuda")
    tri = torch.from_numpy(v.astype(np.float64)[t.astype(np.int64)]).to(dev)
    a, b, c = tri[:, 0], tri[:, 1], tri[:, 2]
    n = torch.linalg.cross(b - a, c - a)
    unit = n / n.norm(dim=1, keepdim=True).clamp_min(1e-300)
    corners = torch.from_numpy(v.astype(np.float64)).to(dev)
    freqs = torch.from_numpy(np.asarray(job.freqs_hz, np.float64)).to(dev)
    wave = 2.0 * math.pi * freqs / C0
    scale = wave * (job.grid_size ** 2 / (job.nx * job.ny)) / (4.0 * math.pi)
    fields = []
    for theta, phi in zip(job.theta_deg, job.phi_deg):
        e, eu, ev, corner = _frame(theta, phi, job.grid_size)
        e, eu, ev, corner = (torch.from_numpy(x).to(dev) for x in (e, eu, ev, corner))
        # rays inside the bounds of the projected mesh
        pu = (corners - corner) @ eu / (eu @ eu) * job.nx - 0.5
        pv = (corners - corner) @ ev / (ev @ ev) * job.ny - 0.5
        i = torch.arange(max(0, int(pu.min()) - 1), min(job.nx, int(pu.max()) + 2), device=dev, dtype=torch.float64)
        j = torch.arange(max(0, int(pv.min()) - 1), min(job.ny, int(pv.max()) + 2), device=dev, dtype=torch.float64)
        ii, jj = (x.reshape(-1, 1) for x in torch.meshgrid((i + 0.5) / job.nx, (j + 0.5) / job.ny, indexing="ij"))
        o = corner + ii * eu + jj * ev
        d = (-e).expand_as(o).contiguous()
        length = torch.zeros(o.shape[0], dtype=torch.float64, device=dev)
        cos = torch.zeros_like(length)
        gone = torch.arange(o.shape[0], device=dev)
        for _ in range(job.max_bounces):
            found = [_closest(o[k:k + 16384], d[k:k + 16384], a, b, c, n, 4096) for k in range(0, o.shape[0], 16384)]
            if not found:
                break
            dist, at = torch.cat([x[0] for x in found]), torch.cat([x[1] for x in found])
            k = at >= 0
            o, d, dist, gone, m = o[k], d[k], dist[k], gone[k], unit[at[k]]
            if not o.shape[0]:
                break
            length[gone] += dist
            dn = (d * m).sum(1, keepdim=True)
            cos[gone] = -dn[:, 0]
            o = o + dist[:, None] * d + 1e-4 * m
            d = d - 2.0 * dn * m
            d = d / d.norm(dim=1, keepdim=True)
        lit = cos > 0
        turn = torch.fmod(2.0 * wave[:, None] * length[lit][None], 2.0 * math.pi)
        amp = 2.0 * scale[:, None] * cos[lit][None]
        fields.append(torch.complex(-(amp * turn.sin()).sum(1), (amp * turn.cos()).sum(1)))
    field = torch.cat(fields).cpu().numpy()
    sigma = 4.0 * math.pi * np.abs(field) ** 2
    return dict(field=field, sigma=sigma, dbsm=10.0 * np.log10(np.maximum(sigma, 1e-10)), counts=None)
