"""The work whose speed counts: calls of the forward operator, its adjoint and the solvers, at the sizes they are used
at (the benchmark workloads ti256 and al99, the autograd test's Fe geometry, the serving configuration's ranges, the
Fourier-slice projector above 400 x 400 pixels).

listed() and draw(rng) give cases (plain dicts), prepare(case, seed) what a program holds before the call (operator and
inputs on the GPU), run(state) one pass through the public entry points, work(case) the bytes and operations a pass
cannot do without, tolerance(case) how far another correct implementation may be off, and exact(case, seed) the
outputs of the same inputs in float64, written here from the model's formulas in plain torch.
"""
import math

import numpy as np
import torch

HEXAGONAL_RINGS = [[1, 0, 0], [0, 0, 2], [1, 0, 1], [1, 0, 2], [1, 1, 0], [1, 0, 3], [2, 0, 0], [1, 1, 2]]   # Ti
CUBIC_RINGS = [[1, 1, 1], [2, 0, 0], [2, 2, 0], [3, 1, 1], [2, 2, 2]]                                       # Al
WAVELENGTH = 0.3        # Angstrom
CUT = 8.0               # the Gaussian is cut at 4 sigma: exponents up to 4^2 / 2


def _case(name, call, pixels, angles, lines, eta, rings, crystal, K, sigma, max_gb, **more):
    """pixels: (Nx, Ny); subsets 0: every angle in one call, else one of that many interleaved omega subsets."""
    c = dict(call=call, Nx=pixels[0], Ny=pixels[1], angles=angles, lines=lines, eta=eta, rings=rings, crystal=crystal,
             K=K, sigma=sigma, max_gb=max_gb, subsets=0, precision="fp32", projector="native", epochs=0)
    c.update(more)
    if name is not None:
        c["name"] = name
    return c


def listed():
    ti256 = dict(pixels=(256, 256), angles=360, lines=263, eta=360, rings=8, crystal="hexagonal", K=2000, sigma=2.0,
                 max_gb=3.9)
    al99 = dict(pixels=(99, 99), angles=180, lines=103, eta=180, rings=5, crystal="cubic", K=1000, sigma=3.0,
                max_gb=2.0)
    small = dict(pixels=(48, 48), angles=90, lines=53, eta=90, rings=3, crystal="cubic", K=500, sigma=5.0, max_gb=2.0)
    return [
        # one omega subset of the smallest slice that is served: an iteration is a few launches
        _case("direct_subset_48", "direct", subsets=8, **small),
        _case("adjoint_subset_48", "adjoint", subsets=8, **small),
        # a small slice of aluminium, every angle in one orientation batch: what a FISTA iteration applies
        _case("direct_99", "direct", **al99),
        _case("adjoint_99", "adjoint", **al99),
        # forward and gradient through autograd, several orientation batches
        _case("autograd_128", "autograd", (128, 128), 180, 133, 120, 5, "cubic", 5000, 3.0, 0.4),
        # the benchmark's slice, the drop-in float32 operator
        _case("direct_256", "direct", **ti256),
        _case("adjoint_256", "adjoint", **ti256),
        # the same on the tensor cores
        _case("direct_256_bf16", "direct", precision="bf16", **ti256),
        _case("adjoint_256_bf16", "adjoint", precision="bf16", **ti256),
        # whole reconstructions: step sizes, epochs with the objective of each, download of the dual variables
        _case("spdhg_99", "spdhg", subsets=10, epochs=20, **al99),
        _case("spdhg_256_bf16", "spdhg", subsets=20, epochs=10, precision="bf16", **ti256),
        # a grid above 400 x 400 pixels: the Fourier-slice projector, forward and adjoint
        _case("pair_416_fourier", "pair", (416, 416), 360, 424, 180, 5, "cubic", 256, 3.0, 2.0, projector="fft"),
    ]


def draw(rng):
    """A case of the same ranges: 48^2 to 256^2 pixels (square or not, odd sizes among them), 90 to 360 angles and eta
    bins, 3 to 8 rings, 200 to 2000 orientations (any count), whole scans and subsets, either precision."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(["direct", "direct", "adjoint", "adjoint", "autograd", "spdhg", "pair"])
    angles, eta = log_int(90, 360), log_int(90, 360)
    # one node per bin resolves kernels at least this wide: the widths that grids for such scans have
    sigma = max(2.0, 1.02 * math.degrees(math.sqrt(((math.pi / angles) ** 2 + (2 * math.pi / eta) ** 2) / (24 * 0.0495))))
    sigma = round(rng.uniform(sigma, max(5.0, 1.2 * sigma)), 3)
    crystal = rng.choice(["cubic", "hexagonal"])
    rings = rng.randint(3, 5 if crystal == "cubic" else 8)
    projector = "fft" if call == "pair" and rng.random() < 0.5 else "native"
    K = log_int(200, 2000)
    nx = log_int(48, 256)
    if call == "spdhg" or projector == "fft":
        nx, K = min(nx, 128), min(K, 1000)
    ny = nx if rng.random() < 0.7 else max(33, int(nx * rng.uniform(0.6, 1.0)))
    lines = max(nx, ny) + rng.randint(1, 9)
    precision = "bf16" if projector == "native" and call in ("direct", "adjoint", "spdhg") and rng.random() < 0.5 else "fp32"
    subsets = rng.choice([0, 0, 8, 10, 20]) if call in ("direct", "adjoint") else (rng.choice([8, 10, 20]) if call == "spdhg" else 0)
    return _case(None, call, (nx, ny), angles, lines, eta, rings, crystal, K, sigma, rng.choice([0.25, 1.0, 3.9]),
                 precision=precision, projector=projector, subsets=subsets,
                 epochs=rng.randint(3, 12) if call == "spdhg" else 0)


# ------------------------------------------------------------------------------------------------ inputs
def _rotations(case, seed):
    """(K, 3, 3) float64 orientations, uniform (normalised Gaussian quaternions)."""
    q = np.random.default_rng([seed, 1]).standard_normal((case["K"], 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    w, x, y, z = q.T
    return np.stack([np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)], -1),
                     np.stack([2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)], -1),
                     np.stack([2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1)], 1)


def _generator(seed, part):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 16 + part)
    return g


def _support(case):
    """(Ny, Nx) bool: pixels that project onto the detector at every angle."""
    x = (np.arange(case["Nx"]) - (case["Nx"] - 1) / 2.0)[None, :]
    y = (np.arange(case["Ny"]) - (case["Ny"] - 1) / 2.0)[:, None]
    ok = np.ones((case["Ny"], case["Nx"]), bool)
    for a in _angles(case):
        ok &= np.abs(np.cos(a - np.pi / 2) * x + np.sin(a - np.pi / 2) * y) <= case["lines"] / 2.0 + 1e-9 * case["lines"]
    return ok


def _grains(case, seed):
    """(orientation of every pixel (-1: outside the sample), the orientations that occur)."""
    rng = np.random.default_rng([seed, 2])
    n = int(min(200, case["K"], 3 + case["Nx"] * case["Ny"] // 300))
    ok = _support(case)
    ys, xs = np.nonzero(ok)
    at = rng.choice(len(ys), n, replace=False)
    which = rng.choice(case["K"], n, replace=False)
    yy, xx = np.mgrid[:case["Ny"], :case["Nx"]]
    owner = np.zeros(ok.shape, np.int64)
    best = np.full(ok.shape, np.inf)
    for i, j in enumerate(at):
        d = (yy - ys[j]) ** 2.0 + (xx - xs[j]) ** 2.0
        owner = np.where(d < best, i, owner)
        best = np.minimum(d, best)
    return np.where(ok, owner, -1), which


def _coefficients(case, seed):
    """(K, Ny, Nx) float32 as a reconstruction holds them: grains of one orientation each over small positive values
    everywhere in the sample."""
    g = _generator(seed, 3)
    owner, which = _grains(case, seed)
    ok = torch.as_tensor(owner >= 0, device="cuda")
    x = torch.rand((case["K"], case["Ny"], case["Nx"]), generator=g, device="cuda")
    x.pow_(3).mul_(0.05).mul_(ok)
    o = torch.as_tensor(owner, device="cuda")
    for i, k in enumerate(which):
        x[int(k)] += (o == i).to(torch.float32)
    return x


def _residual(case, seed):
    """(angles, lines, eta * rings) float32 as the adjoint meets it: signed, about normal, of count noise."""
    g = _generator(seed, 4)
    return torch.randn((case["angles"], case["lines"], case["eta"] * case["rings"]), generator=g, device="cuda")


def _counts(case, seed):
    """Poisson counts, mean 50, of the grains' diffraction (the float64 model of this file)."""
    owner, which = _grains(case, seed)
    o = torch.as_tensor(owner, device="cuda")
    x = torch.stack([(o == i) for i in range(len(which))]).to(torch.float64)
    lam = _forward64(case, _rotations(case, seed)[which], x, _all(case), keep=torch.float32)
    lam *= 50.0 / float(lam.double().mean())
    return torch.poisson(lam, generator=_generator(seed, 5))


def prepare(case, seed):
    from diffractom_b200 import Grid, Material, SinglePhaseForwardOperator
    lattice = dict(a=4.05) if case["crystal"] == "cubic" else dict(a=2.95, c=4.68, gamma=120)
    hkl = (CUBIC_RINGS if case["crystal"] == "cubic" else HEXAGONAL_RINGS)[:case["rings"]]
    mat = Material.from_lattice_parameters(**lattice, symmetry_group=case["crystal"], wavelength_A=WAVELENGTH,
                                           hkl_list=hkl)
    cfg = dict(Nx=case["Nx"], Ny=case["Ny"], My=case["lines"], N_Omega=case["angles"], angle_range=[0, 180],
               cor_offset=0.0, voxel_size=1.0, N_eta=case["eta"], eta_angle_range=[0, 360],
               energy=12.398 / WAVELENGTH, k_direction_0=[0, 0, 1], p_direction_0=[1, 0, 0],
               detector_direction_origin=[0, -1, 0], detector_direction_positive_90=[0, 0, -1])
    grid = Grid.from_rotation_matrices(_rotations(case, seed), np.deg2rad(case["sigma"]))
    op = SinglePhaseForwardOperator(cfg, mat, grid, case["max_gb"], normalized=True, precision=case["precision"],
                                    projector=case["projector"])
    st = dict(case=case, op=op)
    if case["call"] == "spdhg":
        st["b"] = _counts(case, seed)
        return st
    if case["subsets"]:
        op.set_omega_subsets(case["subsets"])
    if case["call"] != "adjoint":
        st["x"] = _coefficients(case, seed)
    if case["call"] != "direct":
        st["d"] = _residual(case, seed)
    if case["call"] in ("direct", "pair"):
        st["data"] = torch.zeros(op.data_shape, dtype=torch.float32, device="cuda")
    if case["call"] in ("adjoint", "pair"):
        st["coeffs"] = torch.zeros(op.coeff_shape, dtype=torch.float32, device="cuda")
    return st


def run(state):
    case, op = state["case"], state["op"]
    subset = 1 if case["subsets"] else None
    if case["call"] == "direct":
        op.direct_cl(state["x"], state["data"], subset=subset)
        return state["data"]
    if case["call"] == "adjoint":
        op.adjoint_cl(state["d"], state["coeffs"], subset=subset)
        return state["coeffs"]
    if case["call"] == "pair":
        op.direct_cl(state["x"], state["data"])
        op.adjoint_cl(state["d"], state["coeffs"])
        return state["data"], state["coeffs"]
    if case["call"] == "autograd":
        from diffractom_b200.autograd import forward_operator
        x = state["x"].detach().requires_grad_(True)
        y = forward_operator(op, x)
        (grad,) = torch.autograd.grad(y, x, state["d"])
        return y.detach(), grad
    from diffractom_b200 import SPDHGPoisson
    solver = SPDHGPoisson(op, subsets=case["subsets"], seed=0)
    x = solver.run(torch.zeros(op.coeff_shape, dtype=torch.float32, device="cuda"), state["b"], case["epochs"])
    return x, solver.state["y"], solver.state["z"]


# ------------------------------------------------------------------------------------------------ what it takes
def work(case):
    """Coefficients and data once each; the projector's taps (two per pixel and angle) and the pole figure's entries
    (the share of the sphere within 4 sigma of a pole axis) times the detector lines, two operations each. The
    Fourier-slice projector: its transforms and 7 x 7 interpolations instead of the taps."""
    npix, K, A = case["Nx"] * case["Ny"], case["K"], case["angles"]
    one = case["call"] in ("direct", "adjoint")
    used = len(range(1, A, case["subsets"])) if one and case["subsets"] else A
    coeffs, data = 4.0 * npix * K, 4.0 * used * case["lines"] * case["eta"] * case["rings"]
    axes = sum(len(np.unique(np.round(_half(v), 5), axis=0)) for v in _images(case))
    entries = used * K * case["eta"] * axes * (1 - math.cos(math.radians(4 * case["sigma"])))
    taps = 2.0 * 2.0 * npix * used * K
    if case["projector"] == "fft":
        m, n = 2.25 * npix, 1.25 * 1.5 * max(case["Nx"], case["Ny"])
        taps = K * (2.5 * m * math.log2(m) + used * n * (98.0 + 2.5 * math.log2(n)))
    flops = taps + 2.0 * entries * case["lines"]
    if one:
        return {"bytes": coeffs + data, "flops": flops}
    if case["call"] in ("pair", "autograd"):
        return {"bytes": 2 * (coeffs + data), "flops": 2 * flops}
    # a run: counts in, x, z and y out; the step sizes and every epoch a forward and an adjoint of all angles, and
    # the epoch's objective a forward more
    return {"bytes": 2 * coeffs + 2 * data, "flops": flops * (2 + 3 * case["epochs"])}


def tolerance(case):
    """Measured against exact() and, for the BF16 run, against the float32 operator's: about four times the float32
    calls' distance (3e-5: the exponents of the pole density near 1 - |n . v| = 0), twice the BF16 run's."""
    if case["call"] == "spdhg":
        return {"rel": 1e-2, "max": 0.9} if case["precision"] == "bf16" else {"rel": 3e-4}
    if case["precision"] == "bf16":
        return {"rel": 1e-2}
    return {"rel": 1e-4}


# ------------------------------------------------------------------------------------------------ float64 model
def _angles(case):
    return (np.arange(case["angles"]) + 0.5) * np.pi / case["angles"]


def _all(case):
    return np.arange(case["angles"])


def _group(case):
    """The proper rotations of the crystal's Laue group."""
    def turn(axis, deg):
        a = np.asarray(axis, float) / np.linalg.norm(axis)
        S = np.array([[0, -a[2], a[1]], [a[2], 0, -a[0]], [-a[1], a[0], 0]])
        t = np.deg2rad(deg)
        return np.eye(3) + np.sin(t) * S + (1 - np.cos(t)) * S @ S
    gens = ([turn((0, 0, 1), 90), turn((1, 1, 1), 120)] if case["crystal"] == "cubic"
            else [turn((0, 0, 1), 60), turn((1, 0, 0), 180)])
    group = [np.eye(3)]
    for g in group:
        for h in gens:
            m = h @ g
            if not any(np.allclose(m, o, atol=1e-9) for o in group):
                group.append(m)
    return np.stack(group)


def _rings(case):
    """Reciprocal vectors of the rings by increasing length (a* along x, c along z)."""
    if case["crystal"] == "cubic":
        hkl, B = CUBIC_RINGS, 2 * np.pi / 4.05 * np.eye(3)
    else:
        a, c = 2.95, 4.68
        ast = 4 * np.pi / (a * math.sqrt(3.0))
        hkl, B = HEXAGONAL_RINGS, np.array([[ast, 0.5 * ast, 0], [0, ast * math.sqrt(0.75), 0], [0, 0, 2 * np.pi / c]])
    h = np.asarray(hkl[:case["rings"]], float) @ B.T
    return h[np.argsort(np.linalg.norm(h, axis=1), kind="stable")]


def _images(case):
    """Per ring the directions of its reflection under the group, (G, 3)."""
    G = _group(case)
    return [G @ (h / np.linalg.norm(h)) for h in _rings(case)]


def _half(v):
    """Axes instead of directions: the first component that is not 0 is positive."""
    v = np.where(np.abs(v) < 1e-6, 0.0, v)
    lead = np.argmax(np.abs(v) > 1e-6, axis=1)
    return v * np.sign(v[np.arange(len(v)), lead])[:, None]


def _pole_figures(case, rot, a):
    """(K, eta * rings) float64: the pole density of every orientation at angle a's probed directions."""
    om = float(_angles(case)[a])
    eta = (np.arange(case["eta"]) + 0.5) * 2 * np.pi / case["eta"]
    base = np.stack([np.zeros_like(eta), -np.cos(eta), -np.sin(eta)], 1)
    R = np.array([[math.cos(om), -math.sin(om), 0], [math.sin(om), math.cos(om), 0], [0, 0, 1.0]])
    s2 = math.radians(case["sigma"]) ** 2
    U = torch.as_tensor(np.ascontiguousarray(rot), device="cuda")
    out = torch.empty((len(rot), case["eta"], case["rings"]), dtype=torch.float64, device="cuda")
    for p, (h, img) in enumerate(zip(_rings(case), _images(case))):
        th = math.asin(np.linalg.norm(h) * WAVELENGTH / (4 * np.pi))
        v = torch.as_tensor((base * math.cos(th) - math.sin(th) * np.array([1.0, 0, 0])) @ R, device="cuda")
        n = torch.einsum("kij,gj->kgi", U, torch.as_tensor(img, device="cuda"))
        e = (n.reshape(-1, 3) @ v.T).abs_().reshape(len(rot), len(img), -1)
        e = (1.0 - e).div_(s2)                          # the other hemisphere's 1 + |n . v| is past the cut
        out[:, :, p] = torch.where(e < CUT, torch.exp(-e), torch.zeros((), dtype=torch.float64, device="cuda")).sum(1)
    return out.reshape(len(rot), -1).div_(8 * math.pi * s2)


def _taps(case, a):
    """The projector of angle a transposed, (Ny * Nx, lines) sparse float64: bins under a pixel's footprint, the
    trapezoid of a unit step along the image axis with the larger coefficient."""
    th = _angles(case)[a] - np.pi / 2
    X, Y, ns = math.cos(th), math.sin(th), case["lines"]
    T0 = (ns - 1) / 2.0 - X * (case["Nx"] - 1) / 2.0 - Y * (case["Ny"] - 1) / 2.0
    x = torch.arange(case["Nx"], dtype=torch.float64, device="cuda")
    y = torch.arange(case["Ny"], dtype=torch.float64, device="cuda")
    t = (X * x[None, :] + Y * y[:, None] + T0).reshape(-1, 1)
    A = max(abs(X), abs(Y))
    s = torch.floor(t - (1 + A) / 2) + torch.arange(1, 4, device="cuda", dtype=torch.float64)[None, :]
    w = ((1 + A) / 2 - (t - s).abs()).clamp(min=0.0, max=A) / A
    w = torch.where((s >= 0) & (s < ns), w, torch.zeros_like(w))
    crow = torch.arange(0, 3 * len(t) + 1, 3, device="cuda")
    return torch.sparse_csr_tensor(crow, s.clamp(0, ns - 1).long().reshape(-1), w.reshape(-1), (len(t), ns))


def _waves(case, a):
    """The Fourier-slice projection of angle a: (e^{-i w x X} (Nx, H), e^{-i w (y Y + T0)} (Ny, H), line transform
    (lines, H)) with projection = Re(line sum_xy f e e)."""
    th = _angles(case)[a] - np.pi / 2
    X, Y, ns = math.cos(th), math.sin(th), case["lines"]
    ang = _angles(case) - np.pi / 2
    Xs, Ys = np.cos(ang), np.sin(ang)
    T0s = (ns - 1) / 2.0 - Xs * (case["Nx"] - 1) / 2.0 - Ys * (case["Ny"] - 1) / 2.0
    c = np.array([[u * (case["Nx"] - 1), v * (case["Ny"] - 1)] for u in (0, 1) for v in (0, 1)], float)
    t = c[:, :1] * Xs + c[:, 1:] * Ys + T0s
    L = int(math.ceil(1.25 * (max(t.max(), ns - 1) - min(t.min(), 0.0) + 4)))
    while L % 2 or not _smooth(L):
        L += 1
    w = torch.arange(L // 2 + 1, dtype=torch.float64, device="cuda") * (2 * np.pi / L)
    x = torch.arange(case["Nx"], dtype=torch.float64, device="cuda")[:, None]
    y = torch.arange(case["Ny"], dtype=torch.float64, device="cuda")[:, None]
    s = torch.arange(ns, dtype=torch.float64, device="cuda")[:, None]
    h = torch.sinc(w / (2 * np.pi)) ** 2 * 2.0 / L
    h[0] /= 2.0
    h[-1] /= 2.0
    one = torch.ones((), dtype=torch.float64, device="cuda")
    return (torch.polar(one.expand(len(x), len(w)), -x * X * w), torch.polar(one.expand(len(y), len(w)), -(y * Y + T0s[a]) * w),
            torch.polar(h.expand(ns, len(w)).contiguous(), s * w))


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _project(case, x, a, W=None):
    """(lines, K) float64 from (K, Ny, Nx) float64."""
    K = x.shape[0]
    if case["projector"] != "fft":
        W = _taps(case, a).to_sparse_coo().t().coalesce().to_sparse_csr() if W is None else W
        return W @ x.reshape(K, -1).t()
    ex, ey, line = _waves(case, a)
    f = torch.complex(x.reshape(-1, case["Nx"]) @ ex.real, x.reshape(-1, case["Nx"]) @ ex.imag)
    f = (f.reshape(K, case["Ny"], -1) * ey[None]).sum(1)
    return (line @ f.t()).real


def _backproject(case, z, a, img, WT=None):
    """img (K, Ny, Nx) += the transpose of _project on (lines, K)."""
    K = z.shape[1]
    if case["projector"] != "fft":
        img += ((_taps(case, a) if WT is None else WT) @ z).t().reshape(img.shape)
        return
    ex, ey, line = _waves(case, a)
    f = torch.complex(line.real.t() @ z, line.imag.t() @ z).t()                 # (K, H)
    g = (f[:, None, :] * ey[None]).reshape(K * case["Ny"], -1)
    img += (g.real @ ex.real.t() - g.imag @ ex.imag.t()).reshape(img.shape)


def _forward64(case, rot, x, rows, keep=torch.float64):
    out = torch.zeros((case["angles"], case["lines"], case["eta"] * case["rings"]), dtype=keep, device="cuda")
    for a in rows:
        out[a] = (_project(case, x, a) @ _pole_figures(case, rot, a)).to(keep)
    return out


def _adjoint64(case, rot, d, rows):
    img = torch.zeros((len(rot), case["Ny"], case["Nx"]), dtype=torch.float64, device="cuda")
    for a in rows:
        _backproject(case, d[a].double() @ _pole_figures(case, rot, a).t(), a, img)
    return img


def exact(case, seed):
    rot = _rotations(case, seed)
    rows = np.arange(1, case["angles"], case["subsets"]) if case["subsets"] else _all(case)
    if case["call"] == "spdhg":
        if case["Nx"] * case["Ny"] * case["K"] * case["epochs"] > 3e8:          # minutes in float64
            return None
        return _spdhg64(case, rot, _counts(case, seed).double())
    if case["call"] == "direct":
        return _forward64(case, rot, _coefficients(case, seed).double(), rows)
    if case["call"] == "adjoint":
        return _adjoint64(case, rot, _residual(case, seed), rows)
    return (_forward64(case, rot, _coefficients(case, seed).double(), rows),
            _adjoint64(case, rot, _residual(case, seed), rows))


def _spdhg64(case, rot, b):
    """SPDHG for the Poisson deviance with the diagonal step sizes, interleaved subsets in random order."""
    M, A, K = case["subsets"], case["angles"], case["K"]
    WT = [_taps(case, a) for a in range(A)]
    W = [m.to_sparse_coo().t().coalesce().to_sparse_csr() for m in WT]
    PF = torch.stack([_pole_figures(case, rot, a) for a in range(A)])
    ok = torch.as_tensor(_support(case), device="cuda").double()
    subsets = [list(range(m, A, M)) for m in range(M)]
    shape = (K, case["Ny"], case["Nx"])

    def forward(x, rows):
        return torch.stack([_project(case, x, a, W[a]) @ PF[a] for a in rows])

    def adjoint(d, rows):
        img = torch.zeros(shape, dtype=torch.float64, device="cuda")
        for i, a in enumerate(rows):
            _backproject(case, d[i] @ PF[a].t(), a, img, WT[a])
        return img

    gamma = math.sqrt(3e4) / float(b.mean())
    rowsum = forward(ok.expand(shape).contiguous(), range(A))
    S = torch.where(rowsum > 0, gamma / rowsum, torch.zeros_like(rowsum))
    T = torch.full(shape, math.inf, dtype=torch.float64, device="cuda")
    for rows in subsets:
        col = adjoint(torch.ones((len(rows),) + tuple(b.shape[1:]), dtype=torch.float64, device="cuda"), rows)
        T = torch.where((col > 0) & (ok > 0), torch.minimum(T, 1.0 / (M * gamma * col)), T)
    T[torch.isinf(T)] = 0.0
    x, z = torch.zeros(shape, dtype=torch.float64, device="cuda"), torch.zeros(shape, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(b)
    rng = np.random.default_rng(0)
    last = None
    for _ in range(case["epochs"]):
        order = rng.permutation(M)
        if M > 1 and int(order[0]) == last:
            order[[0, 1]] = order[[1, 0]]
        last = int(order[-1])
        for m in order:
            rows = subsets[int(m)]
            yo, s = y[rows], S[rows]
            v = yo + s * (forward(x, rows) + float(np.float32(1e-3)))
            yn = 0.5 * (v + 1.0 - torch.sqrt((v - 1.0) ** 2 + 4.0 * s * b[rows]))
            yn = torch.where(s > 0, yn, torch.zeros_like(yn))
            y[rows] = yn
            dz = adjoint(yn - yo, rows)
            z += dz
            x = torch.where(T > 0, (x - T * (z + M * dz)).clamp(min=0.0), torch.zeros_like(x))
    return x, y, z
