"""Timed cases of the fitting paths, through the calls a program makes.

Every case is one fit of a set of voxels whose gradient table, design handles and (but for the
whole-model call) signals are already on the device, which is how the models, the batches and
the server hold them. The matrices of every problem are built here from their equations, and
`exact` fits the same inputs in 64 bits with plain torch.

kinds and what they stand for:
  dti     the tensor maps of a table's masked voxels (OLS or WLS)
  model   DTIModel.fit, raw host volume in, host maps on the grid out
  dki     the kurtosis fit with its maps, constrained (the default) or not
  msmt    MSMT-CSD: a linearly constrained least-squares problem per voxel
  mfod    three-tissue mFOD: rounds of NNLS and fractions, then the 300-direction FOD
  csd     single-shell CSD of the highest shell
  peaks   amplitudes of SH series on the icosphere and the peak search
  drl     single-tissue damped Richardson-Lucy on the 300 directions
"""

from __future__ import annotations

import math
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
DIRS_300 = np.load(ROOT / "larmor_b200" / "data" / "dirs300.npy").astype(np.float64)

MAX_REWEIGHTINGS, LOG_TOL = 20, 1e-6
MAX_ROUNDS, FRACTION_TOL, FINAL_TOL_X, NNLS_TOL_X, RIDGE = 50, 1e-7, 1e-2, 1e-6, 0.1
DRL_ITERATIONS = 200


def listed() -> list[dict]:
    return [
        # One slice of a clinical DTI scan: the smallest call a viewer or a script makes.
        {"name": "dti_slice", "kind": "dti", "voxels": 2_003, "b0": 1, "shells": 1, "dirs": 30, "weighted": True},
        # The benchmark's 64x64x40 DTI volume (mask of 79,912 voxels, 1 b0 + 30 directions).
        {"name": "dti_volume", "kind": "dti", "voxels": 79_912, "b0": 1, "shells": 1, "dirs": 30, "weighted": True},
        # The whole model call on that volume, host arrays in and out.
        {"name": "dti_model", "kind": "model", "nx": 64, "ny": 64, "nz": 40, "b0": 1, "shells": 1, "dirs": 30,
         "weighted": True},
        # A region of interest of a two-shell kurtosis scan, a ragged table.
        {"name": "dki_region", "kind": "dki", "voxels": 3_001, "b0": 5, "shells": 2, "dirs": 45, "weighted": True,
         "constrained": True},
        # The benchmark's 96x96x60 kurtosis volume (199,768 voxels, 134 measurements).
        {"name": "dki_volume", "kind": "dki", "voxels": 199_768, "b0": 6, "shells": 2, "dirs": 64, "weighted": True,
         "constrained": True},
        # MSMT-CSD of a region, and of a brain at 2.5 mm or so.
        {"name": "msmt_region", "kind": "msmt", "voxels": 4_099, "b0": 10, "shells": 3, "dirs": 90, "lmax": 8},
        {"name": "msmt_volume", "kind": "msmt", "voxels": 100_003, "b0": 10, "shells": 3, "dirs": 90, "lmax": 8},
        # A serving request (4k-65k voxels of the three-tissue table), and a large volume.
        {"name": "mfod_request", "kind": "mfod", "voxels": 8_191, "b0": 10, "shells": 3, "dirs": 90},
        {"name": "mfod_volume", "kind": "mfod", "voxels": 250_000, "b0": 10, "shells": 3, "dirs": 90},
        # The benchmark's 110x110x70 mask: its b = 3000 shell, and the peaks of its FODs.
        {"name": "csd_volume", "kind": "csd", "voxels": 500_040, "dirs": 90, "lmax": 8},
        {"name": "peaks_volume", "kind": "peaks", "voxels": 500_040, "lmax": 8, "peaks": 3},
        # Damped Richardson-Lucy of a brain, the default solver's 200 iterations.
        {"name": "drl_volume", "kind": "drl", "voxels": 100_003, "b0": 10, "shells": 3, "dirs": 90,
         "precision": "fp64"},
    ]


def draw(rng) -> dict:
    def spread(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["dti", "model", "dki", "msmt", "mfod", "csd", "peaks", "drl"])
    table = {"b0": rng.randint(1, 10), "shells": rng.randint(2, 3), "dirs": rng.randint(30, 90)}
    if kind == "dti":
        table["shells"] = rng.randint(1, 3)
        return {"kind": kind, "voxels": spread(1_000, 79_912), **table, "weighted": rng.random() < 0.75}
    if kind == "model":
        return {"kind": kind, "nx": rng.randint(24, 64), "ny": rng.randint(24, 64), "nz": rng.randint(8, 40), "b0": 1,
                "shells": 1, "dirs": rng.randint(12, 64), "weighted": rng.random() < 0.75}
    if kind == "dki":
        n = table["b0"] + table["shells"] * table["dirs"]
        return {"kind": kind, "voxels": spread(1_000, 199_768 * min(134, n) // (2 * n)), **table,
                "weighted": rng.random() < 0.85, "constrained": rng.random() < 0.8}
    if kind == "msmt":
        table["dirs"] = rng.randint(60, 90)
        return {"kind": kind, "voxels": spread(2_000, 100_003), **table, "lmax": rng.choice([6, 8])}
    if kind == "mfod":
        return {"kind": kind, "voxels": spread(4_096, 250_000), **table}
    if kind == "csd":
        return {"kind": kind, "voxels": spread(4_000, 500_040), "dirs": rng.randint(45, 90),
                "lmax": rng.choice([6, 8])}
    if kind == "peaks":
        return {"kind": kind, "voxels": spread(4_000, 500_040), "lmax": rng.choice([4, 6, 8]),
                "peaks": rng.randint(2, 5)}
    return {"kind": "drl", "voxels": spread(2_000, 100_003), **table,
            "precision": "tf32x3" if rng.random() < 0.25 else "fp64"}


# ---- tables and matrices -------------------------------------------------------------------


def _table(case) -> tuple[np.ndarray, np.ndarray]:
    """b-values and unit b-vectors: b0s, then `dirs` random directions on each shell of 1000,
    2000, 3000 s/mm^2 (a fixed table for a case's shape)."""
    rng = np.random.default_rng([case.get("b0", 0), case.get("shells", 1), case["dirs"]])
    bvals, bvecs = [np.zeros(case.get("b0", 0))], [np.zeros((case.get("b0", 0), 3))]
    for k in range(case.get("shells", 1)):
        d = rng.normal(size=(case["dirs"], 3))
        bvals.append(np.full(case["dirs"], 1000.0 * (k + 1)))
        bvecs.append(d / np.linalg.norm(d, axis=1, keepdims=True))
    return np.concatenate(bvals), np.vstack(bvecs)


def _tensor_columns(b, g):
    x, y, z = g.T
    return np.stack([b * x * x, 2 * b * x * y, 2 * b * x * z, b * y * y, 2 * b * y * z, b * z * z], axis=1)


KT = ((0, 0, 0, 0), (1, 1, 1, 1), (2, 2, 2, 2), (0, 0, 0, 1), (0, 0, 0, 2), (1, 1, 1, 0), (1, 1, 1, 2), (2, 2, 2, 0),
      (2, 2, 2, 1), (0, 0, 1, 1), (0, 0, 2, 2), (1, 1, 2, 2), (0, 0, 1, 2), (1, 1, 0, 2), (2, 2, 0, 1))
KT_TIMES = (1, 1, 1, 4, 4, 4, 4, 4, 4, 6, 6, 6, 12, 12, 12)


def _kt_columns(g):
    return np.stack([t * g[:, i] * g[:, j] * g[:, k] * g[:, q] for (i, j, k, q), t in zip(KT, KT_TIMES)], axis=1)


def _log_design(case):
    """The log-signal design and constraints of DTI (7 columns) or DKI (22)."""
    b, g = _table(case)
    x = np.column_stack([np.ones(len(b)), -_tensor_columns(b, g)])
    if case["kind"] != "dki":
        return x, np.zeros((0, 7))
    x = np.column_stack([x, (b * b / 6)[:, None] * _kt_columns(g)])
    if not case["constrained"]:
        return x, np.zeros((0, 22))
    i = np.arange(256) + 0.5
    z, phi = 1 - i / 256, np.pi * (3 - np.sqrt(5)) * i
    r = np.sqrt(1 - z * z)
    dirs = np.stack([r * np.cos(phi), r * np.sin(phi), z], axis=1)
    d, v, one = _tensor_columns(np.ones(256), dirs), _kt_columns(dirs), np.zeros((256, 1))
    rows = [np.hstack([one, d, 0 * v]), np.hstack([one, 0 * d, v]), np.hstack([one, 3.0 / b.max() * d, -v])]
    return x, np.vstack(rows)


def _sh(dirs, lmax):
    """The real orthonormal SH basis of even degrees, order l then m = -l..l: sqrt(2) sin |m| phi
    for m < 0, sqrt(2) cos m phi for m > 0, with the Condon-Shortley sign."""
    z = np.clip(dirs[:, 2], -1.0, 1.0)
    s, phi = np.sqrt(1 - z * z), np.arctan2(dirs[:, 1], dirs[:, 0])
    p = {(0, 0): np.full(len(z), math.sqrt(1 / (4 * math.pi)))}
    for m in range(lmax + 1):
        if m:
            p[m, m] = -math.sqrt((2 * m + 1) / (2 * m)) * s * p[m - 1, m - 1]
        for l in range(m + 1, lmax + 1):  # noqa: E741
            a = math.sqrt((4 * l * l - 1) / (l * l - m * m))
            p[l, m] = a * z * p[l - 1, m]
            if l > m + 1:
                p[l, m] = p[l, m] - a * math.sqrt(((l - 1) ** 2 - m * m) / (4 * (l - 1) ** 2 - 1)) * p[l - 2, m]
    cols = []
    for l in range(0, lmax + 1, 2):  # noqa: E741
        for m in range(-l, l + 1):
            c = p[l, abs(m)]
            cols.append(c if m == 0 else math.sqrt(2) * c * (np.sin(-m * phi) if m < 0 else np.cos(m * phi)))
    return np.stack(cols, axis=1)


def _degrees(lmax):
    return np.concatenate([np.full(2 * l + 1, l) for l in range(0, lmax + 1, 2)])  # noqa: E741


def _fibre_response(bvals, lmax):
    """Zonal SH coefficients per b-value of a stick-zeppelin fibre of S0 1000 (Gauss-Legendre)."""
    x, w = np.polynomial.legendre.leggauss(64)
    zonal = _sh(np.stack([np.sqrt(1 - x * x), 0 * x, x], axis=1), lmax)
    zonal = zonal[:, [l * (l + 1) // 2 for l in range(0, lmax + 1, 2)]]  # noqa: E741
    rows = []
    for b in bvals:
        profile = 0.6 * np.exp(-b * 1.7e-3 * x * x) + 0.4 * np.exp(-b * (0.5e-3 + 1.2e-3 * x * x))
        rows.append(2 * np.pi * (w * 1000.0 * profile) @ zonal)
    return np.array(rows)


def _msmt_problem(case):
    """A x ~ s, G x >= 0 and the ridge of MSMT-CSD: white matter of degree lmax, GM, CSF."""
    b, g = _table(case)
    lmax = case["lmax"]
    deg = _degrees(lmax)
    sh = _sh(np.where(b[:, None] > 0, g, [0.0, 0.0, 1.0]), lmax)
    sh[np.ix_(b == 0, deg > 0)] = 0.0
    wm = sh * np.sqrt(4 * np.pi / (2 * deg + 1)) * _fibre_response(b, lmax)[:, deg // 2]
    iso = 1000.0 * np.sqrt(4 * np.pi) * np.stack([np.exp(-b * 0.8e-3), np.exp(-b * 3e-3)], axis=1)
    a = np.ascontiguousarray(np.hstack([wm, iso]))
    n = a.shape[1]
    cons = np.zeros((302, n))
    cons[:300, :n - 2] = _sh(DIRS_300, lmax)
    cons[300, n - 2] = cons[301, n - 1] = 1.0
    return a, cons, float(np.sqrt(1e-10 * (a * a).sum(axis=0).max()))


def _spiral(n):
    """n points of a Saff-Kuijlaars spiral flipped to z >= 0."""
    phi, out = 0.0, []
    for k in range(1, n + 1):
        h = -1 + 2 * (k - 1) / (n - 1)
        theta = np.arccos(h)
        phi = 0.0 if k in (1, n) else (phi + 3.6 / np.sqrt(n * (1 - h * h))) % (2 * np.pi)
        s = np.sign(np.cos(theta))
        out.append([s * np.cos(phi) * np.sin(theta), s * np.sin(phi) * np.sin(theta), s * np.cos(theta)])
    return np.array(out)


def _fibre_kernel(b, g, dirs):
    return np.ascontiguousarray(np.exp(-b[:, None] * (0.2e-3 + 1.5e-3 * (g @ dirs.T) ** 2)))


def _mfod_kernels(case):
    """The low- and high-resolution fibre kernels and the GM and CSF columns."""
    b, g = _table(case)
    iso = np.ascontiguousarray(np.stack([np.exp(-b * 0.8e-3), np.exp(-b * 3e-3)], axis=1))
    low = _spiral(min(len(b), 45))[:-1]
    return _fibre_kernel(b, g, low), _fibre_kernel(b, g, DIRS_300), iso


def _csd_problem(case):
    """The linear start, forward model, weighted constraint rows, norm weight and threshold of a
    single-shell CSD with the default settings (neg_lambda 1, norm_lambda 1, start of degree 4)."""
    _, g = _table({**case, "shells": 1})
    lmax = case["lmax"]
    deg = _degrees(lmax)
    zonal = _fibre_response([3000.0], lmax)[0]
    factor = (zonal / np.sqrt((2 * np.arange(0, lmax + 1, 2) + 1) / (4 * np.pi)))[deg // 2]
    sh = _sh(g, lmax)
    fit = lmax if (lmax + 1) * (lmax + 2) // 2 <= len(g) else lmax - 2
    d = _degrees(fit)
    initial = (np.linalg.pinv(_sh(g, fit)) / factor[:len(d), None])[d <= 4]
    forward = sh * factor
    weight = 50.0 * zonal[0] / 300
    return (np.ascontiguousarray(initial), np.ascontiguousarray(forward),
            np.ascontiguousarray(_sh(DIRS_300, lmax) * weight), 2e-4 * float(forward[:, 0] @ forward[:, 0]), 0.0, 50)


def _icosphere():
    data = np.load(ROOT / "larmor_b200" / "data" / "icosphere642.npz")
    return data["vertices"].astype(np.float64), data["neighbours"].astype(np.int64)


# ---- signals -------------------------------------------------------------------------------


class _Random:
    def __init__(self, seed, device="cuda"):
        self.g = torch.Generator(device=device)
        self.g.manual_seed(int(seed))
        self.device = device

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device=self.device, dtype=torch.float64)

    def uniform(self, low, high, *shape):
        return low + (high - low) * torch.rand(*shape, generator=self.g, device=self.device, dtype=torch.float64)

    def units(self, v):
        d = self.normal(v, 3)
        return d / d.norm(dim=1, keepdim=True)

    def shares(self, counts, v):
        """Dirichlet shares of integer parameters (gammas as sums of exponentials)."""
        s = torch.stack([-torch.log(1 - self.uniform(0, 1, v, c)).sum(dim=1) for c in counts], dim=1)
        return s / s.sum(dim=1, keepdim=True)

    def rician(self, s, sigma):
        return torch.sqrt((s + sigma * self.normal(*s.shape)) ** 2 + (sigma * self.normal(*s.shape)) ** 2)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _dti_signals(rng, b, g, v):
    """Tensors of l1 U[1.2, 2.0]e-3, l2 = l3 U[0.2, 0.6]e-3, random axis, S0 1000, SNR 20."""
    axis, l1, l2 = rng.units(v), rng.uniform(1.2e-3, 2.0e-3, v, 1), rng.uniform(0.2e-3, 0.6e-3, v, 1)
    adc = l2 + (l1 - l2) * (axis @ _dev(g).T) ** 2
    return rng.rician(1000.0 * torch.exp(-_dev(b) * adc), 50.0).float()


def _stick_zeppelin(b, cos2, f, d_par, d_perp):
    return f * torch.exp(-b * d_par * cos2) + (1 - f) * torch.exp(-b * (d_perp + (d_par - d_perp) * cos2))


def _dki_signals(rng, b, g, v):
    """A stick (share U[0.3, 0.7]) in a zeppelin (d_perp U[0.4, 0.8]e-3), S0 1000, SNR 30."""
    cos2 = (rng.units(v) @ _dev(g).T) ** 2
    s = _stick_zeppelin(_dev(b), cos2, rng.uniform(0.3, 0.7, v, 1), 2e-3, rng.uniform(0.4e-3, 0.8e-3, v, 1))
    return rng.rician(1000.0 * s, 1000.0 / 30).float()


def _tissue_signals(rng, b, g, v):
    """1-3 stick-zeppelin fibres (crossing U[30, 90] degrees) with GM and CSF, S0 1000, SNR 25."""
    bb, gg = _dev(b), _dev(g)
    n_fib = torch.randint(1, 4, (v, 1), generator=rng.g, device=rng.device)
    first, shares = rng.units(v), rng.shares([2, 2, 2], v)
    shares = shares * (torch.arange(3, device=rng.device) < n_fib)
    shares = shares / shares.sum(dim=1, keepdim=True)
    wm = torch.zeros((v, len(b)), dtype=torch.float64, device=rng.device)
    for k in range(3):
        axis = first
        if k:
            perp = torch.linalg.cross(first, rng.units(v))
            perp = perp / perp.norm(dim=1, keepdim=True)
            angle = torch.deg2rad(rng.uniform(30.0, 90.0, v, 1))
            axis = torch.cos(angle) * first + torch.sin(angle) * perp
        wm += shares[:, k:k + 1] * _stick_zeppelin(bb, (axis @ gg.T) ** 2, 0.6, 1.7e-3, 0.5e-3)
    pv = rng.shares([6, 2, 1], v)
    s = pv[:, :1] * wm + pv[:, 1:2] * torch.exp(-bb * 0.8e-3) + pv[:, 2:3] * torch.exp(-bb * 3e-3)
    return rng.rician(1000.0 * s, 40.0)


def _series(rng, v, lmax):
    """SH series of 1-3 fibres with a sharp profile and noise on every coefficient."""
    deg = _degrees(lmax)
    profile = _dev(np.exp(-0.02 * deg * (deg + 1)))
    n_fib = torch.randint(1, 4, (v, 1), generator=rng.g, device=rng.device)
    shares = rng.shares([2, 2, 2], v) * (torch.arange(3, device=rng.device) < n_fib)
    shares = shares / shares.sum(dim=1, keepdim=True)
    # Basis values through the dense grid-free formula: rows of the basis per random direction.
    out = 0.02 * rng.normal(v, len(deg))
    for k in range(3):
        out += shares[:, k:k + 1] * _sh_torch(rng.units(v), lmax) * profile
    return out


def _sh_torch(dirs, lmax):
    """_sh on a device tensor of directions."""
    z = dirs[:, 2].clamp(-1, 1)
    s, phi = torch.sqrt(1 - z * z), torch.atan2(dirs[:, 1], dirs[:, 0])
    p = {(0, 0): torch.full_like(z, math.sqrt(1 / (4 * math.pi)))}
    for m in range(lmax + 1):
        if m:
            p[m, m] = -math.sqrt((2 * m + 1) / (2 * m)) * s * p[m - 1, m - 1]
        for l in range(m + 1, lmax + 1):  # noqa: E741
            a = math.sqrt((4 * l * l - 1) / (l * l - m * m))
            p[l, m] = a * z * p[l - 1, m]
            if l > m + 1:
                p[l, m] = p[l, m] - a * math.sqrt(((l - 1) ** 2 - m * m) / (4 * (l - 1) ** 2 - 1)) * p[l - 2, m]
    cols = []
    for l in range(0, lmax + 1, 2):  # noqa: E741
        for m in range(-l, l + 1):
            c = p[l, abs(m)]
            cols.append(c if m == 0 else math.sqrt(2) * c * (torch.sin(-m * phi) if m < 0 else torch.cos(m * phi)))
    return torch.stack(cols, dim=1)


def _inputs(case, seed):
    """The signals of a case on the device, from the seed alone."""
    rng = _Random(seed)
    kind = case["kind"]
    if kind == "peaks":
        return _series(rng, case["voxels"], case["lmax"])
    if kind == "model":
        b, g = _table(case)
        mask = _ellipsoid(case)
        return _dti_signals(rng, b, g, int(mask.sum())), mask
    if kind == "csd":
        b, g = _table({**case, "shells": 1})
        return _tissue_signals(rng, np.full(len(b), 3000.0), g, case["voxels"])
    b, g = _table(case)
    if kind == "dti":
        return _dti_signals(rng, b, g, case["voxels"])
    if kind == "dki":
        return _dki_signals(rng, b, g, case["voxels"])
    s = _tissue_signals(rng, b, g, case["voxels"])
    if kind == "msmt":
        return s
    return torch.minimum(s / s[:, :case["b0"]].mean(dim=1, keepdim=True), torch.ones((), device=s.device))


def _ellipsoid(case):
    shape = (case["nx"], case["ny"], case["nz"])
    total = sum(((g - (n - 1) / 2) / (n / 2)) ** 2 for g, n in zip(np.indices(shape).astype(np.float64), shape))
    return total <= 0.977 ** 2


# ---- what a program holds, and the call ------------------------------------------------------


def prepare(case, seed):
    from larmor_b200 import _core

    kind = case["kind"]
    if kind == "model":
        from larmor_b200.dwi import DTIModel
        from larmor_b200.types import GradientTable, Volume

        inside, mask = _inputs(case, seed)
        data = np.zeros((*mask.shape, inside.shape[1]), dtype=np.float32)
        data[mask] = inside.cpu().numpy()
        return {"kind": kind, "model": DTIModel(fit_method="wls" if case["weighted"] else "ols"),
                "volume": Volume(data, np.eye(4)), "gtab": GradientTable(*_table(case)), "mask": mask}
    signals = _inputs(case, seed)
    v = len(signals)
    state = {"kind": kind, "signals": signals, "case": dict(case)}

    def out(*shape, dtype=torch.float64):
        return torch.empty(shape, dtype=dtype, device="cuda")

    if kind == "dti":
        x, g = _log_design(case)
        state |= {"design": _core.LogDesign(x, g), "floor": torch.full((v,), 1.0, dtype=torch.float64, device="cuda"),
                  "maps": out(16, v, dtype=torch.float32), "npd": out(v, dtype=torch.uint8)}
    elif kind == "dki":
        x, g = _log_design(case)
        b, _ = _table(case)
        s0 = signals[:, :case["b0"]].double().mean(dim=1)
        state |= {"x": x, "g": g, "s0": s0, "floor": 1e-3 * s0, "is_b0": b == 0}
    elif kind == "msmt":
        a, g, ridge = _msmt_problem(case)
        state |= {"design": _core.LsiDesign(a, g, ridge), "x": out(v, a.shape[1]), "conv": out(v, dtype=torch.uint8)}
    elif kind == "mfod":
        low, high, iso = _mfod_kernels(case)
        state |= {"weights": np.ones(len(iso)), "lr": _core.DeconvKernel(low, iso, iso, [(0, low.shape[1])]),
                  "hr": _core.DeconvKernel(high, iso, iso, [(0, 300)]),
                  "lr_solver": _core.FodSolver.l2nnls(low, 0.0, NNLS_TOL_X),
                  "hr_solver": _core.FodSolver.l2nnls(high, RIDGE, NNLS_TOL_X), "fods": out(v, 300),
                  "fractions": out(v, 3)}
    elif kind == "csd":
        state |= {"problem": _core.CsdProblem(*_csd_problem(case))}
    elif kind == "peaks":
        vertices, neighbours = _icosphere()
        state |= {"sphere": _core.PeakSphere(vertices, neighbours),
                  "projector": _core.ShProjector(np.ascontiguousarray(_sh(vertices, case["lmax"])))}
    else:
        k = _fibre_kernel(*_table(case), DIRS_300)
        k_t, k_t_k = np.ascontiguousarray(k.T), np.ascontiguousarray(k.T @ k)
        solver = _core.FodSolver.drl(k_t, k_t_k, _drl_nu(), DRL_ITERATIONS, 1.0 / 300)
        if case["precision"] != "fp64":
            solver.set_precision(case["precision"])
        state |= {"solver": solver}
    return state


def _drl_nu():
    """A damping threshold of the size the calibration on an isotropic tissue gives."""
    return 0.2 * 3.0e-3


def run(state):
    from larmor_b200 import _core

    kind = state["kind"]
    if kind == "model":
        fit = state["model"].fit(state["volume"], state["gtab"], state["mask"])
        return {"dt": fit.dt, "fa": fit.fa, "md": fit.md, "ad": fit.ad, "rd": fit.rd, "pe": fit.pe,
                "eigen_vals": fit.eigen_vals, "npd": fit.npd}
    s = state["signals"]
    if kind == "dti":
        _core.fit_dti_maps_device(state["design"], s, state["floor"], state["case"]["weighted"], state["maps"],
                                  state["npd"])
        maps = state["maps"]
        return {"tensor": maps[:10], "pe": maps[10:13], "eigen_vals": maps[13:], "npd": state["npd"]}
    if kind == "dki":
        from larmor_b200.dwi.dki import fit_dki_device

        maps, npd, broke = fit_dki_device(state["x"], state["g"], s, state["s0"], state["floor"], state["is_b0"],
                                          state["case"]["weighted"])
        return {"tensor": maps[:10], "pe": maps[10:13], "kt": maps[13:32], "kurtosis": maps[32:], "npd": npd,
                "broke": broke}
    if kind == "msmt":
        _core.fit_lsi_device(state["design"], s, state["x"], state["conv"])
        return {"x": state["x"], "converged": state["conv"]}
    if kind == "mfod":
        _core.fit_multi_tissue_device(s, state["weights"], state["lr"], state["lr_solver"], state["hr"],
                                      state["hr_solver"], MAX_ROUNDS, FRACTION_TOL, FINAL_TOL_X, state["fods"],
                                      state["fractions"])
        return {"fods": state["fods"], "fractions": state["fractions"]}
    if kind == "csd":
        fods, conv = _core.fit_csd_device(state["problem"], s)
        return {"fods": fods, "converged": conv}
    if kind == "peaks":
        on_sphere = _core.project_sh_device(state["projector"], s, False)
        dirs, amps = _core.find_peaks_device(state["sphere"], s, state["case"]["lmax"], False, on_sphere,
                                             state["case"]["peaks"], 0.1, 0.0)
        return {"directions": dirs, "amplitudes": amps}
    from larmor_b200.sd.solvers import fit_single_tissue_on_device

    return {"fods": fit_single_tissue_on_device(s, state["solver"])}


def work(case) -> dict:
    """Bytes in and out once, and the arithmetic of one sweep of each product the path is made of
    (iterations past the first where every voxel needs them: damped Richardson-Lucy's)."""
    kind = case["kind"]
    if kind == "peaks":
        v, c = case["voxels"], (case["lmax"] + 1) * (case["lmax"] + 2) // 2
        return {"bytes": v * (8 * c + 32 * case["peaks"]), "flops": v * 2 * c * 642}
    if kind == "csd":
        v, c = case["voxels"], (case["lmax"] + 1) * (case["lmax"] + 2) // 2
        return {"bytes": v * (8 * case["dirs"] + 8 * c + 1), "flops": v * (2 * c * (case["dirs"] + 300) + c ** 3 / 3)}
    n = case["b0"] + case["shells"] * case["dirs"]
    if kind == "model":
        v = int(_ellipsoid(case).sum())
        grid = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": grid * (4 * n + 4 * 16 + 1), "flops": v * n * 2 * (28 + 7 + 7)}
    v = case["voxels"]
    if kind == "dti":
        return {"bytes": v * (4 * n + 8 + 65), "flops": v * n * 2 * (28 + 7 + 7)}
    if kind == "dki":
        return {"bytes": v * (4 * n + 16 + 4 * 36 + 2), "flops": v * (n * 2 * (253 + 22 + 22) + 22 ** 3 / 3)}
    if kind == "msmt":
        c = (case["lmax"] + 1) * (case["lmax"] + 2) // 2 + 2
        return {"bytes": v * (8 * n + 8 * c + 1), "flops": v * 2 * c * (n + 302 + c)}
    if kind == "mfod":
        return {"bytes": v * (8 * n + 8 * 303), "flops": v * 2 * n * (44 + 300 + 44 + 300)}
    return {"bytes": v * 8 * (n + 300), "flops": v * 2.0 * 300 * (n + 300 * DRL_ITERATIONS)}


# ---- the same fits in 64 bits with plain torch -------------------------------------------------


def _rows(v, width, limit=1 << 31):
    """Slices of voxels whose (rows, width) doubles stay within `limit` bytes."""
    step = max(1, min(v, limit // (8 * width)))
    return [slice(i, min(v, i + step)) for i in range(0, v, step)]


def _log_fit(x, y, weighted):
    """The (re)weighted log-signal fits of y (v, n): parameters in unit-norm columns."""
    scale = x.norm(dim=0)
    xs = x / scale
    p = y @ torch.linalg.pinv(xs).T
    if weighted:
        live = torch.arange(len(y), device=y.device)
        for _ in range(MAX_REWEIGHTINGS):
            pred = p[live] @ xs.T
            w = torch.exp(2 * (pred - pred.amax(dim=1, keepdim=True)))
            gram = torch.stack([(w * xs[:, a:a + 1].T) @ xs for a in range(xs.shape[1])], dim=1)
            new = torch.linalg.solve(gram, (w * y[live]) @ xs)
            change = (new @ xs.T - pred).abs().amax(dim=1)
            p[live] = new
            live = live[change > LOG_TOL]
            if not len(live):
                break
    return p, scale, xs


def _nnls(columns, gram_row, corr, tol, c, cap):
    """Lawson-Hanson on normal equations for a batch of problems that share the rule: gram_row(idx,
    live) gives the active Gram blocks (rows, k, k), columns(idx, z, live) the gradient's G z over
    all c columns. corr (v, c)."""
    v, dev = len(corr), corr.device
    x = torch.zeros((v, c), dtype=torch.float64, device=dev)
    active = torch.zeros((v, c), dtype=torch.bool, device=dev)
    inner = torch.zeros(v, dtype=torch.int64, device=dev)
    live = torch.arange(v, device=dev)
    blocked = torch.zeros(v, dtype=torch.bool, device=dev)
    z_of = torch.zeros_like(x)
    while len(live):
        b = blocked[live]
        out_rows = live[~b]
        if len(out_rows):
            k = max(1, int(active[out_rows].sum(dim=1).max()))
            val, idx = active[out_rows].to(torch.int8).topk(k, dim=1)
            idx = idx.sort(dim=1).values
            xa = torch.gather(x[out_rows], 1, idx)
            g = corr[out_rows] - columns(idx, xa, out_rows)
            g = torch.where(active[out_rows], torch.full_like(g, -math.inf), g)
            best, e = g.max(dim=1)
            grow = best > (tol[out_rows] if torch.is_tensor(tol) else tol)
            active[out_rows[grow], e[grow]] = True
            done = out_rows[~grow]
            keep = torch.ones(v, dtype=torch.bool, device=dev)
            keep[done] = False
            live = live[keep[live]]
            if not len(live):
                break
        in_rows = live[blocked[live]]
        if len(in_rows):
            inner[in_rows] += 1
            a, xr, zr = active[in_rows], x[in_rows], z_of[in_rows]
            dist = xr - zr
            step = torch.where(a & (zr <= 0), torch.where(dist > 0, xr / dist, torch.zeros_like(xr)),
                               torch.full_like(xr, math.inf))
            st, j = step.min(dim=1)
            xr = xr + st[:, None] * (zr - xr)
            xr[torch.arange(len(j), device=dev), j] = 0.0
            a[torch.arange(len(j), device=dev), j] = False
            t = tol[in_rows, None] if torch.is_tensor(tol) else tol
            a = a & ~(xr.abs() < t)
            x[in_rows] = xr
            active[in_rows] = a
        n_act = active[live].sum(dim=1)
        k = max(1, int(n_act.max()))
        val, idx = active[live].to(torch.int8).topk(k, dim=1)
        gram = gram_row(idx, live)
        on = val > 0
        both = on[:, :, None] & on[:, None, :]
        gram = torch.where(both, gram, torch.eye(k, dtype=torch.float64, device=dev))
        rhs = torch.where(on, torch.gather(corr[live], 1, idx), torch.zeros((), dtype=torch.float64, device=dev))
        sol = torch.linalg.solve(gram, rhs)
        z = torch.zeros((len(live), c), dtype=torch.float64, device=dev)
        z.scatter_(1, idx, torch.where(on, sol, torch.zeros_like(sol)))
        z_of[live] = z
        bad = (active[live] & (z <= 0)).any(dim=1)
        out = bad & (inner[live] >= cap)
        x[live[~bad | out]] = z[~bad | out]
        blocked[live] = bad & ~out
        live = live[~out]
    return x


def _shared_nnls(gram, corr, tol, cap):
    """_nnls of one Gram matrix."""
    return _nnls(lambda idx, xa, live: torch.zeros((len(live), len(gram)), dtype=torch.float64, device=corr.device)
                 .scatter_add_(1, idx, xa) @ gram,
                 lambda idx, live: gram[idx[:, :, None], idx[:, None, :]], corr, tol, len(gram), cap)


def _fractions(fod, kernel, iso, signals, tol):
    """The tissue fractions: the FOD above its median as one column, next to the isotropic ones."""
    # The mean of the two middle values for even counts.
    s = fod.sort(dim=1).values
    n = fod.shape[1]
    med = s[:, n // 2] if n % 2 else (s[:, n // 2 - 1] + s[:, n // 2]) / 2
    th = torch.where(fod < (med * (1 - 1e-9))[:, None], torch.zeros_like(fod), fod)
    col = th @ kernel.T
    top = col.amax(dim=1, keepdim=True)
    col = torch.where(top > 0, col / top, col)
    cols = torch.cat([col[:, :, None], iso.expand(len(col), -1, -1)], dim=2)
    gram, corr = cols.transpose(1, 2) @ cols, (cols.transpose(1, 2) @ signals[:, :, None])[:, :, 0]
    if tol is None:
        tol = 10 * np.finfo(np.float64).eps * cols.abs().sum(dim=1).amax(dim=1) * max(cols.shape[1:])

    def rows(idx, live):
        return gram[live][torch.arange(len(live), device=idx.device)[:, None, None], idx[:, :, None], idx[:, None, :]]

    def column(idx, xa, live):
        full = torch.zeros_like(corr[live]).scatter_add_(1, idx, xa)
        return (gram[live] @ full[:, :, None])[:, :, 0]

    return _nnls(column, rows, corr, tol, cols.shape[2], 3 * cols.shape[2])


def _tensor_maps(d):
    """dt, FA, MD, AD, RD rows and eigenvalue rows of tensors (v, 6)."""
    m = torch.stack([d[:, 0], d[:, 1], d[:, 2], d[:, 1], d[:, 3], d[:, 4], d[:, 2], d[:, 4], d[:, 5]], dim=1)
    # The batched eigensolver takes a bounded batch.
    l = torch.cat([torch.linalg.eigvalsh(t) for t in m.reshape(-1, 3, 3).split(1 << 14)]).flip(1)  # noqa: E741
    num = ((l[:, 0] - l[:, 1]) ** 2 + (l[:, 1] - l[:, 2]) ** 2 + (l[:, 2] - l[:, 0]) ** 2).sqrt()
    fa = (math.sqrt(0.5) * num / l.norm(dim=1)).clamp(0, 1)
    md = (d[:, 0] + d[:, 3] + d[:, 5]) / 3
    return torch.cat([d.T, fa[None], md[None], l[:, 0][None], (l[:, 1] + l[:, 2])[None] / 2]), l.T


def _dki_params(case, signals):
    """The DKI parameters (v, 22), re-fitted under the constraints where they break one."""
    x, g = (_dev(a) for a in _log_design(case))
    s0 = signals[:, :case["b0"]].double().mean(dim=1, keepdim=True)
    s = signals.double()
    s = torch.cat([s[:, :case["b0"]], torch.minimum(s[:, case["b0"]:], s0)], dim=1)
    y = torch.log(s)
    p, scale, xs = _log_fit(x, y, case["weighted"])
    if case["constrained"]:
        gs = g / scale
        bad = torch.nonzero((p @ gs.T < 0).any(dim=1))[:, 0]
        pred = p[bad] @ xs.T
        w = torch.exp(pred - pred.amax(dim=1, keepdim=True)) if case["weighted"] else torch.ones_like(pred)
        q, r = torch.linalg.qr(w[:, :, None] * xs)
        free = torch.linalg.solve_triangular(r, q.transpose(1, 2) @ (w * y[bad])[:, :, None], upper=True)[:, :, 0]
        # Least distance: min |z| with G R^-1 z >= -G p_free, by NNLS on its dual.
        top = torch.linalg.solve_triangular(r.transpose(1, 2), gs.T.expand(len(bad), -1, -1), upper=False)
        cols = torch.cat([top, -(free @ gs.T)[:, None, :]], dim=1)
        tol = 10 * np.finfo(np.float64).eps * cols.abs().sum(dim=1).amax(dim=1) * len(gs)

        def picked(idx, live):
            return torch.gather(cols[live], 2, idx[:, None, :].expand(-1, cols.shape[1], -1))

        def gram(idx, live):
            a = picked(idx, live)
            return a.transpose(1, 2) @ a

        def column(idx, xa, live):
            res = picked(idx, live) @ xa[:, :, None]
            return (cols[live].transpose(1, 2) @ res)[:, :, 0]

        u = _nnls(column, gram, cols[:, -1, :].contiguous(), tol, len(gs), 50 * len(gs))
        res = (cols @ u[:, :, None])[:, :, 0]
        z = res[:, :-1] / (1 - res[:, -1:])
        p[bad] = free + torch.linalg.solve_triangular(r, z[:, :, None], upper=True)[:, :, 0]
    return p / scale


def exact(case, seed):
    kind = case["kind"]
    v = case.get("voxels", 0)
    if kind == "peaks" or (kind == "drl" and case["precision"] != "fp64"):
        return None  # the climb's stopping point is part of the result; an opt-in reduced precision
    if kind == "model":
        inside, mask = _inputs(case, seed)
        x, _ = _log_design(case)
        p, scale, _ = _log_fit(_dev(x), torch.log(inside.double()), case["weighted"])
        maps, ev = _tensor_maps((p / scale)[:, 1:])

        def grid(rows):
            full = np.zeros((*mask.shape, len(rows)))
            full[mask] = rows.T.cpu().numpy()
            return full

        names = {"fa": 6, "md": 7, "ad": 8, "rd": 9}
        return {"dt": grid(maps[:6]), **{k: grid(maps[i:i + 1])[..., 0] for k, i in names.items()},
                "eigen_vals": grid(ev)}
    signals = _inputs(case, seed)
    if kind == "dti":
        x, _ = _log_design(case)
        p, scale, _ = _log_fit(_dev(x), torch.log(signals.double()), case["weighted"])
        maps, ev = _tensor_maps((p / scale)[:, 1:])
        return {"tensor": maps, "pe": None, "eigen_vals": ev, "npd": None}
    if kind == "dki":
        if case["constrained"] and v > 12_000:
            return None
        p = torch.cat([_dki_params(case, signals[r]) for r in _rows(v, 768 * 23 if case["constrained"] else 22 * 300)])
        maps, ev = _tensor_maps(p[:, 1:7])
        md2 = (maps[7] ** 2).clamp(min=1e-300)
        kt = (p[:, 7:].T / md2)
        return {"tensor": maps, "pe": None, "kt": torch.cat([ev, kt, torch.exp(p[:, 0])[None]]), "kurtosis": None,
                "npd": None, "broke": None}
    if kind == "msmt":
        if v > 12_000:
            return None
        a, g, ridge = (_dev(m) if isinstance(m, np.ndarray) else m for m in _msmt_problem(case))
        n = a.shape[1]
        q, r = torch.linalg.qr(torch.cat([a, ridge * torch.eye(n, dtype=torch.float64, device=a.device)]))
        rot = signals @ q[:len(a)]
        e = torch.linalg.solve_triangular(r.T, g.T, upper=False).T
        norm = e.norm(dim=1, keepdim=True)
        e = e / norm
        f = -(rot @ e.T)
        scale = f.abs().amax(dim=1, keepdim=True)
        f = f / scale
        gram = e @ e.T
        tol = 10 * np.finfo(np.float64).eps * (e.abs().sum(dim=1) + f.abs()).amax(dim=1) * len(g)

        def rows(idx, live):
            fa = torch.gather(f[live], 1, idx)
            return gram[idx[:, :, None], idx[:, None, :]] + fa[:, :, None] * fa[:, None, :]

        def column(idx, xa, live):
            full = torch.zeros((len(live), len(g)), dtype=torch.float64, device=f.device).scatter_add_(1, idx, xa)
            return full @ gram + f[live] * (f[live] * full).sum(dim=1, keepdim=True)

        u = _nnls(column, rows, f, tol, len(g), 3 * len(g))
        z = scale * (u @ e) / (1 - (f * u).sum(dim=1, keepdim=True))
        x = torch.linalg.solve_triangular(r, (z + rot).T, upper=True).T
        return {"x": x, "converged": None}
    if kind == "mfod":
        if v > 12_000:
            return None
        low, high, iso = (_dev(m) for m in _mfod_kernels(case))
        f_iso = torch.zeros((v, 2), dtype=torch.float64, device=signals.device)
        prev = torch.full((v, 3), math.inf, dtype=torch.float64, device=signals.device)
        live = torch.arange(v, device=signals.device)
        gram = low.T @ low
        for _ in range(MAX_ROUNDS):
            s = (signals[live] - f_iso[live] @ iso.T).clamp(min=0)
            fod = _shared_nnls(gram, s @ low, NNLS_TOL_X, 3 * len(gram))
            fr = _fractions(fod, low, iso, signals[live], None)
            moved = ((fr - prev[live]).abs() >= FRACTION_TOL).any(dim=1)
            f_iso[live], prev[live] = fr[:, 1:], fr
            live = live[moved]
            if not len(live):
                break
        s = (signals - f_iso @ iso.T).clamp(min=0)
        gram = high.T @ high + RIDGE ** 2 * torch.eye(300, dtype=torch.float64, device=s.device)
        fod = _shared_nnls(gram, s @ high, NNLS_TOL_X, 900)
        fr = _fractions(fod, high, iso, signals, FINAL_TOL_X)
        return {"fods": fod, "fractions": fr / (fr.sum(dim=1, keepdim=True) + 1e-16)}
    if kind == "csd":
        initial, forward, cons, norm_weight, threshold, iterations = _csd_problem(case)
        i, m, c = (_dev(a) for a in (initial, forward, cons))
        n = m.shape[1]
        base = m.T @ m + norm_weight * torch.eye(n, dtype=torch.float64, device=m.device)
        outer = (c[:, :, None] * c[:, None, :]).reshape(len(c), -1)
        fods = []
        for r in _rows(v, n * n):
            s = signals[r]
            f = torch.zeros((len(s), n), dtype=torch.float64, device=s.device)
            f[:, :len(i)] = s @ i.T
            rhs = s @ m
            live = torch.arange(len(s), device=s.device)
            last = torch.zeros((len(s), len(c)), dtype=torch.bool, device=s.device)
            for it in range(iterations):
                below = f[live] @ c.T < threshold
                if it:
                    new = (below != last[live]).any(dim=1)
                    live, below = live[new], below[new]
                    if not len(live):
                        break
                last[live] = below
                h = base + (below.double() @ outer).reshape(-1, n, n)
                f[live] = torch.cholesky_solve(rhs[live, :, None], torch.linalg.cholesky(h))[:, :, 0]
            fods.append(f)
        return {"fods": torch.cat(fods), "converged": None}
    # Damped Richardson-Lucy.
    k = _dev(_fibre_kernel(*_table(case), DIRS_300))
    gram, nu8 = k.T @ k, _drl_nu() ** 8
    corr = signals @ k
    strength = (1 - 4 * signals.std(dim=1, keepdim=True)).clamp(min=0)
    stop = 1e-4 * signals.amax(dim=1)
    fod = torch.full((v, 300), 1.0 / 300, dtype=torch.float64, device=signals.device)
    live = torch.arange(v, device=signals.device)
    for _ in range(DRL_ITERATIONS):
        f = fod[live]
        pred = f @ gram
        damping = 1 - strength[live] * (1 - f ** 8 / (f ** 8 + nu8))
        new = (f * (1 + damping * (corr[live] - pred) / (pred + 1e-16))).clamp(min=1e-6)
        fod[live] = new
        live = live[(new - f).abs().sum(dim=1) > stop[live]]
        if not len(live):
            break
    return {"fods": fod}
