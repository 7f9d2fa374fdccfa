"""The workloads whose speed is followed: what a user of the library has it
do, through its public entry points.

listed() names the cases, draw() gives more of the same ranges, prepare()
makes what a program holds before the call, run() is one call, work() what the
result cannot do without, and exact() the result in 64-bit torch arithmetic,
written from the filters' definitions.

Kinds of cases:
  insar    NL-SAR of an InSAR pair on the device (nlsar_insar_device)
  host     the drop-in call on numpy arrays, copies included (nlsar_insar)
  covmat   NL-SAR of a 2x2 or 3x3 covariance image on the device
           (dcl_nlsar_covmat_device of the C ABI, which has no Python wrapper)
  batch    a prepared batch of scenes of uneven size (NlsarBatch)
  train    statistics of a homogeneous area (nlsar_train_insar)
  boxcar, goldstein, nlinsar  the other filters, on the device
"""
import ctypes
import functools
import math
import random

import numpy as np
import torch

import despeckcl_b200 as dcl
from despeckcl_b200 import api, synthetic

SEARCH = 21
# patch sizes and scale sizes in use: the benchmark's, the reference's example,
# one patch size at two scales, and a set that sorts as one patch per scale
SETTINGS = {"bench": ((3, 5, 7), (1, 3)), "example": ((3, 5, 7, 9, 11), (1, 3, 5)), "one": ((5,), (1, 3)),
            "small": ((3, 5), (1, 3))}


def listed():
    return [
        # a crop around a target, looked at interactively: one call's latency
        dict(name="insar_small", kind="insar", h=90, w=118, setting="bench", search=21, select="argmax_enl"),
        # the benchmark's small scene
        dict(name="insar_512", kind="insar", h=512, w=512, setting="bench", search=21, select="argmax_enl"),
        # the headline scene
        dict(name="insar_4096", kind="insar", h=4096, w=4096, setting="bench", search=21, select="argmax_enl"),
        # the settings of the reference's example script (15 combinations)
        dict(name="insar_example", kind="insar", h=997, w=1021, setting="example", search=21, select="argmax_enl"),
        # a script written for the reference's Python binding: numpy in and
        # out, the default selection, a scene with odd sides
        dict(name="host_default", kind="host", h=1531, w=1999, setting="bench", search=21, select="reference"),
        # covariance images: an InSAR pair as 8 planes, PolSAR as 18
        dict(name="covmat_2x2", kind="covmat", dim=2, h=1100, w=1203, setting="bench", search=21,
             select="argmax_enl"),
        dict(name="covmat_3x3", kind="covmat", dim=3, h=509, w=512, setting="bench", search=21,
             select="argmax_enl"),
        # a stack of crops filtered again and again by one prepared batch
        dict(name="batch_uneven", kind="batch", scenes=8, smallest=256, largest=1024, setting="bench", search=21,
             select="argmax_enl"),
        # statistics of a new sensor, before filtering
        dict(name="train_128", kind="train", h=128, w=128, setting="bench"),
        # the quick-look filters on large scenes
        dict(name="boxcar_8192", kind="boxcar", h=8192, w=8192, window=7),
        dict(name="goldstein_4099", kind="goldstein", h=4099, w=5003, overlap=4, alpha=0.5),
        # NL-InSAR with the reference's defaults, a few passes
        dict(name="nlinsar_600", kind="nlinsar", h=600, w=700, search=21, patch=7, niter=3, lmin=10),
    ]


def draw(rng):
    kind = rng.choice(["insar", "insar", "insar", "host", "covmat", "covmat", "batch", "train", "boxcar", "goldstein",
                       "nlinsar"])

    def sides(lo, hi):
        return [int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(2)]

    if kind == "train":
        h, w = rng.randint(48, 128), rng.randint(48, 128)
        return dict(kind=kind, h=h, w=w, setting=rng.choice(["bench", "one", "small"]))
    if kind == "boxcar":
        h, w = sides(128, 8192)
        return dict(kind=kind, h=h, w=w, window=rng.choice([3, 5, 7, 9, 11, 15]))
    if kind == "goldstein":
        h, w = sides(128, 4500)
        return dict(kind=kind, h=h, w=w, overlap=rng.choice([2, 4, 7]), alpha=round(rng.uniform(0.2, 0.9), 2))
    if kind == "nlinsar":
        h, w = sides(64, 640)
        return dict(kind=kind, h=h, w=w, search=rng.choice([15, 21]), patch=rng.choice([3, 7]),
                    niter=rng.randint(1, 3), lmin=rng.randint(5, 20))
    setting = rng.choice(["bench", "bench", "example", "one", "small"])
    c = dict(kind=kind, setting=setting, search=rng.choice([21, 21, 21, 15]),
             select=rng.choice(["argmax_enl", "argmax_enl", "reference"]))
    if kind == "batch":
        return dict(c, setting=rng.choice(["bench", "one"]), search=21, scenes=rng.randint(3, 10),
                    smallest=rng.randint(64, 256), largest=rng.randint(257, 1024))
    general = c["search"] != 21 or setting == "small"
    if kind == "covmat":
        c["dim"] = rng.choice([2, 3])
        c["h"], c["w"] = sides(64, 300 if general or setting == "example" else (1100 if c["dim"] == 2 else 512))
    else:
        c["h"], c["w"] = sides(64, 500 if general else (900 if setting == "example" else 2600))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _scene(h, w, seed):
    return synthetic.insar_scene_device(h, w, seed)


def _covmat_scene(dim, h, w, seed):
    """[2 dim^2][h][w] planes of a single-look covariance image."""
    if dim == 2:
        a1, a2, ph = _scene(h, w, seed)
        re, im, z = a1 * a2 * torch.cos(ph), a1 * a2 * torch.sin(ph), torch.zeros_like(a1)
        return torch.stack([a1 * a1, z, re, im, re, -im, a2 * a2, z]).contiguous()
    # three channels of one random covariance, brighter towards the right
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    z = torch.randn((3, 5), generator=g, device="cuda", dtype=torch.complex64)
    chol = torch.linalg.cholesky(z @ z.conj().T / 5)
    k = (chol @ torch.randn((3, h * w), generator=g, device="cuda", dtype=torch.complex64)).reshape(3, h, w)
    k = k * torch.linspace(1.0, 2.0, w, device="cuda")
    cov = k[:, None] * k[None, :].conj()
    return torch.view_as_real(cov.reshape(9, h, w)).permute(0, 3, 1, 2).reshape(18, h, w).contiguous()


def _train_area(h, w, seed):
    """A homogeneous pair: reflectivity 1, coherence 0.6, phase 0."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    x1, x2 = (torch.randn((h, w), generator=g, device="cuda", dtype=torch.complex64) for _ in range(2))
    s2 = 0.6 * x1 + 0.8 * x2
    return x1.abs().contiguous(), s2.abs().contiguous(), torch.angle(x1 * s2.conj()).contiguous()


def _batch_sides(case):
    r = random.Random("%(scenes)d %(smallest)d %(largest)d" % case)
    return [(r.randint(case["smallest"], case["largest"]), r.randint(case["smallest"], case["largest"]))
            for _ in range(case["scenes"])]


@functools.lru_cache(maxsize=8)
def _stats_tables(dim, setting):
    """{(patch, scale): (dmin, dmax, quantiles, chi2)} as a program loads them
    from its statistics file: trained once on a homogeneous area."""
    patches, scales = SETTINGS[setting]
    n = 64 if dim == 2 else 40
    if dim == 2:
        a1, a2, ph = (t.double() for t in _train_area(n, n, 7))
        planes = torch.stack([a1 * a1, 0 * a1, a1 * a2 * torch.cos(ph), a1 * a2 * torch.sin(ph), 0 * a1, 0 * a1,
                              a2 * a2, 0 * a1])
    else:
        planes = _covmat_scene(3, n, n, 7).double()
    return {(p, s): tuple(v.cpu().numpy().astype(np.float32) if torch.is_tensor(v) else np.float32(v)
                          for v in _train(planes, dim, p, s)) for p in patches for s in scales}


def _stats(dim, setting):
    out = dcl.StatsCollection()
    for (p, s), (lo, hi, q, c) in _stats_tables(dim, setting).items():
        out[dcl.Params(p, s)] = dcl.Stats(len(q), lo, hi, q, c)
    return out


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case)
    if kind == "train":
        st["in"] = [t.cpu().numpy() for t in _train_area(case["h"], case["w"], seed)]
        return st
    if kind in ("boxcar", "goldstein", "nlinsar"):
        st["in"] = _scene(case["h"], case["w"], seed)
        return st
    st["stats"] = _stats(case.get("dim", 2), case["setting"])
    st["patches"], st["scales"] = (list(v) for v in SETTINGS[case["setting"]])
    if kind == "insar":
        st["in"] = _scene(case["h"], case["w"], seed)
    elif kind == "host":
        st["in"] = [t.cpu().numpy() for t in _scene(case["h"], case["w"], seed)]
    elif kind == "covmat":
        st["in"] = _covmat_scene(case["dim"], case["h"], case["w"], seed)
        st["out"] = torch.empty_like(st["in"])
    else:
        scenes = [_scene(h, w, seed + 1000 * i) for i, (h, w) in enumerate(_batch_sides(case))]
        st["batch"] = dcl.NlsarBatch(scenes, case["search"], st["patches"], st["scales"], st["stats"],
                                     select_mode=case["select"])
    return st


def run(st):
    kind = st["kind"]
    if kind == "insar":
        return dcl.nlsar_insar_device(*st["in"], st["search"], st["patches"], st["scales"], st["stats"],
                                      select_mode=st["select"])
    if kind == "host":
        return dcl.nlsar_insar(*st["in"], st["search"], st["patches"], st["scales"], st["stats"],
                               select_mode=st["select"])
    if kind == "covmat":
        x, out = st["in"], st["out"]
        keep_p, pp, np_ = api._ints(st["patches"])
        keep_s, sp, ns = api._ints(st["scales"])
        arr, n, keep = api._entries(st["stats"])
        api._check(dcl.lib().dcl_nlsar_covmat_device(
            api._dptr(x), api._dptr(out), x.shape[1], x.shape[2], st["dim"], st["search"], pp, np_, sp, ns, arr, n,
            ctypes.c_float(15.0), ctypes.c_float(49.0), api._mode(st["select"]), api._stream(None)))
        return out
    if kind == "batch":
        return st["batch"].run()
    if kind == "train":
        patches, scales = SETTINGS[st["setting"]]
        got = dcl.nlsar_train_insar(*st["in"], list(patches), list(scales))
        return {"%d_%d" % (k.patch_size, k.scale_size): [s.dissims_min, s.dissims_max, s.quantilles, s.chi2cdf_inv]
                for k, s in got.items()}
    if kind == "boxcar":
        return dcl.boxcar_device(*st["in"], st["window"])
    if kind == "goldstein":
        return dcl.goldstein_device(*st["in"], 32, st["overlap"], st["alpha"])
    return dcl.nlinsar_device(*st["in"], st["search"], st["patch"], st["niter"], st["lmin"])


# ---------------------------------------------------------------------------
# work: planes read and written once, and the arithmetic of the definition
# with every separable sum taken separably and every mirrored weight once
# ---------------------------------------------------------------------------

def _nlsar_flops(dim, search, setting, select):
    patches, scales = SETTINGS[setting]
    if select == "reference":
        patches, scales = patches[-1:], scales[-1:]
    sim, acc = {2: (14, 2 * 8), 3: (60, 2 * 23)}[dim]
    half = (search * search - 1) // 2
    per_weight = sum(2 * (p - 1) + 4 for p in patches)  # box sums and the table index
    return len(scales) * (half * (sim + per_weight) + search * search * acc * len(patches))


def work(case):
    kind = case["kind"]
    if kind == "train":
        flops = 0
        for p in SETTINGS[case["setting"]][0]:
            for s in SETTINGS[case["setting"]][1]:
                n = -(-(case["h"] - s + 1) // p) * -(-(case["w"] - s + 1) // p)
                flops += n * (n - 1) // 2 * p * p * 14
        return {"bytes": 12 * case["h"] * case["w"], "flops": flops}
    if kind == "batch":
        n = sum(h * w for h, w in _batch_sides(case))
    else:
        n = case["h"] * case["w"]
    if kind == "boxcar":
        return {"bytes": 24 * n, "flops": 30 * n}
    if kind == "goldstein":
        # four 32-point FFT passes of 5 N log2 N over the covering patches
        return {"bytes": 20 * n, "flops": int(n * (32 / (32 - 2 * case["overlap"])) ** 2 * 4 * 5 * 5) + 20 * n}
    if kind == "nlinsar":
        half = (case["search"] ** 2 - 1) // 2
        return {"bytes": 36 * n * case["niter"],
                "flops": n * case["niter"] * (half * (60 + 4 * (case["patch"] - 1)) + 2 * half * 8)}
    planes = 2 * case["dim"] ** 2 if kind == "covmat" else 3
    return {"bytes": 2 * 4 * planes * n,
            "flops": n * _nlsar_flops(case.get("dim", 2), case["search"], case["setting"], case["select"])}


# ---------------------------------------------------------------------------
# the definitions in 64 bits
# ---------------------------------------------------------------------------

def _chi2_table(n=256, dof=49.0):
    """Chi-squared quantiles of i / n (bisection on the incomplete gamma
    function); the last entry is 1e5 by definition."""
    p = (torch.arange(n, dtype=torch.float32) * np.float32(1.0 / n)).double()
    lo, hi = torch.zeros(n, dtype=torch.float64), torch.full((n,), 1000.0, dtype=torch.float64)
    half = torch.full((n,), dof / 2, dtype=torch.float64)
    for _ in range(80):
        mid = 0.5 * (lo + hi)
        below = torch.special.gammainc(half, mid / 2) < p
        lo, hi = torch.where(below, mid, lo), torch.where(below, hi, mid)
    q = 0.5 * (lo + hi)
    q[0], q[-1] = 0.0, 1e5
    return q


def _gauss(s):
    h = (s - 1) // 2
    x = torch.arange(-h, h + 1, dtype=torch.float64)
    g = torch.exp(-math.pi * (x[:, None] ** 2 + x[None, :] ** 2) / (h + 0.5) ** 2)
    return (g / g.sum()).tolist()


def _sim_planes(planes, dim, s):
    """Rescaled and Gaussian-averaged similarity reals of the valid region:
    2x2 [C00, C11, Re C01, Im C01]; 3x3 the diagonal, then (Re, Im) of C01,
    C02, C12."""
    pick = [0, 6, 2, 3] if dim == 2 else [0, 8, 16, 2, 3, 4, 5, 10, 11]
    gamma = (1.0 / dim) ** 0.33333
    g = _gauss(s)
    h, w = planes.shape[-2] - s + 1, planes.shape[-1] - s + 1
    out = []
    for k, p in enumerate(pick):
        a = sum(g[i][j] * planes[p, i:i + h, j:j + w] for i in range(s) for j in range(s))
        out.append(a * gamma if k >= dim else a)
    return out


def _det(c):
    if len(c) == 4:
        return c[0] * c[1] - c[2] * c[2] - c[3] * c[3]
    a, b, d, xr, xi, yr, yi, zr, zi = c
    return (a * b * d - a * (zr * zr + zi * zi) - b * (yr * yr + yi * yi) - d * (xr * xr + xi * xi) +
            2 * (xr * zr * yr - xi * zi * yr + xr * zi * yi + xi * zr * yi))


def _glr(ca, la, cb, lb, dim):
    r = 2 * torch.log(_det([x + y for x, y in zip(ca, cb)])) - la - lb - 2 * dim * math.log(2.0)
    return torch.nan_to_num_(r, nan=0.0, posinf=math.inf, neginf=-math.inf)


def _train(planes, dim, p, s):
    """(dmin, dmax, quantiles, chi2) of one patch and scale size."""
    c = _sim_planes(planes, dim, s)
    h, w = c[0].shape
    nh, nw = -(-h // p), -(-w // p)
    dev = planes.device
    y = (torch.arange(nh, device=dev)[:, None] * p + torch.arange(p, device=dev)).clamp(max=h - 1)
    x = (torch.arange(nw, device=dev)[:, None] * p + torch.arange(p, device=dev)).clamp(max=w - 1)
    pat = [t[y[:, None, :, None], x[None, :, None, :]].reshape(nh * nw, p * p) for t in c]
    ld = torch.log(_det(pat))
    n = nh * nw
    i, j = torch.tril_indices(n, n, -1, device=dev)
    parts = []
    for k in range(0, i.numel(), 1 << 20):
        a, b = i[k:k + (1 << 20)], j[k:k + (1 << 20)]
        parts.append(sum(_glr([t[a, e] for t in pat], ld[a, e], [t[b, e] for t in pat], ld[b, e], dim)
                         for e in range(p * p)))
    d = torch.cat(parts)
    d = torch.sort(d[torch.isfinite(d)]).values
    step = (d[-1] - d[0]) / 256
    at = d[0] + step * torch.arange(256, device=dev, dtype=torch.float64)
    return float(d[0]), float(d[-1]), torch.searchsorted(d, at).double() / d.numel(), _chi2_table()


def _clamped(t, top, left, h, w):
    """Rows top .. top + h - 1 and columns left .. of the clamp-extended t."""
    y = torch.arange(top, top + h, device=t.device).clamp(0, t.shape[-2] - 1)
    x = torch.arange(left, left + w, device=t.device).clamp(0, t.shape[-1] - 1)
    return t[..., y, :][..., x]


def _box(t, p):
    """p x p sums, valid region."""
    h, w = t.shape[-2] - p + 1, t.shape[-1] - p + 1
    r = sum(t[..., k:k + w] for k in range(p))
    return sum(r[..., k:k + h, :] for k in range(p))


def _nlsar(planes, dim, case):
    """Blended weighted means [2 dim^2][h][w] of an NL-SAR call."""
    patches, scales = SETTINGS[case["setting"]]
    tables = _stats_tables(dim, case["setting"])
    keys = sorted(tables)
    chosen = keys[-1:] if case["select"] == "reference" else keys
    h, w = planes.shape[-2:]
    wsh = (case["search"] - 1) // 2
    overlap = wsh + (max(patches) - 1) // 2 + (max(scales) - 1) // 2
    # the last output row (column) is the one `overlap` past the scene
    H, W = h + overlap, w + overlap
    best = torch.full((H, W), -1.0, dtype=torch.float64, device=planes.device)
    best_rank = torch.full((H, W), 1 << 30, device=planes.device)
    blend = None
    centre = _clamped(planes, 0, 0, H, W)
    around = _clamped(planes, -wsh, -wsh, H + 2 * wsh, W + 2 * wsh)
    diag = [0, 6] if dim == 2 else [0, 8, 16]
    # planes that hold something: the 2x2 images' lower triangle mirrors the upper
    used = [k for k in range(len(planes)) if bool((planes[k] != 0).any())]
    for s in sorted({k[1] for k in chosen}):
        group = [k for k in chosen if k[1] == s]
        phm, shm = max((k[0] - 1) // 2 for k in group), (s - 1) // 2
        g = phm + wsh
        c = _sim_planes(_clamped(planes, -g - shm, -g - shm, H + 2 * (g + shm), W + 2 * (g + shm)), dim, s)
        ld = torch.log(_det(c))
        acc = {k: [torch.zeros((H, W), dtype=torch.float64, device=planes.device)
                   for _ in range(2 + dim + len(used))] for k in group}

        def shifted(t, dy, dx, m):
            return t[..., wsh + dy:wsh + dy + H + 2 * m, wsh + dx:wsh + dx + W + 2 * m]

        for dy in range(-wsh, wsh + 1):
            for dx in range(-wsh, wsh + 1):
                v = {q: around[q, wsh + dy:wsh + dy + H, wsh + dx:wsh + dx + W] for q in used}
                sim = None
                if dy or dx:
                    sim = _glr([shifted(t, 0, 0, phm) for t in c], shifted(ld, 0, 0, phm),
                               [shifted(t, dy, dx, phm) for t in c], shifted(ld, dy, dx, phm), dim)
                for k in group:
                    A = acc[k]
                    if sim is None:
                        wt = torch.ones((H, W), dtype=torch.float64, device=planes.device)
                    else:
                        lo, hi, q, chi = tables[k]
                        m = phm - (k[0] - 1) // 2
                        d = _box(sim[m:sim.shape[0] - m, m:sim.shape[1] - m], k[0])
                        tab = torch.from_numpy(chi.astype(np.float64)[(q * np.float32(255)).astype(np.int64)])
                        tab = torch.exp(-(tab - 49.0).abs() / 15.0).to(planes.device)
                        lo, hi = float(lo), float(hi)
                        i = ((d.clamp(lo, hi) - lo) / (hi - lo) * 255).to(torch.int64)
                        wt = torch.where(d > hi, 0.0, tab[i])
                    A[0] += wt
                    A[1].addcmul_(wt, wt)
                    for e, p in enumerate(diag):
                        A[2 + e].addcmul_(wt, v[p] * v[p])
                    for e, p in enumerate(used):
                        A[2 + dim + e].addcmul_(wt, v[p])
        for k in group:
            A = acc[k]
            alpha = torch.zeros_like(A[0])
            for e, p in enumerate(diag):
                mean = A[2 + dim + used.index(p)] / A[0]
                var = A[2 + e] / A[0] - mean * mean
                alpha = torch.maximum(alpha, torch.nan_to_num((var - mean * mean) / var, nan=0.0).clamp(min=0.0))
            enl = A[0] * A[0] / A[1]
            enl = enl / ((1 - alpha) ** 2 + (alpha * alpha + 2 * alpha * (1 - alpha) / A[0]) * enl)
            rank = keys.index(k)
            take = (enl > best) | ((enl == best) & (rank < best_rank)) | (case["select"] == "reference")
            best, best_rank = torch.where(take, enl, best), torch.where(take, rank, best_rank)
            mine = torch.zeros_like(centre)
            for e, p in enumerate(used):
                mine[p] = (1 - alpha) * A[2 + dim + e] / A[0] + alpha * centre[p]
            blend = mine if blend is None else torch.where(take, mine, blend)
        del acc
    rows = torch.arange(h, device=planes.device)
    rows[-1] = H - 1
    cols = torch.arange(w, device=planes.device)
    cols[-1] = W - 1
    return blend[:, rows, :][:, :, cols]


def _insar_planes(a1, a2, ph):
    a1, a2, ph = a1.double(), a2.double(), ph.double()
    z = torch.zeros_like(a1)
    return torch.stack([a1 * a1, z, a1 * a2 * torch.cos(ph), a1 * a2 * torch.sin(ph), z, z, a2 * a2, z])


def _insar(a1, a2, ph, case):
    c = _nlsar(_insar_planes(a1, a2, ph), 2, case)
    am, as_ = torch.sqrt(c[0]), torch.sqrt(c[6])
    return (0.25 * (am + as_) ** 2, torch.atan2(c[3], c[2]), torch.sqrt(c[2] * c[2] + c[3] * c[3]) / (am * as_))


def _boxcar(a1, a2, ph, w):
    a1, a2, ph = a1.double(), a2.double(), ph.double()
    r = (w - 1) // 2
    h, wd = a1.shape
    z = torch.stack([0.5 * (a1 * a1 + a2 * a2), a1 * a2 * torch.cos(ph), a1 * a2 * torch.sin(ph)])
    del a1, a2, ph
    rows, cols = torch.arange(h), torch.arange(wd)
    rows[-1] += r
    cols[-1] += r
    y = [(rows + k).clamp(0, h - 1).to(z.device) for k in range(-r, r + 1)]
    x = [(cols + k).clamp(0, wd - 1).to(z.device) for k in range(-r, r + 1)]
    t = sum(z[:, :, i] for i in x)
    del z
    t = sum(t[:, i, :] for i in y)
    return t[0] / (w * w), torch.atan2(t[2], t[1]), torch.sqrt(t[1] ** 2 + t[2] ** 2) / t[0]


def _goldstein(a1, a2, ph, ov, alpha):
    amp, ph = 0.5 * (a1.double() + a2.double()), ph.double()
    z = torch.complex(amp * torch.cos(ph), amp * torch.sin(ph))
    h, w = z.shape
    p, s = 32, 32 - 2 * ov
    m = max(h, w) + 2 * ov
    sub = m - m % s + s
    n = sub // s
    out = torch.empty_like(z)
    step = sub - 2 * ov
    tops, lefts = list(range(-ov, h, step)), list(range(-ov, w, step))
    pos = torch.arange(n * s + 2 * ov, device=z.device) - ov  # tile positions that patches cover
    edge = torch.where((pos < ov) | (pos >= sub - ov), 2.0, 1.0).double()
    k = torch.arange(p, device=z.device)
    ends = torch.where((k < 2 * ov) | (k >= p - 2 * ov), 0.5, 1.0).double()
    for i, h0 in enumerate(tops):
        for j, w0 in enumerate(lefts):
            tile = _clamped(z, h0, w0, sub, sub)
            ext = _clamped(tile, -ov, -ov, sub + 2 * ov, sub + 2 * ov)
            pat = ext.unfold(0, p, s).unfold(1, p, s)  # [n][n][p][p]
            back = torch.zeros_like(ext)
            for py in range(0, n, 32):  # strips of patch rows
                f = torch.fft.fft2(pat[py:py + 32])
                f = torch.fft.ifft2(f * f.abs() ** alpha) * (ends[:, None] * ends[None, :])
                for a in range(f.shape[0]):
                    top = (py + a) * s
                    for b in range(2):  # patches of one parity do not overlap
                        view = back[top:top + p, b * s:]
                        q = f[a, b::2]
                        if q.shape[0]:
                            view.as_strided((q.shape[0], p, p), (2 * s, back.stride(0), 1),
                                            view.storage_offset()).add_(q)
            back = (back * (edge[:, None] * edge[None, :]))[ov:ov + sub, ov:ov + sub] + tile
            last_r, last_c = i == len(tops) - 1, j == len(lefts) - 1
            y0, x0 = min(i * step, h - 1), min(j * step, w - 1)
            y1 = h if last_r else min((i + 1) * step, h - 1)
            x1 = w if last_c else min((j + 1) * step, w - 1)
            if y1 <= y0 or x1 <= x0:
                continue
            ty = torch.arange(y0, y1, device=z.device) - h0
            tx = torch.arange(x0, x1, device=z.device) - w0
            if last_r:
                ty[-1] = sub - ov - 1
            if last_c:
                tx[-1] = sub - ov - 1
            out[y0:y1, x0:x1] = back[ty][:, tx]
    return out.abs(), out.angle()


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        planes = _insar_planes(*_train_area(case["h"], case["w"], seed))
        patches, scales = SETTINGS[case["setting"]]
        out = {}
        for p in patches:
            for s in scales:
                lo, hi, q, c = _train(planes, 2, p, s)
                out["%d_%d" % (p, s)] = [lo, hi, q.cpu().numpy(), c.numpy()]
        return out
    if kind == "boxcar":
        return _boxcar(*_scene(case["h"], case["w"], seed), case["window"])
    if kind == "goldstein":
        return _goldstein(*_scene(case["h"], case["w"], seed), case["overlap"], case["alpha"])
    if kind == "nlinsar":
        # its smoothing keeps the lmin largest of 441 weights and switches
        # where two of them agree to the last bits, and each pass feeds the
        # next: runs in 32 and in 64 bits part on a share of the pixels
        return None
    if kind == "covmat":
        return _nlsar(_covmat_scene(case["dim"], case["h"], case["w"], seed).double(), case["dim"], case)
    if kind == "batch":
        return [_insar(*_scene(h, w, seed + 1000 * i), case) for i, (h, w) in enumerate(_batch_sides(case))]
    got = _insar(*_scene(case["h"], case["w"], seed), case)
    return [t.cpu().numpy() for t in got] if kind == "host" else got
